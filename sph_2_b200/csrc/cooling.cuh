// cooling.cuh -- device functions of the implicit cooling solve, shared by
// the exact solver (cooling.cu) and the surrogate's fallback (mlp.cu).
//
// Same structure as DoCooling (GPU_sph/With_cooling/Model_C/
// myPhotoLibsGPU.h:615-686): solve  u - u_old - ratefact * Lambda_net(u) * dt = 0
// with ratefact = nH^2/rho, by bracketing (factors of 1.1) and bisection to
// |du/u| <= tol, in FP64 and with every loop bounded.  Lambda_net is the
// synthetic cooling function of the cooling-cloud workload: a log-log table of
// Lambda(T) (n_bins power-law pieces between T0 and T1) and a constant heating
// per H atom; T = (gamma-1) mu m_H u / k_B.
#pragma once
#include "sph_internal.cuh"

#define KB_CGS 1.380649e-16
#define MH_CGS 1.6726e-24

// one bin of the fast cooling function: Lambda = lamT T (T / T_e)^sm1 with T_e
// the bin's lower edge, and the first and last bin of the run of bins around it
// where Lambda does not fall with T (the bin itself where it does fall)
struct __align__(16) CoolBin {
    double lamT, invT, T;  // Lambda(T_e) / T_e, 1 / T_e, T_e
    float sm1;             // d ln Lambda / d ln T - 1
    short dn, un;
    double logL, s, diff;  // log10 Lambda(T_e), the slope, the rise
    double pad;
};
constexpr int COOL_EDGES = 4097;  // edges of the largest table
// the cooling tables in one allocation: log Lambda at the edges, a CoolBin per bin,
// and (log Lambda, slope) per bin in FP32
constexpr size_t COOL_AT_BIN = sizeof(double) * (COOL_EDGES + 1);
constexpr size_t COOL_AT_BINF = COOL_AT_BIN + sizeof(CoolBin) * COOL_EDGES;
constexpr size_t COOL_BYTES = COOL_AT_BINF + sizeof(float2) * COOL_EDGES;

struct CoolDev {
    const double *logL;
    const CoolBin *bin;
    const float2 *binf;  // (log10 Lambda(T_e), slope) in FP32
    int nb;
    double logT0, logT1, mu, gamma, XH, gheat, tol;
    double kT, invkT;     // T = kT u
    double dl;            // (logT1 - logT0) / nb
    float l2T0, l2inv;    // bin of T: (log2 T - l2T0) l2inv
    int max_iter;
};

// The cooling function Lambda(T): a power of T in each bin of the table, the end
// bins' beyond it.  One copy of its log10 and exp10: inlined at each of the solve's ten
// call sites they overran the instruction cache (no_instruction the first
// stall, 5.3 of 11.8 cycles per issue).
static __device__ __noinline__ double cool_lambda_call(const CoolBin *bin, int nb, double logT0,
                                                       double dl, double T) {
    const double lt = log10(T);
    int k = (int)floor((lt - logT0) / dl);
    k = k < 0 ? 0 : (k > nb - 1 ? nb - 1 : k);
    return exp10(bin[k].logL + bin[k].s * (lt - (logT0 + k * dl)));
}

// x / 1.1 in round to nearest: x times a two-part reciprocal in one FMA
// (Brisebarre, Muller and Raina, IEEE Trans. Computers 53, 2004).  The product
// is off by less than 2^-106 before it is rounded, so only a quotient that
// close to a midpoint of two doubles could round differently; every such
// mantissa (the solutions of 2^(s+1) X = (2 M + 1) C + d for small d) was
// checked exactly.  For x whose x zl is normal; div_1_1 takes the others too.
__device__ __forceinline__ double div_1_1_normal(double x) {
    return fma(x, 0.9090909090909091, x * -4.3124365419324254e-17);
}
__device__ __forceinline__ double div_1_1(double x) {
    return x > 1e-250 && x < 1e300 ? div_1_1_normal(x) : x / 1.1;
}

// The residual r(u) = u - u_old - ratefact net(u) dt of one row.  The
// bracketing and the bisection read nothing of it but its sign, and the FP64
// cooling function is a log10 and an exp10 (some 150 FP64 instructions with the
// residual), so most signs are taken without it; each shortcut below decides a
// sign only where it is certain, with the FP64 residual for the rest, so u and
// the count are those of the plain iteration.
struct CoolRes {
    double u_old, dt, nH, ratefact, A, heat;
    double sum;  // u_old + heat; infinite where not plain: no sign is certain then
    bool plain;  // finite, positive: the shortcuts' arithmetic and bounds hold
    __device__ __forceinline__ CoolRes(const CoolDev &c, double rho, double u_old_, double dt_)
        : u_old(u_old_), dt(dt_) {
        nH = c.XH * rho / MH_CGS;
        ratefact = nH * nH / rho;
        A = ratefact * dt;
        heat = A * (c.gheat / nH);
        plain = u_old > 0.0 && u_old < 1e30 && A > 0.0 && A < 1e300 && heat >= 0.0 && heat < 1e300;
        sum = plain ? u_old + heat : (double)INFINITY;
    }
    __device__ __forceinline__ int bin(const CoolDev &c, double T) const {
        const int k = (int)floorf((__log2f((float)T) - c.l2T0) * c.l2inv);
        return k < 0 ? 0 : (k > c.nb - 1 ? c.nb - 1 : k);
    }
    __device__ __forceinline__ double exact(const CoolDev &c, double u) const {
        const double T = (c.gamma - 1.0) * c.mu * MH_CGS / KB_CGS * u;
        const double net = c.gheat / nH - cool_lambda_call(c.bin, c.nb, c.logT0, c.dl, T);
        return u - u_old - ratefact * net * dt;
    }
    // A Lambda(u) with the power (T / T_e)^sm1 formed in FP32 on the SFU, and a
    // bound on its relative error: T / T_e is a FP64 product rounded once; the
    // SFU's log2 is within 2^-21.4 near 1 and 3 ulp beyond, its exp2 within
    // 2 ulp plus the argument's own error times ln 2, together below
    // 5e-7 (1 + |sm1| (1 + |x|)), four times which is allowed; a bin one off
    // at an edge changes nothing (the pieces meet there)
    __device__ __forceinline__ double fast(const CoolDev &c, double u, float &sm1, float &rel) const {
        const double T = c.kT * u;
        const CoolBin b = c.bin[bin(c, T)];
        const float x = __log2f((float)(T * b.invT));
        sm1 = b.sm1;
        rel = 2e-6f * (1.f + fabsf(sm1) * (1.f + fabsf(x)));
        return A * b.lamT * T * (double)exp2f(sm1 * x);
    }
    __device__ __forceinline__ int sign(const CoolDev &c, double u) const {
        float sm1, rel;
        const double cool = fast(c, u, sm1, rel), r = u - u_old - (heat - cool);
        // (values outside the FP32 range give a bound that is not finite)
        if (fabs(r) > cool * (double)rel + 1e-14 * (u + sum + cool)) return r > 0.0 ? 1 : -1;
        const double re = exact(c, u);
        return re > 0.0 ? 1 : (re < 0.0 ? -1 : 0);
    }
    // r at the lower edge of bin k with lam Lambda there (or a bound of it):
    // certainly of sign s?
    __device__ __forceinline__ bool edge_is(int s, double ue, double lam) const {
        const double cool = A * lam, v = ue - u_old + cool - heat;
        return s * v > 1e-12 * (ue + u_old + cool + heat);
    }
    // How far from u_old the sign s0 of r(u_old) certainly holds: edges of the
    // table, towards smaller (s0 > 0) or larger u, where r needs no
    // transcendental.  Over a run of bins where Lambda does not fall r only
    // increases, so the run's end decides for all of it; in a bin where it
    // falls, u and Lambda at their unfavourable ends bound r.  Returns the last
    // such edge's u (u_old if none); [k0, k1] becomes the run or bin beyond.
    __device__ __forceinline__ double reach(const CoolDev &c, int s0, int &k0, int &k1) const {
        const double T0 = c.kT * u_old;
        int k = bin(c, T0);
        if (k > 0 && c.bin[k].T > T0) k--;
        if (k < c.nb - 1 && c.bin[k + 1].T <= T0) k++;
        double safe = u_old;
        while (true) {
            const CoolBin b = c.bin[k];
            const bool rise = b.sm1 >= -1.f;
            k0 = rise ? b.dn : k;
            k1 = rise ? b.un : k;
            // the run's far edge, unless the table ends with it
            const int e = s0 > 0 ? k0 : k1 + 1;
            if (e == 0 || e == c.nb) return safe;
            const CoolBin x = c.bin[e];
            double lam = x.lamT * x.T;
            if (!rise) {
                // Lambda falls: smallest at the bin's top, largest at its bottom
                if (s0 > 0 ? k == c.nb - 1 : T0 < c.bin[0].T) return safe;
                const CoolBin y = s0 > 0 ? c.bin[k + 1] : b;
                lam = y.lamT * y.T;
            }
            if (!edge_is(s0, x.T * c.invkT, lam)) return safe;
            safe = x.T * c.invkT;
            k = s0 > 0 ? e - 1 : e;
        }
    }
    // r increases all over bin b of the table: r' = 1 + A s Lambda / u > 0,
    // smallest where the slope s is negative at the bin's lower edge
    __device__ __forceinline__ bool rises(const CoolDev &c, const CoolBin &b) const {
        return b.sm1 >= -1.f || 1.0 + A * ((double)b.sm1 + 1.0) * b.lamT * c.kT > 1e-4;
    }
    // r increases all over [lo, up]
    __device__ __forceinline__ bool monotone(const CoolDev &c, double lo, double up) const {
        const double Tl = c.kT * lo;
        for (int k = bin(c, Tl * (1.0 - 1e-4)), ke = bin(c, c.kT * up * (1.0 + 1e-4)); k <= ke; k++) {
            const CoolBin b = c.bin[k];
            if (b.sm1 < -1.f && !(Tl > c.bin[0].T && rises(c, b))) return false;
        }
        return true;
    }
    // An interval [a, b] that holds the root of r between lo and up, where r
    // increases: with S = u_old + heat the root solves u + A Lambda(u) = S, a
    // rising line of slopes between 1 and s in (log u, log(u + A Lambda)), so a
    // few Newton steps there in FP32, kept inside the bracket that they narrow,
    // reach it to some 1e-6; then one step on the FP64 residual, and the FP64
    // signs 2e-9 of u on either side.  An end that they do not confirm is left
    // alone.
    __device__ __forceinline__ void enclose(const CoolDev &c, double lo, double up, double start,
                                            double &a, double &b) const {
        const double S = u_old + heat, iS = 1.0 / S;
        float x = __log2f((float)(start * iS)), sm1 = 0.f, rel;
        float xl = lo > 0.0 ? __log2f((float)(lo * iS)) : -INFINITY, xh = __log2f((float)(up * iS));
        double u = start, cool = 0.0;
#pragma unroll 1
        for (int it = 0; it < 12; it++) {
            cool = fast(c, u, sm1, rel);
            const float v = (float)(u * iS), q = (float)(cool * iS), y = __log2f(v + q);
            if (y > 0.f) xh = fminf(xh, x); else xl = fmaxf(xl, x);
            float nx = x - __fdividef(y * (v + q), v + (sm1 + 1.f) * q);
            if (!(nx >= xl && nx <= xh)) nx = isfinite(xl + xh) ? 0.5f * (xl + xh) : x - 1.f;
            const float dx = fabsf(nx - x);
            x = nx;
            u = S * (double)exp2f(x);
            if (dx < 4e-6f + 2.5e-7f * fabsf(x)) break;
        }
        const double rp = 1.0 + cool * (double)(sm1 + 1.f) / u;
        if (!(u > lo && u < up && rp > 0.0)) return;
        u -= exact(c, u) / rp;
        const double w = 2e-9 * u + 1e-13 * (u + u_old + heat + cool) / rp;
        if (u - w > lo && u - w < up && exact(c, u - w) < 0.0) a = u - w;
        if (u + w < up && u + w > lo && exact(c, u + w) > 0.0) b = u + w;
    }
};

// |du / u| > tol, dividing only where the product cannot tell
__device__ __forceinline__ bool cool_wide(const CoolDev &c, double du, double u) {
    const double x = fabs(du), y = c.tol * fabs(u);
    if (x > y * (1.0 + 1e-14)) return true;
    if (x < y * (1.0 - 1e-14)) return false;
    return fabs(du / u) > c.tol;
}

// The iteration with every sign from the FP64 residual, for rows outside the
// shortcuts' range (a step back in time, a heating rate below zero, magnitudes
// beyond it): their bounds take every term to be positive.  Not inlined, so that
// the other rows' registers do not pay for it (2^20 plain rows: 279 us, against 292
// with such rows in the loops below).
struct CoolOut {
    double u;
    int count;
};
static __device__ __noinline__ CoolOut cool_solve_bare(CoolDev c, double rho, double u_old, double dt) {
    const CoolRes res(c, rho, u_old, dt);
    double u = u_old, up = u, lo = u;
    const double r0 = res.exact(c, u);
    int guard = 0;
    if (r0 > 0.0) {
        while (res.exact(c, up) > 0.0 && guard++ < 2000) up /= 1.1;
        lo = up;
        up = lo * 1.1;
    } else if (r0 < 0.0) {
        while (res.exact(c, up) < 0.0 && guard++ < 2000) up *= 1.1;
        lo = up / 1.1;
    } else {
        return {u, 0};
    }
    double du = u;
    int it = 1;
    while (cool_wide(c, du, u) && it < c.max_iter) {
        u = 0.5 * (lo + up);
        if (res.exact(c, u) > 0.0) up = u; else lo = u;
        du = fabs(up - lo);
        it++;
    }
    return {u, cool_wide(c, du, u) ? -1 : it};
}

// Returns the bisection count, -1 if the tolerance was not reached.  What is
// known of r's sign is kept as r < 0 on [kl, a] and r > 0 on [b, kh]; with the
// root enclosed, bracket and bisection only compare with it.  2^20 states of
// the training range: 1.49 ms with every sign from the FP64 residual, 0.65
// ms with sign() alone (a row takes 46 bracket steps and 17 bisections, the
// longest of a warp 168), 0.25 ms with the reach and the enclosure, 13 of whose
// 49 thousand cycles a warp are the bracket's divisions.
// BARE: rows that are not plain leave by a call; without it they stay in these loops
// with every sign exact, for kernels whose registers a call would cost more (the
// tensor-core surrogate: 129 us, with it 135).
template <bool BARE = true>
__device__ __forceinline__ int cool_solve(const CoolDev &c, double rho, double u_old, double dt, double *u_new) {
    const CoolRes res(c, rho, u_old, dt);
    if (BARE && !res.plain) {
        const CoolOut o = cool_solve_bare(c, rho, u_old, dt);
        *u_new = o.u;
        return o.count;
    }
    double u = u_old, up = u, lo = u;
    const int s0 = res.sign(c, u);
    int guard = 0;
    if (s0 == 0) {
        *u_new = u;
        return 0;
    }
    double kl = INFINITY, a = -INFINITY, b = INFINITY, kh = -INFINITY;
    bool enclosed = false;
    if (BARE || res.plain) {
        int k0, k1;
        const double safe = res.reach(c, s0, k0, k1);
        // r increases over the run (or the bin) beyond the reach: its root, if
        // it is there
        const CoolBin b0 = c.bin[k0];
        const double e0 = k0 > 0 ? b0.T * c.invkT : 0.0;
        const double e1 = k1 < c.nb - 1 ? c.bin[k1 + 1].T * c.invkT : 1e300;
        const bool inc = res.rises(c, b0) && (k0 > 0 || b0.sm1 >= -1.f);
        if (s0 > 0) {
            kh = u_old;
            b = safe * (1.0 + 1e-12);
            if (inc) {
                res.enclose(c, e0, safe, safe, a, b);
                kl = e0;
            }
            enclosed = a > 0.0 && b < safe;
        } else {
            kl = u_old;
            a = safe * (1.0 - 1e-12);
            if (inc) {
                res.enclose(c, safe, e1, safe, a, b);
                kh = e1;
            }
            enclosed = b < 1e300 && a > safe;
        }
    }
    auto sgn = [&](double v) {
        if (v >= b && v <= kh) return 1;
        if (v <= a && v >= kl) return -1;
        return res.sign(c, v);
    };
    if (s0 > 0) {
        // four steps at a time while the last of them is still known
        while (guard < 1996 && up <= kh && up > 1e-200) {
            const double t = div_1_1_normal(div_1_1_normal(div_1_1_normal(div_1_1_normal(up))));
            if (!(t >= b)) break;
            up = t;
            guard += 4;
        }
        while (sgn(up) > 0 && guard++ < 2000) up = div_1_1(up);
        lo = up;
        up = lo * 1.1;
    } else {
        while (guard < 1996) {
            const double t = up * 1.1 * 1.1 * 1.1 * 1.1;
            if (!(t <= a && up >= kl)) break;
            up = t;
            guard += 4;
        }
        while (sgn(up) < 0 && guard++ < 2000) up *= 1.1;
        lo = div_1_1(up);
    }
    if ((BARE || res.plain) && !enclosed && res.monotone(c, lo, up)) {
        // (only what this confirms about the bracket counts)
        a = -INFINITY;
        b = INFINITY;
        res.enclose(c, lo, up, 0.5 * (lo + up), a, b);
        kl = lo;
        kh = up;
    }
    double du = u;
    int it = 1;
    while (cool_wide(c, du, u) && it < c.max_iter) {
        u = 0.5 * (lo + up);
        if (sgn(u) > 0) up = u; else lo = u;
        du = fabs(up - lo);
        it++;
    }
    *u_new = u;
    return cool_wide(c, du, u) ? -1 : it;
}

// ---- the surrogate's side in FP32 -------------------------------------------
// The surrogate is accepted to a relative error of mlp_err_tol (1e-3 by
// default), far above FP32 rounding, so its Newton polish, error estimate and
// monotonicity test run in FP32, where the logarithm and exponential are
// single SFU instructions (the FP64 ones are long FMA-pipe sequences and made
// the FP64 polish as slow as the exact bisection it should replace).  The
// residual u - u_old - ratefact * net * dt is formed in FP32 from FP32 u and
// u_old: its rounding (~1e-7 u) is four orders below the tolerance.  The
// products are ordered so that no intermediate leaves the FP32 range:
// ratefact = nH^2 / rho reaches 1e29 and ratefact * dt 1e42, but ratefact *
// Lambda stays below 1e10 and its product with dt below 1e25.  The exact
// solver and the fallback stay in FP64.
__device__ __forceinline__ float cool_lambda_f(const CoolDev &c, float T, float *slope) {
    const float lt = __log10f(T);
    const float lT0 = (float)c.logT0;
    const float dl = (float)((c.logT1 - c.logT0) / c.nb);
    int k = (int)floorf((lt - lT0) / dl);
    k = k < 0 ? 0 : (k > c.nb - 1 ? c.nb - 1 : k);
    const float2 b = c.binf[k];
    if (slope) *slope = b.y;
    return __exp10f(b.x + b.y * (lt - (lT0 + k * dl)));
}

// Newton steps of u - u_old - ratefact net(u) dt = 0 from an approximate solution
// *u (the surrogate's prediction): at each iterate r(u) and r'(u) = 1 + ratefact
// dt s Lambda(T) / u (Lambda ~ T^s inside a bin, T ~ u) give the error estimate
// |r / r'| / u; the iterate is kept as soon as that is within tol / 4, else
// u <- u - r / r' (while r' > 0 and u stays positive), at most four steps.
// *est <- the estimate of the returned *u (+inf where it is void).
__device__ __forceinline__ void cool_newton_polish_f(const CoolDev &c, double rho, double u_old,
                                                     double dt, double *u, double *est, double tol) {
    const double nHd = c.XH * rho / MH_CGS;
    const float ratefact = (float)(nHd * nHd / rho);
    const float kT = (float)((c.gamma - 1.0) * c.mu * MH_CGS / KB_CGS);
    const float gn = (float)(c.gheat / nHd);
    const float uo = (float)u_old, fdt = (float)dt, ftol = (float)tol;
    float uu = (float)*u;
    *est = INFINITY;
    for (int it = 0; it < 5; it++) {
        float s;
        const float lam = cool_lambda_f(c, kT * uu, &s);
        const float r = uu - uo - (ratefact * (gn - lam)) * fdt;
        const float rp = 1.f + (ratefact * lam) * fdt * s / uu;
        if (!(rp > 0.f) || !(uu > 0.f)) break;  // the estimate is void here
        const float e = fabsf(r / rp) / uu;
        *u = (double)uu;
        *est = (double)e;
        if (e <= 0.25f * ftol || it == 4) break;
        const float u1 = uu - r / rp;
        if (!(u1 > 0.f)) break;
        uu = u1;
    }
}

// True when r(u) increases strictly on [u_lo, u_hi].  Inside a bin Lambda / u ~
// T^(s-1): r' > 1 where s >= 0, and where s < 0 r' grows with T, so it is smallest
// at the bin's lower end.  r' > 0 at T(u_lo) (when its bin has s < 0) and at the
// lower edge of every bin with s < 0 that starts inside the interval decides;
// Lambda / T at the edges is tabulated, so only T(u_lo) needs a transcendental.
__device__ __forceinline__ bool cool_monotone_f(const CoolDev &c, double rho, double dt, double u_lo,
                                                double u_hi) {
    // A = ratefact * dt can pass the FP32 range: it is applied in FP64 to
    // the Lambda / T values (two multiplies, no transcendental)
    const double A = (c.XH * rho / MH_CGS) * (c.XH * rho / MH_CGS) / rho * dt;
    const float kT = (float)((c.gamma - 1.0) * c.mu * MH_CGS / KB_CGS);
    const float lT0 = (float)c.logT0;
    const float dl = (float)((c.logT1 - c.logT0) / c.nb);
    const float T0 = kT * (float)u_lo, T1 = kT * (float)u_hi;
    if (!(T0 > 0.f) || !(T1 >= T0)) return false;
    const float l0 = __log10f(T0), l1 = __log10f(T1);
    int k = (int)floorf((l0 - lT0) / dl);
    k = k < 0 ? 0 : (k > c.nb - 1 ? c.nb - 1 : k);
    float s = (float)(c.logL[k + 1] - c.logL[k]) / dl;
    if (s < 0.f) {
        const float lam = __exp10f((float)c.logL[k] + s * (l0 - (lT0 + k * dl)));
        if (!(1.0 + A * (double)(s * (lam / T0) * kT) > 0.0)) return false;
    }
    int kend = (int)floorf((l1 - lT0) / dl);
    kend = kend > c.nb - 1 ? c.nb - 1 : kend;
    // only the bins where Lambda falls can fail: the rising runs between them
    // are stepped over whole (a test of every bin was half of the surrogate
    // kernel's instructions: 1.52e8 -> 0.79e8 for 2^20 rows)
    for (int e = k + 1; e <= kend;) {
        const CoolBin b = c.bin[e];
        if (b.sm1 >= -1.f) {
            e = b.un + 1;
            continue;
        }
        s = (float)b.diff / dl;
        if (s < 0.f) {
            if (!(1.0 + A * (double)s * b.lamT * (double)kT > 0.0)) return false;
        }
        e++;
    }
    return true;
}

// accept a surrogate solution un (after the polish, estimate est)?
__device__ __forceinline__ bool cool_accept_f(const CoolDev &c, double rho, double u_old, double dt,
                                              double un, double est, double tol) {
    if (!(est <= tol) || !(un > 0.0)) return false;
    const double lo = fmin(u_old, un / 1.1), hi = fmax(u_old, un * 1.1);
    return cool_monotone_f(c, rho, dt, lo, hi);
}

static inline CoolDev cool_dev_of(const sph_ctx *ctx) {
    const sph_cooling_params &p = ctx->cool;
    CoolDev c;
    c.logL = ctx->cool_table;
    c.bin = (const CoolBin *)((const char *)ctx->cool_table + COOL_AT_BIN);
    c.binf = (const float2 *)((const char *)ctx->cool_table + COOL_AT_BINF);
    c.nb = p.n_bins;
    c.logT0 = p.logT0;
    c.logT1 = p.logT1;
    c.kT = (p.gamma - 1.0) * p.mu * MH_CGS / KB_CGS;
    c.invkT = 1.0 / c.kT;
    c.dl = (p.logT1 - p.logT0) / p.n_bins;
    c.l2T0 = (float)(p.logT0 * 3.321928094887362);  // log2(10)
    c.l2inv = (float)(p.n_bins / ((p.logT1 - p.logT0) * 3.321928094887362));
    c.mu = p.mu;
    c.gamma = p.gamma;
    c.XH = p.XH;
    c.gheat = p.gamma_heat;
    c.tol = p.tol;
    c.max_iter = p.max_iter;
    return c;
}
