// ngb.cu -- neighbour search over the radix tree and the Newton
// smoothing-length iteration.
//
// Replaces ngbDB_new_v2 (ngb_v3.h:124-238: a per-thread scan of 27 cells of a
// 10^3 grid, radius grown until 70-190 candidates, atomics-ordered output,
// host exit on failure) and smoothing_h_ngb (hfvCLibs_v7_hfv_v2.h:367-455: a
// count-based +-coeff*2h iteration of up to 200 rounds over the list).
//
// Search: one warp per group (a tree node of at most 32 Morton-contiguous
// particles of one cloud).  The warp walks the tree 32 nodes at a time with the
// group's box (LIFO stack in shared memory); buckets that can hold neighbours
// are flattened into a shared list of candidate particles, staged 32 at a time
// in shared memory, and every lane tests the staged candidates against its own
// particle.  Rows are written in traversal order (deterministic);
// sph_get_neighbours exports them sorted.
//
// h iteration (fused with the candidate search): the search writes each
// lane's candidate slots into its particle's row (max_ngb entries) and
// accumulates the kernel sums of the first Newton evaluation on the way; every
// lane then runs a bracketed Newton iteration on (4pi/3)(2h)^3 rho(h) = n_ngb m
// with FP64 updates and convergence test, gathering its row again only for
// the rare second and later evaluations.  Particles whose h outgrows the
// candidate radius are flagged and searched again in the next round; a row
// that overflows shrinks the radius instead.  Between sorts a group keeps its
// rows without a search while the distances its particles and the particles
// near them moved since the rows' search leave the rows complete for a
// radius above 2 h (refit steps move particles by 1e-4 to 1e-2 h each).
#include <climits>

#include "sph_internal.cuh"

namespace {

constexpr int SEARCH_WARPS = 4;
// particles per SM up to which a cloud's searches take 32, 8, 4 or 2 lanes per
// particle (search_split; the measurements behind the lines stand there), and
// the longest searches, in chunks per particle per SM, past which the next h
// iteration leaves 8 lanes for 32 or 32 for 8 (k_kept_shift)
constexpr int SPLIT32_PER_SM = 34, SPLIT8_PER_SM = 68, SPLIT4_PER_SM = 140, SPLIT2_PER_SM = 300;
constexpr double LONG8 = 1.6, LONG32 = 0.45;
// A node that does not fit the stack would leave particles out of rows and lists.
// A round of `take` nodes adds at most `take` entries, so near the stack's end a
// round takes fewer, down to one, whose descent the last SRES entries hold (63
// key bits and 27 index bits of equal keys).
constexpr int SSTK = 512, SRES = 96;
constexpr unsigned FULL = 0xffffffffu;
// pending bucket particles: ranges of consecutive slots, range r starting at
// slot rf[r] and at offset rs[r] of the pending stream (rs ascending; at most
// 31 carried ranges + 32 appended by one round)
constexpr int NRANGE = 64;

struct SearchSmem {
    int stk[SSTK];
    int flat[32];  // slots of the chunk being processed
    int rf[NRANGE], rs[NRANGE];
    double4 stage[32];
    double smass[32];
    // FP32 copies of the staged positions relative to the group's centre and
    // of their h, one array per field (four entries per 128-bit load)
    __align__(8) float fx[32];
    __align__(8) float fy[32];
    __align__(8) float fz[32];
    __align__(8) float fh[32];
    // the same per candidate (x, y, z, m) for the hit loop of the h iteration
    float4 fq[32];
};

__device__ __forceinline__ float2 ldf2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ float4 ldf4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 bc2(float a) { return make_float2(a, a); }

template <class R> struct R2;
template <> struct R2<float> { typedef float2 T; };
template <> struct R2<double> { typedef double2 T; };

// Sums of the h iteration at one trial h: S = sum m_j w(q), D = sum m_j
// w'(q)-form (q = r_ij / h, M4 kernel without its 1/(pi h^3) factor)
template <class R> struct HSums {
    KSum<R> S, D;
    R inv_h;
    // kernel terms at distance r, branch-free in the B-spline form of the
    // two pieces: with a = (2 - q)+ and b = (1 - q)+,
    //   w  = a^3 / 4 - b^3                    (1 - 1.5 q^2 + 0.75 q^3 up to q = 1)
    //   dw = 1.5 a^2 (1 - q) - 3 b^2 (1 - 2q)  (3 - 7.5 q^2 + 4.5 q^3 up to q = 1)
    // both zero from q = 2 on
    __device__ __forceinline__ void terms(R r, R &w, R &dw) const {
        const R q = r * inv_h;
        const R a = fmax(R(2) - q, R(0)), b = fmax(R(1) - q, R(0));
        const R a2 = a * a, b2 = b * b;
        w = fma(R(0.25) * a2, a, -(b2 * b));
        dw = fma(R(1.5) * a2, R(1) - q, R(-3) * b2 * fma(R(-2), q, R(1)));
    }
    __device__ __forceinline__ void add(R r, R m) {
        const R q = r * inv_h;
        if (q < R(2)) {
            R w, dw;
            if (q <= R(1)) {
                w = R(1) - R(1.5) * q * q + R(0.75) * q * q * q;
                dw = R(3) - R(7.5) * q * q + R(4.5) * q * q * q;
            } else {
                const R t = R(2) - q;
                w = R(0.25) * t * t * t;
                dw = R(1.5) * t * t * (R(1) - q);
            }
            S.add(m * w);
            D.add(m * dw);
        }
    }
};

// |r_ij| in the sums' type: the difference taken in FP64, then rounded
template <class R>
__device__ __forceinline__ R pair_r(const double4 &pi, const double4 &pj) {
    const R rx = (R)(pi.x - pj.x), ry = (R)(pi.y - pj.y), rz = (R)(pi.z - pj.z);
    return qsqrt<R>(rx * rx + ry * ry + rz * rz);
}

__device__ __forceinline__ double wmin(double v) {
    for (int o = 16; o; o >>= 1) v = fmin(v, __shfl_xor_sync(FULL, v, o));
    return v;
}
__device__ __forceinline__ double wmax(double v) {
    for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

struct SearchArgs {
    const int *gstart, *gcount, *gcloud, *croot;
    const int *cloud;  // per particle
    double4 *p0;
    // node boxes in FP32 rounded outward: (min rounded down, h_max rounded
    // up), (max rounded up, 0)
    const float4 *sA, *sB;
    const int4 *wL;  // per node: first particle, count, left and right child
    int leaf_size, K;
    int *rows, *cnt;
    int *ngb_cnt;  // list counts written by k_lists_cand (cnt holds candidate counts)
    double *hnb;   // per particle: the largest h_j of its list (written by the list builds)
    // candidate rows of the h iteration: the slots j inside the particle's
    // candidate radius, max_ngb entries per particle (row i at i K)
    int *cidx;
    const void *p1;  // Real4 (v, m)
    // exact search restricted to the particles with only[i] != 0, or to all
    // of them when *only_all != 0 (null: every particle)
    const int *only, *only_all;
    // with only: the marked particles also listed (mlist, *mcount entries): up
    // to mmax of them are searched one by one (k_lists_list), more by k_lists
    const int *mlist, *mcount;
    int mmax;
    __device__ __forceinline__ bool listed() const { return !*only_all && *mcount <= mmax; }
    long long *status;
};

// Walk the tree from `root` and write the rows of the active lanes' particles.
// MODE 0: candidates r^2 <= ri^2 (ri = 2 hc_i, the h iteration's gather radius)
//         with the first Newton evaluation's kernel sums
// MODE 1: exact lists |r|^2 <= (h_i + h_j)^2
// MODE 2: candidates r^2 <= ri^2 alone (the count iteration)
// SPLIT consecutive lanes hold the same particle and each takes 32 / SPLIT of
// the 32 staged candidates of a chunk (see Unit below); a particle's row is in
// candidate order for every SPLIT.  hs then holds the lane's part of the sums.
// Returns the particle's full count on each of its lanes.
template <int MODE, class R = double, int SPLIT = 1>
__device__ __forceinline__ int group_search(SearchSmem &S, const SearchArgs &A, int root, bool act,
                                            int i, const double4 &pi, double ri,
                                            HSums<R> *hs = nullptr, int *chunks = nullptr) {
    static_assert(MODE != 0 || SPLIT == 1, "split searches leave the sums to the rows");
    typedef typename R4<R>::T V4;
    const int lane = threadIdx.x & 31;
    constexpr int SW = 32 / SPLIT;  // staged candidates per lane of a chunk
    const int sl = lane & (SPLIT - 1), k0 = sl * SW;
    const unsigned lt = (1u << lane) - 1u;
    const double gx0 = wmin(act ? pi.x : INFINITY), gy0 = wmin(act ? pi.y : INFINITY),
                 gz0 = wmin(act ? pi.z : INFINITY);
    const double gx1 = wmax(act ? pi.x : -INFINITY), gy1 = wmax(act ? pi.y : -INFINITY),
                 gz1 = wmax(act ? pi.z : -INFINITY);
    const double rmax = wmax(act ? ri : 0.0);
    const double ri2 = ri * ri;
    const int K = A.K;
    // the traversal's box test in FP32 with directed rounding: the group box
    // rounded outward, the gap between the boxes rounded down and the reach
    // rounded up, so a node is opened whenever the FP64 test would open it
    const float fgx0 = __double2float_rd(gx0), fgy0 = __double2float_rd(gy0),
                fgz0 = __double2float_rd(gz0);
    const float fgx1 = __double2float_ru(gx1), fgy1 = __double2float_ru(gy1),
                fgz1 = __double2float_ru(gz1);
    const float frmax = fmaxf(__double2float_ru(rmax), 1e-18f);
    // candidate row of particle i: entries [i K, i K + K)
    const size_t cbase = MODE != 1 ? (size_t)i * K : 0;
    int count = 0;
    double hnb = 0.0;
    int sp = 1, nflat = 0, nr = 0;
    bool overflow = false;
    if (lane == 0) S.stk[0] = root;
    __syncwarp();

    // FP32 prefilter: distances relative to the group's centre, compared
    // with the threshold widened by a margin; the candidates it passes get
    // the exact FP64 test, so the rows are the same as an FP64-only scan.
    // The relative error of the FP32 r^2 is at most about 2^-21 (2E/R + 3)
    // (E the group's half-diagonal, R the search radius: the coordinates are
    // rounded at their distance from the centre, which is at most E + R), so
    // the margin is 1e-4 plus a bound of that size: 1e-4 alone while E stays
    // below about 100 R, wider for a sparse group.
    const double cx = 0.5 * (gx0 + gx1), cy = 0.5 * (gy0 + gy1), cz = 0.5 * (gz0 + gz1);
    const double ex = 0.5 * sqrt((gx1 - gx0) * (gx1 - gx0) + (gy1 - gy0) * (gy1 - gy0) +
                                 (gz1 - gz0) * (gz1 - gz0));
    const double rsearch = MODE == 1 ? pi.w : ri;
    const float mrg = (float)(1e-4 + ldexp(2.0 * ex / fmax(rsearch, 1e-300) + 3.0, -20));
    const float2 pfx = bc2((float)(pi.x - cx)), pfy = bc2((float)(pi.y - cy)),
                 pfz = bc2((float)(pi.z - cz));
    const float2 ri2f = bc2((float)ri2 * (1.f + mrg)), hif = bc2((float)pi.w);
    // FP32 h iteration: a candidate whose FP32 distance is below the
    // threshold narrowed by the same margin is inside in FP64 too and skips
    // the FP64 test; its kernel terms use the FP32 relative coordinates and
    // are summed plainly over the chunk (at most 32 terms), then added to the
    // Kahan sums
    constexpr bool FAST = MODE == 0 && std::is_same<R, float>::value;
    const float2 ri2lo = bc2((float)ri2 * (1.f - mrg));
    const float2 m1 = bc2(-1.f), nwiden = bc2(-(1.f + mrg)), nri2f = bc2(-ri2f.x);

    // slot of the particle at offset t of the pending stream: the last range
    // starting at or before t
    auto part_slot = [&](int t) {
        int r = 0;
#pragma unroll
        for (int step = NRANGE / 2; step; step >>= 1) {
            const int c = r + step;
            if (c < nr && S.rs[c] <= t) r = c;
        }
        return S.rf[r] + (t - S.rs[r]);
    };
    // the m pending candidates from stream offset h
    auto process = [&](int m, int h) {
        if (chunks) ++*chunks;
        if (lane < m) {
            const int j = part_slot(h + lane);
            S.flat[lane] = j;
            const double4 q = A.p0[j];
            S.stage[lane] = q;
            const float qx = (float)(q.x - cx), qy = (float)(q.y - cy), qz = (float)(q.z - cz);
            S.fx[lane] = qx;
            S.fy[lane] = qy;
            S.fz[lane] = qz;
            if (FAST) {
                const float mj = (float)((const V4 *)A.p1)[j].w;
                S.fh[lane] = mj;
                S.fq[lane] = make_float4(qx, qy, qz, mj);
            } else {
                S.fh[lane] = (float)q.w;
            }
            if (MODE == 0 && !FAST) S.smass[lane] = (double)((const V4 *)A.p1)[j].w;
        } else if (SPLIT > 1 || lane < ((m + 3) & ~3)) {
            // the tail of a chunk (up to a multiple of four where one lane
            // takes them all): entries that never pass
            S.fx[lane] = S.fy[lane] = S.fz[lane] = INFINITY;
            S.fh[lane] = 0.f;
        }
        __syncwarp();
        const int m4 = (m + 3) & ~3;
        unsigned hit = 0;
        if (act) {
            // d = r^2 - lim accumulated from -lim: a set sign bit is a hit
            // (within a few ulps of the widened threshold, which lies outside
            // the true radius, a candidate may count either way); the sign
            // bits are shifted into acc one per candidate, the newest at bit 0
            unsigned acc = 0;
            auto pair = [&](float2 qx, float2 qy, float2 qz, float2 qh) {
                const float2 dx = __ffma2_rn(qx, m1, pfx);
                const float2 dy = __ffma2_rn(qy, m1, pfy);
                const float2 dz = __ffma2_rn(qz, m1, pfz);
                float2 nlim = nri2f;
                if (MODE == 1) {
                    const float2 sh = __fadd2_rn(hif, qh);
                    nlim = __fmul2_rn(__fmul2_rn(sh, sh), nwiden);
                }
                const float2 d = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, nlim)));
                acc = __funnelshift_l(__float_as_uint(d.x), acc, 1);
                acc = __funnelshift_l(__float_as_uint(d.y), acc, 1);
            };
            if (SW < 4) {
                // a candidate or two per lane
#pragma unroll
                for (int k = k0; k < k0 + SW; k++) {
                    const float dx = pfx.x - S.fx[k], dy = pfy.x - S.fy[k], dz = pfz.x - S.fz[k];
                    float nlim = nri2f.x;
                    if (MODE == 1) {
                        const float sh = hif.x + S.fh[k];
                        nlim = sh * sh * nwiden.x;
                    }
                    const float d = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, nlim)));
                    acc = __funnelshift_l(__float_as_uint(d), acc, 1);
                }
            } else if ((reinterpret_cast<uintptr_t>(S.fx) & 15u) == 0) {
                // four candidates per 128-bit shared load
#pragma unroll 2
                for (int k = SPLIT > 1 ? k0 : 0; k < (SPLIT > 1 ? k0 + SW : m4); k += 4) {
                    const float4 X = ldf4(&S.fx[k]), Y = ldf4(&S.fy[k]), Z = ldf4(&S.fz[k]);
                    const float4 H = MODE == 1 ? ldf4(&S.fh[k]) : X;
                    pair(lo2(X), lo2(Y), lo2(Z), lo2(H));
                    pair(hi2(X), hi2(Y), hi2(Z), hi2(H));
                }
            } else {
                // (a shared array placed on an 8-byte boundary only)
#pragma unroll 4
                for (int k = SPLIT > 1 ? k0 : 0; k < (SPLIT > 1 ? k0 + SW : m4); k += 2)
                    pair(ldf2(&S.fx[k]), ldf2(&S.fy[k]), ldf2(&S.fz[k]),
                         MODE == 1 ? ldf2(&S.fh[k]) : bc2(0.f));
            }
            // candidate k's sign bit is at bit m4 - 1 - k (m4 = m rounded up
            // to a multiple of four, 4..32; the padding entries never pass)
            // (SPLIT > 1: candidate k0 + q at bit q)
            const int sh = SPLIT > 1 ? 32 - SW : 32 - m4;
            hit = (__brev(acc) >> sh) & (0xffffffffu >> sh);
        }
        R cs = R(0), cd = R(0);
        auto exact_in = [&](int k) {
            const double4 pj = S.stage[k];
            const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            return dx * dx + dy * dy + dz * dz <= ri2;
        };
        if constexpr (SPLIT > 1) {
            // the lane's hits, exactly; their places in the row follow those
            // of the particle's lower lanes.  A candidate inside the FP32
            // threshold narrowed by the margin is inside in FP64 too, so the
            // long FP64 chain runs for the few near the threshold only.
            unsigned ok = 0;
            for (unsigned hh = hit; hh; hh &= hh - 1) {
                const int q = __ffs(hh) - 1, k = k0 + q;
                const float ax = pfx.x - S.fx[k], ay = pfy.x - S.fy[k], az = pfz.x - S.fz[k];
                float in2 = ri2lo.x;
                if (MODE == 1) {
                    const float sh = hif.x + S.fh[k];
                    in2 = sh * sh * (1.f - mrg);
                }
                bool in = fmaf(az, az, fmaf(ay, ay, ax * ax)) <= in2;
                if (!in) {
                    const double4 pj = S.stage[k];
                    in = MODE == 1 ? ngb_pred(pi.x, pi.y, pi.z, pi.w, pj.x, pj.y, pj.z, pj.w)
                                   : exact_in(k);
                }
                if (in) ok |= 1u << q;
            }
            const int c = __popc(ok);
            int incl = c;
#pragma unroll
            for (int o = 1; o < SPLIT; o <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, o, SPLIT);
                if (sl >= o) incl += t;
            }
            int pos = count + incl - c;
            count += __shfl_sync(FULL, incl, SPLIT - 1, SPLIT);
            for (; ok; ok &= ok - 1, pos++) {
                const int k = k0 + __ffs(ok) - 1;
                if (MODE == 1) {
                    if (pos < K) A.rows[(size_t)i * K + pos] = S.flat[k];
                    hnb = fmax(hnb, S.stage[k].w);
                } else if (pos < K) {
                    A.cidx[cbase + pos] = S.flat[k];
                }
            }
        } else if (FAST) {
            // two hits per trip (independent chains for the scheduler), the
            // sums and the row entries in the same order as one per trip
            while (hit) {
                const int k1 = __ffs(hit) - 1;
                hit &= hit - 1;
                const bool two = hit != 0;
                const int k2 = two ? __ffs(hit) - 1 : k1;
                hit &= hit - 1;
                // the prefilter's FP32 r^2, rounded the same way: below the
                // narrowed threshold the candidate is inside in FP64 too
                const float4 c1 = S.fq[k1], c2 = S.fq[k2];
                const float ax = pfx.x - c1.x, ay = pfy.x - c1.y, az = pfz.x - c1.z;
                const float bx = pfx.x - c2.x, by = pfy.x - c2.y, bz = pfz.x - c2.z;
                const float r2a = fmaf(az, az, fmaf(ay, ay, ax * ax));
                const float r2b = fmaf(bz, bz, fmaf(by, by, bx * bx));
                bool in1 = r2a <= ri2lo.x, in2 = two && r2b <= ri2lo.x;
                if (!in1) in1 = exact_in(k1);
                if (two && !in2) in2 = exact_in(k2);
                // r = r^2 rsqrt(r^2 + 1e-30): the same r for the candidates'
                // r^2 (far above 1e-30), 0 for the particle itself
                R w1, dw1, w2, dw2;
                hs->terms(r2a * rsqrtf(r2a + 1e-30f), w1, dw1);
                hs->terms(r2b * rsqrtf(r2b + 1e-30f), w2, dw2);
                if (in1) {
                    cs = fmaf(c1.w, w1, cs);
                    cd = fmaf(c1.w, dw1, cd);
                    if (count < K) A.cidx[cbase + count] = S.flat[k1];
                    count++;
                }
                if (in2) {
                    cs = fmaf(c2.w, w2, cs);
                    cd = fmaf(c2.w, dw2, cd);
                    if (count < K) A.cidx[cbase + count] = S.flat[k2];
                    count++;
                }
            }
        }
        while (SPLIT == 1 && !FAST && hit) {
            const int k = __ffs(hit) - 1;
            hit &= hit - 1;
            const double4 pj = S.stage[k];
            if (MODE != 1) {
                const double dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                if (dx * dx + dy * dy + dz * dz <= ri2) {
                    // the first Newton evaluation (at h = pi.w) rides on the
                    // search: rows are only re-read by later iterations
                    if (MODE == 0) hs->add(pair_r<R>(pi, pj), (R)S.smass[k]);
                    if (count < K) A.cidx[cbase + count] = S.flat[k];
                    count++;
                }
            } else {
                if (ngb_pred(pi.x, pi.y, pi.z, pi.w, pj.x, pj.y, pj.z, pj.w)) {
                    if (count < K) A.rows[(size_t)i * K + count] = S.flat[k];
                    count++;
                    hnb = fmax(hnb, pj.w);
                }
            }
        }
        if (FAST) {
            hs->S.add(cs);
            hs->D.add(cd);
        }
        __syncwarp();
    };

    while (sp > 0 || nflat > 0) {
        if (sp > 0) {
            const int take = min(min(sp, 32), max(1, SSTK - SRES - sp));
            sp -= take;
            int nd = 0, f = 0, cn = 0, cl = 0, cr = 0;
            bool open = false;
            if (lane < take) {
                nd = S.stk[sp + lane];
                const float4 a = A.sA[nd], b = A.sB[nd];
                const int4 L = A.wL[nd];
                f = L.x;
                cn = L.y;
                cl = L.z;
                cr = L.w;
                const float ex = fmaxf(fmaxf(__fsub_rd(a.x, fgx1), __fsub_rd(fgx0, b.x)), 0.f);
                const float ey = fmaxf(fmaxf(__fsub_rd(a.y, fgy1), __fsub_rd(fgy0, b.y)), 0.f);
                const float ez = fmaxf(fmaxf(__fsub_rd(a.z, fgz1), __fsub_rd(fgz0, b.z)), 0.f);
                const float d2 = __fmaf_rd(ez, ez, __fmaf_rd(ey, ey, __fmul_rd(ex, ex)));
                const float reach = MODE != 1 ? frmax : __fadd_ru(a.w, frmax);
                open = d2 <= __fmul_ru(__fmul_ru(reach, reach), 1.000001f);
            }
            __syncwarp();
            const bool leafy = cn <= A.leaf_size;
            const unsigned pm = __ballot_sync(FULL, open && !leafy);
            const int npush = 2 * __popc(pm);
            if (sp + npush <= SSTK) {
                if (open && !leafy) {
                    int pos = sp + 2 * __popc(pm & lt);
                    S.stk[pos] = cr;
                    S.stk[pos + 1] = cl;
                }
                sp += npush;
            } else {
                overflow = true;
            }
            const bool bucket = open && leafy;
            const unsigned lm = __ballot_sync(FULL, bucket);
            __syncwarp();
            if (lm) {
                // opened buckets join the pending stream in lane order: one
                // range per bucket at the scanned offset
                const int cnt = bucket ? cn : 0;
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                if (bucket) {
                    const int r = nr + __popc(lm & lt);
                    S.rf[r] = f;
                    S.rs[r] = nflat + incl - cnt;
                }
                nr += __popc(lm);
                nflat += __shfl_sync(FULL, incl, 31);
                __syncwarp();
                if (nflat >= 32) {
                    int h = 0;
                    do {
                        process(32, h);
                        h += 32;
                    } while (nflat - h >= 32);
                    nflat -= h;
                    // keep the ranges from the one holding offset h on, their
                    // offsets taken from h (<= 31 of them: each keeps at
                    // least one of the < 32 pending candidates)
                    int r0 = nr;
                    if (nflat > 0) {
                        r0 = 0;
#pragma unroll
                        for (int step = NRANGE / 2; step; step >>= 1) {
                            const int c = r0 + step;
                            if (c < nr && S.rs[c] <= h) r0 = c;
                        }
                    }
                    const int keep = nr - r0;
                    int vf = 0, vs = 0;
                    if (lane < keep) {
                        vf = S.rf[r0 + lane];
                        vs = S.rs[r0 + lane] - h;
                    }
                    __syncwarp();
                    if (lane < keep) {
                        S.rf[lane] = vf;
                        S.rs[lane] = vs;
                    }
                    nr = keep;
                    __syncwarp();
                }
            }
        }
        if (sp == 0 && nflat > 0) {
            process(nflat, 0);
            nflat = 0;
            nr = 0;
        }
    }
    if (MODE == 1 && SPLIT > 1)
        for (int o = SPLIT / 2; o; o >>= 1) hnb = fmax(hnb, __shfl_xor_sync(FULL, hnb, o));
    if (act && sl == 0) {
        if (MODE != 1) {
            // the full count: the Newton step shrinks the gather radius of a
            // row that did not fit instead of iterating on a truncated one
            A.cnt[i] = count;
        } else {
            A.cnt[i] = min(count, K);
            if (count > K) status_add(A.status, SPH_S_NGB_OVERFLOW, 1);
            A.hnb[i] = hnb;
        }
    }
    if (overflow && lane == 0) status_add(A.status, SPH_S_STACK_OVERFLOW, 1);
    __syncwarp();
    return count;
}

// The unit of work of a warp: 1 / SPLIT of a group, 32 / SPLIT particles with
// SPLIT lanes each.  A group's search is one long chain (tree rounds, then the
// hits of its busiest lane, chunk by chunk), so a small cloud is bound by the
// length of that chain on a few warps: with SPLIT lanes per particle the chain
// of hits is SPLIT times shorter and SPLIT times as many warps run.  The tree
// walk is repeated by each unit, so a cloud that fills the chip keeps SPLIT 1.
template <int SPLIT> struct Unit {
    int g, s0, gc, i;
    bool in;
    __device__ __forceinline__ Unit(const SearchArgs &A, int item) {
        constexpr int PW = 32 / SPLIT;
        const int part = item & (SPLIT - 1);
        g = item / SPLIT;
        s0 = A.gstart[g] + part * PW;
        gc = min(A.gcount[g] - part * PW, PW);
        const int p = (threadIdx.x & 31) / SPLIT;
        in = p < gc;
        i = in ? s0 + p : A.gstart[g];
    }
};

// exact lists for every particle
template <int SPLIT>
__global__ void __launch_bounds__(SEARCH_WARPS * 32)
    k_lists(const int *__restrict__ ngroup_p, SearchArgs A, unsigned *queue) {
    __shared__ SearchSmem smem[SEARCH_WARPS];
    const int w = threadIdx.x >> 5;
    const int nunit = *ngroup_p * SPLIT;
    if (A.only && A.listed()) return;  // k_lists_list
    for (int it = q_first(queue, blockIdx.x * SEARCH_WARPS + w); it < nunit;
         it = q_next(queue, it, gridDim.x * SEARCH_WARPS)) {
        const Unit<SPLIT> u(A, it);
        bool act = u.in;
        if (A.only && !*A.only_all) act = act && A.only[u.i];
        if (!__any_sync(FULL, act)) continue;
        const double4 pi = A.p0[u.i];
        group_search<1, double, SPLIT>(smem[w], A, A.croot[A.gcloud[u.g]], act, u.i, pi, pi.w);
    }
}

// exact lists for the listed particles (A.mlist, *A.mcount entries; nothing
// when they are too many, which k_lists covers): one warp per particle, its own box, a
// staged candidate per lane (one lane for all of them: 10k 27 us, 1M 50; here 18 and 35)
__global__ void __launch_bounds__(SEARCH_WARPS * 32)
    k_lists_list(SearchArgs A) {
    __shared__ SearchSmem smem[SEARCH_WARPS];
    const int w = threadIdx.x >> 5;
    if (!A.listed()) return;
    const int m = *A.mcount;
    for (int e = blockIdx.x * SEARCH_WARPS + w; e < m; e += gridDim.x * SEARCH_WARPS) {
        const int i = A.mlist[e];
        const double4 pi = A.p0[i];
        group_search<1, double, 32>(smem[w], A, A.croot[A.cloud[i]], true, i, pi, pi.w);
    }
}

// Exact lists from the candidate rows of the h iteration.  A pair with
// |r| <= h_i + h_j lies inside 2 max(h_i, h_j), so it sits in the candidate
// row of the particle with the larger h (2 h <= 2 hc, the radius of that
// particle's last candidate search).  The particle's LANES lanes filter its row
// with the exact predicate (same rounding as the tree search), the list in
// candidate order; where a pair's partner j did not hold i in its own row (|r|
// beyond 2 hc_j, with a margin for rounding), j's list may miss i and j is
// marked for the tree search and listed.  A row that is not a complete
// candidate set (overflow, or h above the candidate radius after the last
// round) sends every particle to the tree search.  Bound by the latency of its
// gathers, two rounds of them under way at a time (a lane per particle, 100k:
// 130 us; with 4 lanes 63).
template <int LANES>
__global__ void __launch_bounds__(256)
    k_lists_cand(int n, SearchArgs A, const double *__restrict__ hc, int *__restrict__ full,
                 int *__restrict__ full_all, int *__restrict__ full_any, int *__restrict__ mlist,
                 int *__restrict__ mcount) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(t / LANES), sl = (int)(t % LANES);
    const int lane = threadIdx.x & 31, K = A.K;
    const unsigned seg = LANES == 32 ? FULL : ((1u << LANES) - 1u) << (lane & ~(LANES - 1));
    const unsigned below = (1u << lane) - 1u;
    const bool valid = i < n;
    const double4 *__restrict__ p0 = A.p0;
    double4 pi = make_double4(0.0, 0.0, 0.0, 1.0);
    int craw = 0;
    bool whole = false;
    if (valid) {
        pi = p0[i];
        craw = A.cnt[i];
        whole = craw <= K && pi.w <= hc[i];
        if (!whole) {
            craw = 0;
            if (sl == 0) {
                *full_all = 1;
                *full_any = 1;
            }
        }
    }
    // one trip count for the warp: the ballots need every lane
    int kmax = craw;
    for (int o = 16; o; o >>= 1) kmax = max(kmax, __shfl_xor_sync(FULL, kmax, o));
    const int *crow = A.cidx + (size_t)(valid ? i : 0) * K;
    int count = 0;
    double hnb = 0.0;
    constexpr int U = 2;
    for (int k0 = 0; k0 < kmax; k0 += U * LANES) {
        int jj[U];
        double4 pj[U];
        double hj[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = k0 + u * LANES + sl;
            jj[u] = k < craw ? __ldg(&crow[k]) : -1;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            pj[u] = pi;
            hj[u] = 0.0;
            if (jj[u] >= 0) {
                pj[u] = ld_wide(p0 + jj[u]);
                hj[u] = __ldg(&hc[jj[u]]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = jj[u];
            const bool hit =
                j >= 0 && ngb_pred(pi.x, pi.y, pi.z, pi.w, pj[u].x, pj[u].y, pj[u].z, pj[u].w);
            const unsigned m = __ballot_sync(FULL, hit) & seg;
            if (hit) {
                const int pos = count + __popc(m & below);
                if (pos < K) A.rows[(size_t)i * K + pos] = j;
                hnb = fmax(hnb, pj[u].w);
                const double dx = pi.x - pj[u].x, dy = pi.y - pj[u].y, dz = pi.z - pj[u].z;
                const double rj = 2.0 * hj[u];
                if (dx * dx + dy * dy + dz * dz > rj * rj * (1.0 - 1e-9)) {
                    // j joins the list of particles to search once
                    if (atomicExch(&full[j], 1) == 0) mlist[atomicAdd(mcount, 1)] = j;
                    *full_any = 1;
                }
            }
            count += __popc(m);
        }
    }
    for (int o = LANES / 2; o; o >>= 1) hnb = fmax(hnb, __shfl_xor_sync(FULL, hnb, o));
    if (whole && sl == 0) {
        A.ngb_cnt[i] = min(count, K);
        if (count > K) status_add(A.status, SPH_S_NGB_OVERFLOW, 1);
        A.hnb[i] = hnb;
    }
}

// candidate radius 2 hc: a margin `grow` over h for the iteration, widened
// to reach h_i + 1.05 h_nb (the largest neighbour h of the last list build) so
// that the next list is complete from the particle's own candidates, at most
// to 2 (1.5 h)
__device__ __forceinline__ double cand_half_radius(double h, double hnb, double grow) {
    return fmax(h * grow, fmin(0.5 * (h + 1.05 * hnb), 1.5 * h));
}

// the smallest room a kept row must leave above h: a Newton root beyond it
// sends the particle to the search; and the reach it must keep towards the
// largest neighbour h of the last list build (times REACH), below which the
// list pass would send that neighbour to a tree search: at most REACH_CAP h,
// just below the 1.5 h that caps a search's own reach
#ifndef SPH_REUSE_ROOM
#define SPH_REUSE_ROOM 1.01
#endif
#ifndef SPH_REUSE_REACH
#define SPH_REUSE_REACH 1.01
#endif
#ifndef SPH_REUSE_REACH_CAP
#define SPH_REUSE_REACH_CAP 1.48
#endif

// the radius / 2 a kept row must still cover
__device__ __forceinline__ double reuse_need(double h, double hnb) {
    return fmax(h * SPH_REUSE_ROOM,
                fmin(0.5 * (h + SPH_REUSE_REACH * hnb), SPH_REUSE_REACH_CAP * h));
}

// Row reuse.  A search at radius 2 hsr_i listed every j within 2 hsr_i of
// particle i's position then.  Since that search i moved at most dmv_i and
// every j at most dmv_j, so the row still lists every j now within
// 2 hsr_i - dmv_i - M of i, M the largest dmv_j of the particles now that
// close: half of that is the particle's candidate radius hc without a
// search.  M = the cloud's largest dmv decides here (retry 2); where that is
// too coarse but the particle's own move leaves room (retry 3), the first
// search round bounds M by the particles of the tree nodes near its group.
// An h iteration that searches every particle (the rows dropped, reuse off,
// or the last attempt kept fewer than an eighth of the rows) restarts the
// distances moved, so the next one can keep rows again.
struct ReuseArgs {
    int on;                     // rows may be kept
    const int *rows_ok;         // device flag: the rows belong to the storage order
    const double *hsr;
    double *dmv;
    unsigned long long *dmv_max;
    const int *cloud;
    int *kept;                  // rows kept: [0] this h iteration, [1] the last attempt
                                // (INT_MAX after a full search), [2] this one attempts
};

// the kept-row counts moved on by one h iteration, and the choice of its units
// (one thread).  With 8 lanes per particle a unit is four particles; where the
// cloud has grown a dense core, the units of its rim meet hundreds of chunks of
// the core's particles (10k Evrard particles: 29 at the start, 44 after 60
// steps, 250 after 120) and the launch lasts as long as they do.  A unit of one
// particle meets a sixth of them (12, 27 and 38) but the cloud's walks are
// repeated four times.  The four h iterations of a call, us, 8 / 32 lanes:
//   10k FP64  460 / 685 at the start, 699 / 817 after 60 steps, 1552 / 1006 after 120
//   7k FP64   311 / 472, 539 / 651, 1620 / 927;  5k FP64  283 / 337, 639 / 508, 1056 / 555
// so the last iteration's longest search decides, 8 lanes up to LONG8 chunks per
// particle of an SM's share, and back below LONG32 of them.  (A load and a
// restart begin anew: launch_units_reset.  Clouds above SPLIT8_PER_SM, with 4
// lanes or fewer, have no such choice: the same was not measured there.)  (The same by a
// second launch for the particles left after the first round: 10k 1422 after 150
// steps, against 1936 without and 1092 with 32 lanes.)
__global__ void k_kept_shift(int *kept, int long8, int long32) {
    kept[1] = kept[2] ? kept[0] : INT_MAX;
    kept[0] = 0;
    kept[2] = 0;
    kept[4] = kept[3] > (kept[4] ? long32 : long8);
    kept[3] = 0;
}

__global__ void k_h_init(int n, const double *__restrict__ h, const double *__restrict__ hnb,
                         double *__restrict__ hc, int *__restrict__ retry, double grow,
                         double *__restrict__ hover, ReuseArgs U) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double hi = h[i], hn = hnb[i];
    double c = cand_half_radius(hi, hn, grow);
    int r = 1;
    const bool attempt = U.on && *U.rows_ok && U.kept[1] >= n / 8;
    if (U.kept && i == 0) U.kept[2] = attempt ? 1 : 0;
    if (attempt) {
        const double hs = U.hsr[i], own = U.dmv[i];
        const double cl = __longlong_as_double((long long)U.dmv_max[U.cloud[i]]);
        const double keep = (hs - 0.5 * (own + cl)) * (1.0 - 1e-12);
        const double need = reuse_need(hi, hn);
        if (hs > 0.0 && keep >= need) {
            c = keep;
            r = 2;
        } else if (hs > 0.0 && (hs - 0.5 * own) * (1.0 - 1e-12) >= need) {
            r = 3;
        }
    } else if (U.dmv) {
        U.dmv[i] = 0.0;
        if (i == 0 || U.cloud[i] != U.cloud[i - 1]) U.dmv_max[U.cloud[i]] = 0ull;
    }
    hc[i] = c;
    retry[i] = r;
    if (hover) hover[i] = INFINITY;
}

// per particle: the largest distance moved in its group, rounded up to FP32
// (every tree node of at most 32 particles lies inside one group); one warp
// per group
__global__ void k_group_moved(const int *__restrict__ ngroup_p, const int *__restrict__ gstart,
                              const int *__restrict__ gcount, const double *__restrict__ dmv,
                              float *__restrict__ gdm) {
    const int lane = threadIdx.x & 31;
    const int ngroup = *ngroup_p;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < ngroup; g += nw) {
        const int s0 = gstart[g], gc = gcount[g];
        double d = lane < gc ? dmv[s0 + lane] : 0.0;
        for (int o = 16; o; o >>= 1) d = fmax(d, __shfl_xor_sync(FULL, d, o));
        if (lane < gc) gdm[s0 + lane] = __double2float_ru(d);
    }
}

// The largest distance moved (gdm) over the particles of the tree nodes of
// the cloud whose boxes come within frmax of the box [fg0, fg1] (boxes as the
// search tests them, rounded outward): every particle now that close to the
// box is in one of them.  INFINITY as soon as it passes lim, or if the
// stack would overflow.
__device__ float moved_near(SearchSmem &S, const SearchArgs &A, int root, float fgx0, float fgy0,
                           float fgz0, float fgx1, float fgy1, float fgz1, float frmax, float lim,
                           const float *__restrict__ gdm) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const float reach2 = __fmul_ru(__fmul_ru(frmax, frmax), 1.000001f);
    int sp = 1;
    if (lane == 0) S.stk[0] = root;
    __syncwarp();
    float m = 0.f;
    bool bad = false;
    while (sp > 0) {
        const int take = min(sp, 32);
        sp -= take;
        int f = 0, cn = 0, cl = 0, cr = 0;
        bool open = false;
        if (lane < take) {
            const int nd = S.stk[sp + lane];
            const float4 a = A.sA[nd], b = A.sB[nd];
            const int4 L = A.wL[nd];
            f = L.x;
            cn = L.y;
            cl = L.z;
            cr = L.w;
            const float ex = fmaxf(fmaxf(__fsub_rd(a.x, fgx1), __fsub_rd(fgx0, b.x)), 0.f);
            const float ey = fmaxf(fmaxf(__fsub_rd(a.y, fgy1), __fsub_rd(fgy0, b.y)), 0.f);
            const float ez = fmaxf(fmaxf(__fsub_rd(a.z, fgz1), __fsub_rd(fgz0, b.z)), 0.f);
            const float d2 = __fmaf_rd(ez, ez, __fmaf_rd(ey, ey, __fmul_rd(ex, ex)));
            open = d2 <= reach2;
        }
        __syncwarp();
        const bool small = cn <= 32;
        if (open && small) m = fmaxf(m, gdm[f]);
        const unsigned pm = __ballot_sync(FULL, open && !small);
        const int npush = 2 * __popc(pm);
        if (sp + npush > SSTK || __any_sync(FULL, m > lim)) {
            bad = true;
            break;
        }
        if (open && !small) {
            const int pos = sp + 2 * __popc(pm & lt);
            S.stk[pos] = cr;
            S.stk[pos + 1] = cl;
        }
        sp += npush;
        __syncwarp();
    }
    __syncwarp();
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
    return bad ? INFINITY : m;
}

struct NewtonArgs {
    const void *p1;  // Real4 (v, m)
    double *h_out, *hc;
    double *hover;   // per particle: the smallest candidate radius / 2 whose row overflowed
    double *hsr;     // per particle: radius / 2 of the search that wrote the row (0: incomplete)
    const double *hnb;
    const double *dmv;  // distances moved (with hsr: the bound of a kept row)
    const float *gdm;   // per particle: its group's largest dmv, rounded up
    int *kept;       // count of the particles that kept their row (null: not counted)
    int *retry;
    int *longest;  // the most chunks a unit has gone through; [1]: a unit is one particle
    double n_ngb, tol, grow, regrow;
    int max_iter, rounds;
};

// Kernel sums of the rows of the particles of mask m (one lane each, holding
// the particle i, its trial h and its row's length c), L lanes per row over
// interleaved entries and 32 / L rows at a time, each row's sums handed to its
// particle's lane.  The whole warp calls.  One lane per row took as long as
// the row whatever the number of rows; the first Newton evaluation, which the
// search leaves, is enough for all but a few particles of a settled step.
template <class R, int L, int U>
__device__ __forceinline__ void row_sums(const SearchArgs &A, const NewtonArgs &B, unsigned m,
                                         int i, double h, int c, double &Ss, double &Ds) {
    typedef typename R4<R>::T V4;
    constexpr int NR = 32 / L;
    const int lane = threadIdx.x & 31, q = lane / L, sl = lane & (L - 1);
    while (m) {
        unsigned t = m;
        for (int x = 0; x < q; x++) t &= t - 1;
        const int src = t ? __ffs(t) - 1 : lane;
        const int ii = __shfl_sync(FULL, i, src), cc = __shfl_sync(FULL, c, src);
        const double hh = __shfl_sync(FULL, h, src);
        HSums<R> hk;
        hk.inv_h = R(1.0 / hh);
        if (t) {
            const double4 pp = A.p0[ii];
            const int *rw = A.cidx + (size_t)ii * A.K;
            // U entries per trip, their loads and their chains of arithmetic
            // side by side (an entry alone waits for two loads in turn)
            for (int k = sl; k < cc; k += U * L) {
                int j[U];
                R r[U], m[U];
#pragma unroll
                for (int x = 0; x < U; x++) j[x] = k + x * L < cc ? rw[k + x * L] : -1;
#pragma unroll
                for (int x = 0; x < U; x++) {
                    r[x] = R(0);
                    m[x] = R(0);
                    if (j[x] >= 0) {
                        r[x] = pair_r<R>(pp, A.p0[j[x]]);
                        m[x] = (R)((const V4 *)B.p1)[j[x]].w;
                    }
                }
#pragma unroll
                for (int x = 0; x < U; x++) {
                    R w, dw;
                    hk.terms(r[x], w, dw);
                    hk.S.add(m[x] * w);
                    hk.D.add(m[x] * dw);
                }
            }
        }
        const double sS = seg_sum<L>(hk.S.value()), sD = seg_sum<L>(hk.D.value());
        const int rank = __popc(m & ((1u << lane) - 1u));
        const double tS = __shfl_sync(FULL, sS, (rank * L) & 31),
                     tD = __shfl_sync(FULL, sD, (rank * L) & 31);
        if ((m >> lane & 1u) && rank < NR) {
            Ss = tS;
            Ds = tD;
        }
        for (int x = 0; x < NR; x++) m &= m - 1;
    }
}

// sums at h of the particles with want set, on every lane of the particle
template <class R, int SPLIT>
__device__ __forceinline__ void eval_rows(const SearchArgs &A, const NewtonArgs &B, bool want, int i,
                                          double h, int c, double &Ss, double &Ds) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(FULL, want && (lane & (SPLIT - 1)) == 0);
    if (!m) return;
    constexpr int U = SPLIT > 1 ? 4 : 2;
    if (SPLIT >= 8 || __popc(m) <= 4) row_sums<R, 16, U>(A, B, m, i, h, c, Ss, Ds);
    else row_sums<R, 4, U>(A, B, m, i, h, c, Ss, Ds);
    if (SPLIT > 1) {
        Ss = __shfl_sync(FULL, Ss, lane & ~(SPLIT - 1));
        Ds = __shfl_sync(FULL, Ds, lane & ~(SPLIT - 1));
    }
}

// Newton iteration of the particles of every lane with run set, FP32 or FP64
// kernel sums with FP64 update and convergence test.  The first evaluation (at
// h = pi.w), S0 and D0, comes from the search (searched) or from the kept
// row; later ones, rare once h has settled from step to step, gather the
// candidates again through the particle's slot row.  Every lane of the warp
// calls; the SPLIT lanes of a particle run the same iteration and the first
// of them writes.  pi.w and hc (the candidate radius / 2) are updated; returns
// whether the particle has to be searched again.
template <class R, int SPLIT>
__device__ __forceinline__ bool newton_rows(const SearchArgs &A, const NewtonArgs &B, bool run,
                                            int i, double4 &pi, double &hc, int craw, double S0,
                                            double D0, bool searched, bool last_round) {
    typedef typename R4<R>::T V4;
    const V4 *p1 = (const V4 *)B.p1;
    const bool own = (threadIdx.x & (SPLIT - 1)) == 0;
    bool again = false;
    bool live = run;
    if (run && searched && own) B.hsr[i] = craw > A.K ? 0.0 : hc;
    if (run && craw > A.K) {
        // more candidates inside 2 hc than the row holds: the sums would miss
        // some, so remember that radius, shrink hc towards a three-quarter
        // full row and search again; h restarts at most just below the new
        // radius
        live = false;
        if (!last_round) {
            if (own) {
                B.hover[i] = fmin(B.hover[i], hc);
                status_add(A.status, SPH_S_H_RETRY, 1);
            }
            hc = hc * fmax(0.5, cbrt(0.75 * A.K / (double)craw));
            pi.w = fmin(pi.w, hc / B.grow);
            again = true;
            if (own) {
                B.h_out[i] = pi.w;
                A.p0[i].w = pi.w;
            }
        } else if (own) {
            status_add(A.status, SPH_S_NGB_OVERFLOW, 1);
            status_add(A.status, SPH_S_H_NOCONV, 1);
        }
    }
    const bool iterated = live;
    const double mi = (double)p1[i].w;
    const double cap = hc;
    const double cfac = 4.0 * SPH_PI / 3.0 * 8.0;
    double h = pi.w, lo = 0.0, hi = INFINITY;
    bool ok = false, need = false;
    double Ssum = S0, Dsum = D0;
    for (int it = 1; it <= B.max_iter; it++) {
        if (live && h > cap) {  // 2h would pass the candidate radius 2*cap
            need = true;
            live = false;
        }
        if (!__any_sync(FULL, live)) break;
        if (SPLIT > 1 || it > 1) eval_rows<R, SPLIT>(A, B, live, i, h, craw, Ssum, Dsum);
        if (!live) continue;
        const double h3 = h * h * h;
        const double rho = SPH_SIG / h3 * Ssum;
        const double drho = -SPH_SIG / (h3 * h) * Dsum;
        const double f = cfac * h3 * rho - B.n_ngb * mi;
        const double fp = cfac * h * h * (3.0 * rho + h * drho);
        if (f < 0.0) lo = h; else hi = h;
        double hn = fp > 0.0 ? h - f / fp : -1.0;
        // a Newton step below the tolerance is accepted before any bracket
        // test: in FP64 it can round to exactly h (= a bracket end); one that
        // ends beyond the candidate radius needs the wider search first
        if (fp > 0.0 && fabs(f / fp) < B.tol * h) {
            h = hn;
            if (h > cap) need = true;
            else ok = true;
            live = false;
            continue;
        }
        // at most a factor 1.25 per iteration (keeps retries inside the rows)
        if (hn > 1.25 * h) hn = 1.25 * h;
        if (hn > 0.0 && hn < h / 1.25) hn = h / 1.25;
        if (!(hn > lo && hn < hi)) {
            if (hi == INFINITY) hn = 1.25 * h;
            else if (lo == 0.0) hn = h / 1.25;
            else hn = 0.5 * (lo + hi);
        }
        // an iterate beyond the candidate radius first tries the radius
        // itself, where the row still holds every term: only a root beyond
        // it sends the particle to another search (an overshooting Newton
        // step alone used to)
        bool clamped = false;
        if (hn > cap && h < cap) {
            hn = cap;
            clamped = true;
        }
        const double dh = hn - h;
        h = hn;
        if (!clamped && fabs(dh) < B.tol * fabs(h - dh)) {
            if (h > cap) need = true;
            else ok = true;
            live = false;
        }
    }
    if (!iterated) return again;
    if (need && !last_round) {
        // a wider search, kept below a radius whose row already overflowed;
        // a kept row that h outgrew is searched at the usual radius
        const double ov = B.hover[i];
        const double g = searched ? h * B.regrow : cand_half_radius(h, B.hnb[i], B.grow);
        hc = h < ov ? fmin(g, h + 0.5 * (ov - h)) : g;
        again = true;
    } else if (!ok && own) {
        status_add(A.status, SPH_S_H_NOCONV, 1);
    }
    pi.w = h;
    if (own) {
        if (need) status_add(A.status, SPH_S_H_RETRY, 1);
        B.h_out[i] = h;
        A.p0[i].w = h;  // p0 is written only by the lane owning particle i
    }
    return again;
}

// Candidate search + Newton iteration of each unit's particles: the first
// round for the flagged ones (retry 1) and from the kept rows (retry 2 and 3),
// then the particles whose h left their candidate radius again, at most
// `rounds` times.  A particle's rounds depend on no other particle's h, so a
// warp finishes its unit at once: a launch per round cost a pass over all
// groups and a tail of half-empty SMs each (8 rounds of 100k particles 732 us,
// here 448 with the rows re-read by four lanes; the three empty rounds of a
// 10k step 25 us).  Latency-bound: at SPLIT 1 8 blocks per SM, 64 registers,
// measured faster than 95; a split cloud fills fewer blocks and takes the
// registers for the unrolled chains instead.
template <class R, int SPLIT>
__device__ __forceinline__ void newton_units(SearchSmem &smem, int ngroup, const SearchArgs &A,
                                             const NewtonArgs &B, unsigned *queue) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nunit = ngroup * SPLIT;
    const bool own = (lane & (SPLIT - 1)) == 0;
    for (int item = q_first(queue, blockIdx.x * SEARCH_WARPS + w); item < nunit;
         item = q_next(queue, item, gridDim.x * SEARCH_WARPS)) {
        const Unit<SPLIT> u(A, item);
        const int i = u.i;
        const int rt = u.in ? B.retry[i] : 0;
        double4 pi = A.p0[i];
        // a unit keeps its rows only as a whole: a lane gathering its row
        // alone would hold up the warp's search for the others
        bool part = __any_sync(FULL, rt == 1);
        double hci = B.hc[i];
        const int root = A.croot[A.gcloud[u.g]];
        if (!part && __any_sync(FULL, rt == 3)) {
            // the moves of the particles near the unit decide: M, bounded
            // over the tree nodes within the largest kept radius of the
            // unit's box, must leave each lane's row the radius it needs
            const bool l3 = rt == 3;
            const double hs = l3 ? B.hsr[i] : 0.0, own_mv = l3 ? B.dmv[i] : 0.0;
            const double lim =
                l3 ? 2.0 * (hs - reuse_need(pi.w, B.hnb[i]) / (1.0 - 1e-12)) - own_mv : INFINITY;
            const float flim = __double2float_rd(wmin(lim));
            const float fgx0 = __double2float_rd(wmin(l3 ? pi.x : INFINITY)),
                        fgy0 = __double2float_rd(wmin(l3 ? pi.y : INFINITY)),
                        fgz0 = __double2float_rd(wmin(l3 ? pi.z : INFINITY));
            const float fgx1 = __double2float_ru(wmax(l3 ? pi.x : -INFINITY)),
                        fgy1 = __double2float_ru(wmax(l3 ? pi.y : -INFINITY)),
                        fgz1 = __double2float_ru(wmax(l3 ? pi.z : -INFINITY));
            const float frmax = __double2float_ru(wmax(2.0 * hs));
            const float M = flim >= 0.f ? moved_near(smem, A, root, fgx0, fgy0, fgz0, fgx1, fgy1,
                                                     fgz1, frmax, flim, B.gdm)
                                        : INFINITY;
            if (M <= flim) {
                if (l3) hci = (hs - 0.5 * (own_mv + (double)M)) * (1.0 - 1e-12);
            } else {
                part = true;
            }
        }
        bool act = rt == 1 || (rt >= 2 && part);
        const bool keep = rt >= 2 && !part;
        const unsigned km = __ballot_sync(FULL, keep && own);
        if (km && lane == 0 && B.kept) atomicAdd(B.kept, __popc(km));
        // searched after all, at the usual radius
        if (rt >= 2 && part) hci = cand_half_radius(pi.w, B.hnb[i], B.grow);
        int chunks = 0;
        for (int round = 0; round < B.rounds; round++) {
            const bool first_keep = km && round == 0;
            const bool any = __any_sync(FULL, act);
            if (!any && !first_keep) break;
            int craw = 0;
            double S0 = 0.0, D0 = 0.0;
            bool run = act;
            if (any) {
                if constexpr (SPLIT > 1) {
                    // the sums from the rows: a chunk leaves a few hits to a unit, so sums
                    // inside the search kept most lanes waiting (10k FP64 150 -> 137 us)
                    craw = group_search<2, R, SPLIT>(smem, A, root, act, i, pi, 2.0 * hci, nullptr,
                                                     &chunks);
                } else {
                    HSums<R> hs;
                    hs.inv_h = R(1.0 / pi.w);
                    craw = group_search<0, R, SPLIT>(smem, A, root, act, i, pi, 2.0 * hci, &hs);
                    S0 = hs.S.value();
                    D0 = hs.D.value();
                }
            } else {
                // the unit kept its rows (no lane searches)
                if (keep) craw = A.cnt[i];
                if constexpr (SPLIT == 1) eval_rows<R, SPLIT>(A, B, keep, i, pi.w, craw, S0, D0);
                run = keep;
            }
            act = newton_rows<R, SPLIT>(A, B, run, i, pi, hci, craw, S0, D0, any,
                                        round == B.rounds - 1);
            __syncwarp();
        }
        if (u.in && own && rt) {
            B.hc[i] = hci;
            B.retry[i] = 0;
        }
        if (SPLIT >= 8 && lane == 0 && chunks > B.longest[0]) atomicMax(B.longest, chunks);
        __syncwarp();
    }
}

template <class R, int SPLIT>
__global__ void __launch_bounds__(SEARCH_WARPS * 32, SPLIT > 1 ? 4 : 8)
    k_cand_newton(const int *__restrict__ ngroup_p, SearchArgs A, NewtonArgs B, unsigned *queue) {
    __shared__ SearchSmem smem[SEARCH_WARPS];
    SearchSmem &S = smem[threadIdx.x >> 5];
    if (SPLIT == 8 && B.longest[1]) newton_units<R, 32>(S, *ngroup_p, A, B, queue);
    else newton_units<R, SPLIT>(S, *ngroup_p, A, B, queue);
}

struct CountArgs {
    double *h_out, *hc;
    int *retry;
    int lo_n, hi_n, max_iter, rounds;
    double frac, grow;
};

__device__ __forceinline__ double ref_dist(const double4 &pi, const double4 &pj) {
    const double dx = xsub(pj.x, pi.x), dy = xsub(pj.y, pi.y), dz = xsub(pj.z, pi.z);
    return __dsqrt_rn(xadd(xadd(xmul(dx, dx), xmul(dy, dy)), xmul(dz, dz)));
}

// The distances of one particle's row, entry 32 e + lane in d[e] (infinity past
// the row's c <= 32 N entries, N 4 or 16): each row is gathered once, by the
// whole warp.  Most rows have 70 to 110 entries: the short form has no branch per
// entry and a quarter of the code, which otherwise waited for instructions (count
// iteration of 30k particles 248 -> 172 us, 100k 652 -> 408; k-th neighbour 50 of
// 100k 443 -> 338).
constexpr int SEL_MAX = 16, SEL_SHORT = 4;
template <int N> struct RowDist {
    double d[N];
    int c;
    __device__ __forceinline__ RowDist(const SearchArgs &A, int i, const double4 &pi, int craw)
        : c(craw) {
        const int lane = threadIdx.x & 31;
        const int *row = A.cidx + (size_t)i * A.K;
#pragma unroll
        for (int e = 0; e < N; e++) {
            d[e] = INFINITY;
            if (32 * e < c && 32 * e + lane < c) d[e] = ref_dist(pi, A.p0[row[32 * e + lane]]);
        }
    }
    // the k-th smallest distance (k = 1 the smallest), infinity when the row
    // has fewer; every distance is at most `bound`.  Bisection between 0 and the
    // bound until a trial value has k or k - 1 distances at or below it, which
    // names the k-th; equal distances never separate, so the interval also
    // shrinks by at least one bit pattern a trial (non-negative doubles order
    // like their patterns) down to the value itself.
    __device__ __forceinline__ double kth(int k, double bound) const {
        if (c < k) return INFINITY;
        unsigned long long lo = 0ull, hi = (unsigned long long)__double_as_longlong(bound);
        while (lo < hi) {
            const double a = __longlong_as_double((long long)lo), b = __longlong_as_double((long long)hi);
            unsigned long long mid = (unsigned long long)__double_as_longlong(0.5 * (a + b));
            mid = mid < lo ? lo : (mid >= hi ? hi - 1 : mid);
            const double v = __longlong_as_double((long long)mid);
            int n = 0;
            double below = 0.0, above = INFINITY;
#pragma unroll
            for (int e = 0; e < N; e++) {
                // (the few of a short row all at once: past the end at infinity)
                if (N <= SEL_SHORT || 32 * e < c) {
                    const bool in = d[e] <= v;
                    n += __popc(__ballot_sync(FULL, in));
                    if (in) below = fmax(below, d[e]);
                    else above = fmin(above, d[e]);
                }
            }
            if (n == k) return wmax(below);
            if (n == k - 1) return wmin(above);
            if (n > k) hi = mid;
            else lo = mid + 1;
        }
        return __longlong_as_double((long long)lo);
    }
};

// The reference's count iteration (h_smooth_fast_mpi, MPI_sph/sph_code/
// libsx.py:854-902) for the particle of each lane: with d_j = |r_j - r_i|
// (self included) and n(h) = #{j : d_j < 2 h}, h <- h - f h while n(h) > hi_n
// and h <- h + f h while n(h) < lo_n.  d_j is rounded as the reference writes it
// (dx = x_j - x_i, dx dx + dy dy, + dz dz, correctly rounded square root), so
// the result is bit-exact with it on the same positions.
// n(h) >= k exactly when the k-th smallest distance is below 2 h, so two order
// statistics of the row decide every iteration: t_lo, the lo_n-th distance, and
// t_hi, the (hi_n + 1)-th.  The iteration's only state is h, so a particle
// whose 2 h would pass its candidate radius 2 hc stops and resumes after a
// wider search: the sequence of h is that of one uninterrupted iteration.
// The wider radius is a guess from the row's count; `step` is the radius that h
// alone would have led to by now, B.grow past h whenever h passes it.  A guess
// whose row overflows (a clump just outside the window, a row capacity just above
// it) goes back to that, and the particle takes the small steps to the end (step
// infinite).
// Returns whether the particle has to be searched again.
__device__ __forceinline__ bool count_lane(const SearchArgs &A, const CountArgs &B, bool own,
                                           double &h, double &hc, double &step, int &it,
                                           int craw, double t_lo, double t_hi, bool last_round) {
    const double cap = hc;
    bool ok = false, done = false, again = false;
    if (craw > A.K) {
        // the row cannot hold every candidate: narrow the radius, for a row that
        // no guess has widened towards a half-full one, and search again
        hc = cap > step ? step : cap * fmax(0.5, cbrt(0.5 * A.K / (double)craw));
        step = INFINITY;
        again = true;
    } else {
        // every j with d_j < 2 lim is in the row: the search's r^2 test is
        // not rounded as d_j is, so lim keeps a margin below the radius
        const double lim = cap * (1.0 - 1e-12);
        if (h > lim) {
            // h beyond the complete radius: n(h) >= n(lim), so while n(lim)
            // is above the window every decrement is the reference's own
            if (t_hi < 2.0 * lim) {
                while (h > lim) {
                    h = xsub(h, xmul(B.frac, h));
                    if (++it > B.max_iter) {
                        done = true;
                        break;
                    }
                }
            } else {
                again = true;  // too few inside: search wider
            }
        }
        while (!done && !again && h <= lim) {
            const double h2 = 2.0 * h;
            if (t_hi < h2) {
                h = xsub(h, xmul(B.frac, h));
            } else if (!(t_lo < h2)) {
                h = xadd(h, xmul(B.frac, h));
                if (h > step * (1.0 - 1e-12)) step = h * B.grow;
            } else {
                ok = true;
                break;
            }
            if (++it > B.max_iter) done = true;
        }
        if (!ok && !done && !again) again = true;  // h passed the radius
        // the wider radius: past h, and past where a uniform density holds
        // the window's count
        if (again)
            hc = step < INFINITY
                     ? fmax(h * B.grow, cap * fmin(1.5, cbrt(1.2 * (B.hi_n + 1) / (double)max(craw, 1))))
                     : h * B.grow;
    }
    if (again && own) status_add(A.status, SPH_S_H_RETRY, 1);
    again = again && !last_round;
    if (!ok && !again && own) status_add(A.status, SPH_S_H_NOCONV, 1);
    return again;
}

// Candidate search + count iteration of each unit's particles, at most
// `rounds` searches per particle.  Each row is read once per search (RowDist);
// one lane gathering its row in every iteration took 2.3 ms for the first
// round of 30k particles and 3.7 ms in all (a launch per round), this 0.26 ms.
template <int SPLIT>
__global__ void __launch_bounds__(SEARCH_WARPS * 32, 4)
    k_cand_count(const int *__restrict__ ngroup_p, SearchArgs A, CountArgs B, unsigned *queue) {
    __shared__ SearchSmem smem[SEARCH_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nunit = *ngroup_p * SPLIT;
    const bool own = (lane & (SPLIT - 1)) == 0;
    for (int item = q_first(queue, blockIdx.x * SEARCH_WARPS + w); item < nunit;
         item = q_next(queue, item, gridDim.x * SEARCH_WARPS)) {
        const Unit<SPLIT> u(A, item);
        const double4 pi = A.p0[u.i];
        const int root = A.croot[A.gcloud[u.g]];
        double h = pi.w, hc = B.hc[u.i];
        int it = 0;
        double step = hc;
        bool act = u.in;
        for (int round = 0; round < B.rounds && __any_sync(FULL, act); round++) {
            const int craw = group_search<2, double, SPLIT>(smem[w], A, root, act, u.i, pi, 2.0 * hc);
            double t_lo = INFINITY, t_hi = INFINITY;
            for (unsigned m = __ballot_sync(FULL, act && own && craw <= A.K); m; m &= m - 1) {
                const int src = __ffs(m) - 1;
                const int ii = __shfl_sync(FULL, u.i, src), cc = __shfl_sync(FULL, craw, src);
                // every row entry lies within 2 hc up to the rounding of the
                // search's r^2 test
                const double bound = 2.0 * __shfl_sync(FULL, hc, src) * (1.0 + 1e-9);
                const auto both = [&](const auto &R) {
#pragma unroll 1
                    for (int q = 0; q < 2; q++) {
                        const double v = R.kth(q ? B.hi_n + 1 : B.lo_n, bound);
                        if ((lane & ~(SPLIT - 1)) == src) (q ? t_hi : t_lo) = v;
                    }
                };
                if (cc <= 32 * SEL_SHORT) both(RowDist<SEL_SHORT>(A, ii, A.p0[ii], cc));
                else both(RowDist<SEL_MAX>(A, ii, A.p0[ii], cc));
            }
            if (act) act = count_lane(A, B, own, h, hc, step, it, craw, t_lo, t_hi, round == B.rounds - 1);
        }
        if (u.in && own) {
            B.hc[u.i] = hc;
            B.retry[u.i] = 0;
            B.h_out[u.i] = h;
            A.p0[u.i].w = h;
        }
        __syncwarp();
    }
}

// Half the k-th smallest distance (self at index 0) of each unit's particles
// (smoothing_length_mpi, MPI_sph/sph_code/libsx.py:777-800: np.sort(dist)[50] /
// 2), rounded as the reference computes it.  With a complete row (every j with
// d_j <= 2 hc) holding at least k + 1 entries, the (k + 1)-th smallest
// distance overall is the row's.  A row with too few entries widens the
// radius, one that overflows narrows it, and the particle searches again, at
// most `rounds` times.
template <int SPLIT>
__global__ void __launch_bounds__(SEARCH_WARPS * 32, 4)
    k_cand_kth(const int *__restrict__ ngroup_p, SearchArgs A, CountArgs B, int k, unsigned *queue) {
    __shared__ SearchSmem smem[SEARCH_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nunit = *ngroup_p * SPLIT;
    const bool own = (lane & (SPLIT - 1)) == 0;
    for (int item = q_first(queue, blockIdx.x * SEARCH_WARPS + w); item < nunit;
         item = q_next(queue, item, gridDim.x * SEARCH_WARPS)) {
        const Unit<SPLIT> u(A, item);
        const double4 pi = A.p0[u.i];
        const int root = A.croot[A.gcloud[u.g]];
        double hc = B.hc[u.i];
        bool act = u.in;
        for (int round = 0; round < B.rounds && __any_sync(FULL, act); round++) {
            const int craw = group_search<2, double, SPLIT>(smem[w], A, root, act, u.i, pi, 2.0 * hc);
            double d = INFINITY;
            for (unsigned m = __ballot_sync(FULL, act && own && craw <= A.K && craw > k); m; m &= m - 1) {
                const int src = __ffs(m) - 1;
                const int ii = __shfl_sync(FULL, u.i, src), cc = __shfl_sync(FULL, craw, src);
                const double bound = 2.0 * __shfl_sync(FULL, hc, src) * (1.0 + 1e-9);
                const double v = cc <= 32 * SEL_SHORT
                                     ? RowDist<SEL_SHORT>(A, ii, A.p0[ii], cc).kth(k + 1, bound)
                                     : RowDist<SEL_MAX>(A, ii, A.p0[ii], cc).kth(k + 1, bound);
                if ((lane & ~(SPLIT - 1)) == src) d = v;
            }
            if (!act) continue;
            bool again = true;
            if (craw > A.K) {
                hc *= fmax(0.5, cbrt(0.75 * A.K / (double)craw));
            } else if (craw < k + 1) {
                hc *= craw > 0 ? fmin(2.0, fmax(1.1, cbrt(1.5 * (k + 1) / (double)craw))) : 2.0;
            } else if (d > 2.0 * hc * (1.0 - 1e-12)) {
                // at the radius itself a particle outside the row could be
                // nearer by a rounding: search again, wider
                hc *= 1.1;
            } else {
                again = false;
                if (own) {
                    B.h_out[u.i] = 0.5 * d;
                    A.p0[u.i].w = 0.5 * d;
                }
            }
            if (again && own) {
                status_add(A.status, SPH_S_H_RETRY, 1);
                if (round == B.rounds - 1) status_add(A.status, SPH_S_H_NOCONV, 1);
            }
            act = again;
        }
        if (u.in && own) {
            B.hc[u.i] = hc;
            B.retry[u.i] = 0;
        }
        __syncwarp();
    }
}

// canonical CSR export, each row sorted ascending
__global__ void k_export(int n, const int *__restrict__ rows, const int *__restrict__ cnt, int K,
                         const long long *__restrict__ off, int *__restrict__ lst) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = cnt[i];
    int *o = lst + off[i];
    for (int k = 0; k < c; k++) {
        int v = rows[(size_t)i * K + k];
        int p = k;
        while (p > 0 && o[p - 1] > v) {
            o[p] = o[p - 1];
            p--;
        }
        o[p] = v;
    }
}

SearchArgs search_args(sph_ctx *ctx, int *rows, int *cnt) {
    SearchArgs A;
    A.gstart = ctx->gstart;
    A.gcount = ctx->gcount;
    A.gcloud = ctx->groot_g;
    A.croot = ctx->croot;
    A.p0 = ctx->p0;
    A.sA = (const float4 *)ctx->node_box;
    A.sB = A.sA + 2 * (size_t)ctx->cfg.n_max;
    A.wL = ctx->wL;
    A.leaf_size = ctx->cfg.leaf_size;
    A.K = ctx->cfg.max_ngb;
    A.rows = rows;
    A.cnt = cnt;
    A.cidx = ctx->cand_idx;
    A.ngb_cnt = ctx->ngb_cnt;
    A.hnb = ctx->st[ctx->cur][ST_HNB];
    A.cloud = ctx->cloud[ctx->cur];
    A.only = nullptr;
    A.only_all = nullptr;
    A.mlist = nullptr;
    A.mcount = nullptr;
    A.mmax = 0;
    A.p1 = ctx->p1;
    A.status = ctx->status;
    return A;
}

// Lanes per particle of the searches: a cloud whose groups (about 20 particles
// each) leave warps of the chip idle splits them (see Unit).  Measured with 1 /
// 2 / 4 / 8 lanes, us, N particles of an Evrard sphere on 148 SMs:
//   h iteration, settled, FP32:  2k 122 / 73 / 59 / 46;  10k 130 / 83 / 69 / 70;
//     20k 136 / 97 / 101;  30k 150 / 113 / 123;  45k 160 / 151 / 165;
//     60k 167 / 171 / 195;  100k 202 / 263 / 309
//   the same in FP64:  10k 169 / 108 / 84 / 83;  45k 205 / 195 / 201;
//     60k 208 / 219 / 244
//   lists, tree search:  2k 64 / 56 / 44 / 34;  20k 77 / 70 / 59;
//     60k 100 / 107 / 114
//   count iteration:  2k 219 / 160 / 97 / 67;  30k 323 / 251 / 253;
//     45k 328 / 392 / 369
// and with 8 / 32 lanes (settled and evolved h iterations: k_kept_shift):
//   lists, tree search:  1k 31 / 18;  3k 33 / 23;  5k 39 / 31;  8k 42 / 40
//   count iteration:  1k 106 / 83;  3k 108 / 82;  5k 91 / 92;  8k 130 / 127
//   h iterations of a call, FP64:  1k 210 / 200;  3k 257 / 227 and 667 / 440 after
//     60 steps;  5k 283 / 337 and 639 / 508
int search_split(const sph_ctx *ctx) {
    const long long n = ctx->n, sm = ctx->num_sms;
    return n <= SPLIT32_PER_SM * sm ? 32 : n <= SPLIT8_PER_SM * sm ? 8 : n <= SPLIT4_PER_SM * sm ? 4 : n <= SPLIT2_PER_SM * sm ? 2 : 1;
}
#define SPH_SPLIT(ctx, rc, call)                                          \
    switch (search_split(ctx)) {                                          \
        case 32: { constexpr int SPLIT = 32; rc = call; break; }          \
        case 8: { constexpr int SPLIT = 8; rc = call; break; }            \
        case 4: { constexpr int SPLIT = 4; rc = call; break; }            \
        case 2: { constexpr int SPLIT = 2; rc = call; break; }            \
        default: { constexpr int SPLIT = 1; rc = call; break; }           \
    }

// one search kernel over the units of the groups on the work queue
template <class... P, class... Q>
int search_launch(sph_ctx *ctx, void (*kern)(const int *, P...), int split, Q... args) {
    // groups hold 1..32 particles, about 20 on average
    const int units = (div_up(ctx->n, 16) + ctx->ncloud) * split;
    int g;
    unsigned *q;
    int rc = queue_launch(ctx, ctx->stream, WQ_SEARCH, (const void *)kern, SEARCH_WARPS * 32,
                          max(1, div_up(units, SEARCH_WARPS)), &g, &q);
    if (rc) return rc;
    kern<<<g, SEARCH_WARPS * 32, 0, ctx->stream>>>(ctx->d_ngroup, args..., q);
    return SPH_OK;
}

}  // namespace

// margin of the step's first candidate radius over h: h may grow by this
// factor inside the first search round before the particle is searched again
#ifndef SPH_H_GROW
#define SPH_H_GROW 1.05
#endif
static const double H_GROW = SPH_H_GROW;
// the wider margin of a repeated search (a few particles per step), so that
// the step's four rounds follow a growth of h by 1.05 x 1.25^3 = 2.05
static const double H_REGROW = 1.25;
// the margin of the count and k-th iterations, whose round counts are sized
// for it
static const double H_GROW_COUNT = 1.08;

int launch_smoothing_h(sph_ctx *ctx) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    cudaStream_t s = ctx->stream;
    const int c = ctx->cur;
    // rows kept from the last h iteration when they can be: decided per
    // particle and group on the device; the host only knows whether to try
    const bool reuse = ctx->rows_host && !(ctx->cfg.flags & SPH_FLAG_NO_ROW_REUSE);
    ReuseArgs U;
    U.on = reuse ? 1 : 0;
    U.rows_ok = ctx->rows_ok;
    U.hsr = ctx->hsr;
    U.dmv = ctx->dmv;
    U.dmv_max = ctx->dmv_max;
    U.cloud = ctx->cloud[c];
    U.kept = ctx->kept_cnt;
    const double per_sm = (double)n / ctx->num_sms;
    k_kept_shift<<<1, 1, 0, s>>>(ctx->kept_cnt, (int)(LONG8 * per_sm), (int)(LONG32 * per_sm));
    ctx->kept_counted = true;
    k_h_init<<<div_up(n, 256), 256, 0, s>>>(n, ctx->st[c][ST_H], ctx->st[c][ST_HNB], ctx->hcand,
                                            ctx->retry, H_GROW, ctx->hover, U);
    if (reuse)
        k_group_moved<<<ctx->num_sms * 4, 256, 0, s>>>(ctx->d_ngroup, ctx->gstart, ctx->gcount,
                                                       ctx->dmv, ctx->gdm);
    SearchArgs A = search_args(ctx, nullptr, ctx->cand_cnt);
    NewtonArgs B;
    B.p1 = ctx->p1;
    B.h_out = ctx->st[c][ST_H];
    B.hc = ctx->hcand;
    B.hover = ctx->hover;
    B.hsr = ctx->hsr;
    B.hnb = ctx->st[c][ST_HNB];
    B.dmv = ctx->dmv;
    B.gdm = ctx->gdm;
    B.kept = ctx->kept_cnt;
    B.retry = ctx->retry;
    B.longest = ctx->kept_cnt + 3;
    B.n_ngb = ctx->cfg.n_ngb;
    B.tol = ctx->cfg.h_tol;
    B.grow = H_GROW;
    B.regrow = H_REGROW;
    B.max_iter = ctx->cfg.h_max_iter;
    B.rounds = ctx->prologue_done ? 4 : 8;
    int rc;
    if (ctx->cfg.precision == SPH_PREC_MIXED) {
        SPH_SPLIT(ctx, rc, search_launch(ctx, k_cand_newton<float, SPLIT>, SPLIT, A, B));
    } else {
        SPH_SPLIT(ctx, rc, search_launch(ctx, k_cand_newton<double, SPLIT>, SPLIT, A, B));
    }
    if (rc) return rc;
    // every row now lists the candidates of its hsr (or is marked incomplete)
    CK(cudaMemsetAsync(ctx->rows_ok, 1, sizeof(int), s));
    ctx->rows_host = true;
    ctx->lists_ok = false;
    ctx->cand_ok = true;
    return ctx_check_launch(ctx, "smoothing_h");
}

int launch_smoothing_h_count(sph_ctx *ctx, int n_target, int n_tol, double frac, int max_iter) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    cudaStream_t s = ctx->stream;
    const int c = ctx->cur;
    // these iterations write the rows without their search radii
    int rc0 = launch_rows_invalidate(ctx);
    if (rc0) return rc0;
    ctx->kept_counted = false;
    k_h_init<<<div_up(n, 256), 256, 0, s>>>(n, ctx->st[c][ST_H], ctx->st[c][ST_HNB], ctx->hcand,
                                            ctx->retry, H_GROW_COUNT, nullptr, ReuseArgs{});
    SearchArgs A = search_args(ctx, nullptr, ctx->cand_cnt);
    CountArgs B;
    B.h_out = ctx->st[c][ST_H];
    B.hc = ctx->hcand;
    B.retry = ctx->retry;
    B.lo_n = n_target - n_tol;
    B.hi_n = n_target + n_tol;
    B.max_iter = max_iter;
    B.frac = frac;
    B.grow = H_GROW_COUNT;
    // each round widens the radius by at least H_GROW_COUNT, so 16 rounds
    // cover a 3.4x change of h; one more for a guess that overflows the row
    B.rounds = 17;
    int rc;
    SPH_SPLIT(ctx, rc, search_launch(ctx, k_cand_count<SPLIT>, SPLIT, A, B));
    if (rc) return rc;
    ctx->lists_ok = false;
    ctx->cand_ok = true;
    ctx->p2_dirty = true;
    return ctx_check_launch(ctx, "smoothing_h_count");
}

// h = half the k-th neighbour distance, the search radius started from the
// current h
int launch_smoothing_kth(sph_ctx *ctx, int k) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    cudaStream_t s = ctx->stream;
    const int c = ctx->cur;
    // these iterations write the rows without their search radii
    int rc0 = launch_rows_invalidate(ctx);
    if (rc0) return rc0;
    ctx->kept_counted = false;
    k_h_init<<<div_up(n, 256), 256, 0, s>>>(n, ctx->st[c][ST_H], ctx->st[c][ST_HNB], ctx->hcand,
                                            ctx->retry, H_GROW_COUNT, nullptr, ReuseArgs{});
    SearchArgs A = search_args(ctx, nullptr, ctx->cand_cnt);
    CountArgs B{};
    B.h_out = ctx->st[c][ST_H];
    B.hc = ctx->hcand;
    B.retry = ctx->retry;
    B.grow = H_GROW_COUNT;
    B.rounds = 24;
    int rc;
    SPH_SPLIT(ctx, rc, search_launch(ctx, k_cand_kth<SPLIT>, SPLIT, A, B, k));
    if (rc) return rc;
    ctx->lists_ok = false;
    ctx->cand_ok = false;  // the rows are candidate sets of the search radius, not of h
    ctx->p2_dirty = true;
    return ctx_check_launch(ctx, "smoothing_kth");
}

// restrict a list search to the particles the pass over the rows marked.  One
// by one they cost about 1 us per 79 of them, the groups' search of 100k
// particles 277 us however few a group holds: the lines cross near a fifth.
static void marked_lists(const sph_ctx *ctx, SearchArgs &A) {
    A.only = ctx->lflag;
    A.only_all = ctx->lflag + ctx->n;
    A.mlist = ctx->mlist;
    A.mcount = ctx->lflag + ctx->n + 2;
    A.mmax = max(1024, ctx->n / 8);
}

int launch_neighbours(sph_ctx *ctx) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    cudaStream_t s = ctx->stream;
    SearchArgs A = search_args(ctx, ctx->ngb, ctx->ngb_cnt);
    if (ctx->cand_ok) {
        // lists from the candidate rows, then the tree search for the
        // particles whose rows cannot show that their list is complete
        CK(cudaMemsetAsync(ctx->lflag, 0, sizeof(int) * (n + 3), s));
        marked_lists(ctx, A);
        const int l = max(4, pass_lanes(ctx));
        auto kern = l == 4 ? k_lists_cand<4> : l == 8 ? k_lists_cand<8>
                                           : l == 16 ? k_lists_cand<16> : k_lists_cand<32>;
        kern<<<div_up((long long)n * l, 256), 256, 0, s>>>(
            n, search_args(ctx, ctx->ngb, ctx->cand_cnt), ctx->hcand, ctx->lflag, ctx->lflag + n,
            ctx->lflag + n + 1, ctx->mlist, ctx->lflag + n + 2);
    }
    // node h_max only matters to the tree search: skipped when no list needs it
    int rc = launch_refit_hmax(ctx, ctx->cand_ok ? ctx->lflag + n + 1 : nullptr);
    if (rc) return rc;
    SPH_SPLIT(ctx, rc, search_launch(ctx, k_lists<SPLIT>, SPLIT, A));
    if (rc) return rc;
    if (A.only) k_lists_list<<<ctx->num_sms * 2, SEARCH_WARPS * 32, 0, s>>>(A);
    ctx->lists_ok = true;
    ctx->rho_ok = ctx->divcurl_ok = false;
    return ctx_check_launch(ctx, "neighbours");
}

// the tree search for the particles marked in ctx->lflag (all of them when
// lflag[n] is set), after the node h_max refit (skipped when nothing is marked)
int launch_lists_marked(sph_ctx *ctx) {
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    SearchArgs A = search_args(ctx, ctx->ngb, ctx->ngb_cnt);
    marked_lists(ctx, A);
    int rc = launch_refit_hmax(ctx, ctx->lflag + n + 1);
    if (rc) return rc;
    SPH_SPLIT(ctx, rc, search_launch(ctx, k_lists<SPLIT>, SPLIT, A));
    if (rc) return rc;
    k_lists_list<<<ctx->num_sms * 2, SEARCH_WARPS * 32, 0, ctx->stream>>>(A);
    return ctx_check_launch(ctx, "lists_marked");
}

int launch_export_neighbours(sph_ctx *ctx, int64_t *off_dev, int *lst_dev, int64_t cap) {
    (void)cap;
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    k_export<<<div_up(n, 128), 128, 0, ctx->stream>>>(n, ctx->ngb, ctx->ngb_cnt, ctx->cfg.max_ngb,
                                                       (const long long *)off_dev, lst_dev);
    return ctx_check_launch(ctx, "export_neighbours");
}
