// sort.cu -- per-cloud bounding box, 63-bit Morton keys, stable LSD radix
// sort and the permutation of the particle state into key order.
//
// Replaces compute_bounding_box_kernel (bh_tree_iteration_v2.h:76-145: one
// block, a global spin lock, box accumulators started at 0) and the 10^3-cell
// counting sort CountBodies/ComputeOffset/GroupBodies (ngb_v3.h:58-117, with
// an atomicAdd-ordered, nondeterministic result).  Here the box is an exact
// FP64 min/max (order independent), keys are computed with the roundings
// spelled out so they equal the oracle's bit for bit, and the sort is stable
// so the permutation is a pure function of (keys, storage order).
#include <algorithm>
#include <cuda/atomic>

#include "sph_internal.cuh"

namespace {

constexpr int SORT_THREADS = 256, SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_PASSES = 8;  // 8-bit digits of the 63-bit key
static_assert(SORT_PASSES % 2 == 0, "the sorted keys and values end in buffer 0");

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w < v ? w : v;
    }
    return v;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// box[6*c + 0..2] = ordered min, [3..5] = ordered max; reset to (~0, 0)
__global__ void k_box_reset(unsigned long long *box, int ncloud) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 6 * ncloud) box[i] = (i % 6) < 3 ? ~0ULL : 0ULL;
}

__global__ void k_box(const double *__restrict__ x, const double *__restrict__ y,
                      const double *__restrict__ z, const int *__restrict__ cloud, int n,
                      unsigned long long *box, long long *status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool ok = i < n;
    int c = ok ? cloud[i] : -1;
    unsigned long long o[3];
    double p[3] = {ok ? x[i] : 0.0, ok ? y[i] : 0.0, ok ? z[i] : 0.0};
    bool fin = isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]);
    if (ok && !fin) status_add(status, SPH_S_NONFINITE, 1);
    for (int d = 0; d < 3; d++) o[d] = dbl_to_ord(p[d]);
    // one set of atomics per block when the whole block holds one cloud (the
    // usual case: clouds are contiguous), else per warp or per particle
    __shared__ unsigned long long smn[3][8], smx[3][8];
    __shared__ int scl[8];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned same = __match_any_sync(0xffffffffu, c);
    const bool uni = same == 0xffffffffu && c >= 0;
    if (uni) {
        for (int d = 0; d < 3; d++) {
            const unsigned long long mn = warp_min_u64(o[d]), mx = warp_max_u64(o[d]);
            if (lane == 0) {
                smn[d][w] = mn;
                smx[d][w] = mx;
            }
        }
    } else if (ok) {
        for (int d = 0; d < 3; d++) {
            atomicMin(&box[6 * c + d], o[d]);
            atomicMax(&box[6 * c + 3 + d], o[d]);
        }
    }
    if (lane == 0) scl[w] = uni ? c : -1;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (threadIdx.x == 0) {
        bool block_uni = scl[0] >= 0;
        for (int k = 1; k < nw; k++) block_uni = block_uni && scl[k] == scl[0];
        if (block_uni) {
            for (int d = 0; d < 3; d++) {
                unsigned long long mn = smn[d][0], mx = smx[d][0];
                for (int k = 1; k < nw; k++) {
                    mn = smn[d][k] < mn ? smn[d][k] : mn;
                    mx = smx[d][k] > mx ? smx[d][k] : mx;
                }
                atomicMin(&box[6 * scl[0] + d], mn);
                atomicMax(&box[6 * scl[0] + 3 + d], mx);
            }
        } else {
            for (int k = 0; k < nw; k++)
                if (scl[k] >= 0)
                    for (int d = 0; d < 3; d++) {
                        atomicMin(&box[6 * scl[k] + d], smn[d][k]);
                        atomicMax(&box[6 * scl[k] + 3 + d], smx[d][k]);
                    }
        }
    }
}

__device__ __forceinline__ unsigned long long spread3(unsigned long long v) {
    v &= 0x1fffffULL;
    v = (v | v << 32) & 0x1f00000000ffffULL;
    v = (v | v << 16) & 0x1f0000ff0000ffULL;
    v = (v | v << 8) & 0x100f00f00f00f00fULL;
    v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
    v = (v | v << 2) & 0x1249249249249249ULL;
    return v;
}

__device__ __forceinline__ unsigned long long cell_coord(double x, double lo, double ext, int bits) {
    double t = xdiv(xsub(x, lo), ext);
    double s = xmul(t, (double)(1ULL << bits));
    unsigned long long c = s <= 0.0 ? 0ULL : (unsigned long long)s;
    unsigned long long cmax = (1ULL << bits) - 1ULL;
    return c > cmax ? cmax : c;
}

// key = (cloud << 3*bits) | interleave(ix, iy, iz), x in the top bit of each
// triple; cubic cells of side ext/2^bits with ext the box's largest side
__device__ __forceinline__ unsigned long long morton_key(
    const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
    const int *__restrict__ cloud, int i, const unsigned long long *__restrict__ box, int bits) {
    int c = cloud[i];
    double lo[3], hi[3];
    for (int d = 0; d < 3; d++) {
        lo[d] = ord_to_dbl(box[6 * c + d]);
        hi[d] = ord_to_dbl(box[6 * c + 3 + d]);
    }
    double ext = fmax(xsub(hi[0], lo[0]), fmax(xsub(hi[1], lo[1]), xsub(hi[2], lo[2])));
    if (!(ext > 0.0)) ext = 1.0;
    unsigned long long ix = cell_coord(x[i], lo[0], ext, bits);
    unsigned long long iy = cell_coord(y[i], lo[1], ext, bits);
    unsigned long long iz = cell_coord(z[i], lo[2], ext, bits);
    return ((unsigned long long)c << (3 * bits)) | (spread3(ix) << 2) | (spread3(iy) << 1) |
           spread3(iz);
}

// ---- stable LSD radix sort, 8-bit digits, one launch per digit ----
// A digit's counts do not depend on the order of the keys, so k_keys counts all
// eight digits while it makes the keys (tot[pass][digit]).  A pass then reads
// each key once: its tiles take their place among equal digits of earlier
// tiles by a decoupled look-back (Merrill and Garland, 2016): every tile
// publishes its digit counts, adds up those of the tiles before it until one
// has published the sum of all up to itself, and publishes its own sum.  Tiles
// are numbered in the order in which they start, so a tile only waits for
// tiles that run or have run.  (Three launches a digit -- histogram, scan and a
// scatter of 8 rounds with five barriers each -- took 17.4 us of 10k to 100k
// particles and 28 us of 1M; one takes 4.9, 7.7 and 24.8.)
// state[tile][digit]: 0 not yet, LOCAL | count of the tile, TOTAL | count up to
// and including it.
constexpr unsigned LOCAL = 1u << 30, TOTAL = 2u << 30, VALUE = (1u << 30) - 1u;
constexpr int LOOK = 4;  // tiles read per step of the look-back (8, 16: 1 to 4 % slower)
// Polls of a thread that find nothing new before it gives up waiting and counts
// its digit among the keys of the tiles that it has not added yet: the same sum
// from the pass's input, so the permutation is right whatever the other tiles do.
constexpr int LOOK_LIMIT = 1 << 22;

__global__ void __launch_bounds__(SORT_THREADS)
    k_keys(const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
           const int *__restrict__ cloud, int n, const unsigned long long *__restrict__ box, int bits,
           unsigned long long *__restrict__ key, unsigned *__restrict__ tot) {
    __shared__ unsigned h[SORT_PASSES][256];
    for (int k = threadIdx.x; k < SORT_PASSES * 256; k += SORT_THREADS) (&h[0][0])[k] = 0u;
    __syncthreads();
    for (int i = blockIdx.x * SORT_THREADS + threadIdx.x; i < n; i += gridDim.x * SORT_THREADS) {
        const unsigned long long v = morton_key(x, y, z, cloud, i, box, bits);
        key[i] = v;
#pragma unroll
        for (int p = 0; p < SORT_PASSES; p++) atomicAdd(&h[p][(unsigned)(v >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < SORT_PASSES * 256; k += SORT_THREADS)
        if (const unsigned c = (&h[0][0])[k]) atomicAdd(&tot[k], c);
}

// exclusive sum over the block's 256 threads
__device__ __forceinline__ unsigned scan256(unsigned v, unsigned *tmp) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) tmp[w] = x;
    __syncthreads();
    unsigned before = 0;
#pragma unroll
    for (int k = 0; k < SORT_WARPS; k++) before += k < w ? tmp[k] : 0u;
    return before + x - v;
}

// One digit.  Warp w of a tile holds its elements 32 ITEMS w .., item k of lane l
// the one at 32 k + l of them, so tile, warp, item, lane is the storage order.
// EXCHANGE: the tile is put in digit order in shared memory first, so that equal
// digits leave in runs (64 bytes on average of 2048 keys) instead of one by one
template <int ITEMS, bool EXCHANGE>
__global__ void __launch_bounds__(SORT_THREADS)
    k_radix_pass(const unsigned long long *__restrict__ kin, const int *__restrict__ vin,
                 unsigned long long *__restrict__ kout, int *__restrict__ vout, int n, int shift,
                 const unsigned *__restrict__ tot, unsigned *state, unsigned *ticket, int polls,
                 long long *status) {
    __shared__ unsigned cnt[SORT_WARPS][256];  // counts, then places, per warp and digit
    __shared__ unsigned tmp[SORT_WARPS], tmp2[SORT_WARPS];
    __shared__ int stile;
    __shared__ unsigned long long xkey[EXCHANGE ? SORT_THREADS * ITEMS : 1];
    __shared__ int xval[EXCHANGE ? SORT_THREADS * ITEMS : 1];
    __shared__ unsigned to[EXCHANGE ? 256 : 1];  // from a place in the tile to the output
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    if (t == 0) stile = (int)atomicAdd(ticket, 1u);
    for (int k = t; k < SORT_WARPS * 256; k += SORT_THREADS) (&cnt[0][0])[k] = 0u;
    __syncthreads();
    const int tile = stile;
    const int base = (tile * SORT_WARPS + w) * (32 * ITEMS) + lane;
    const unsigned lt = (1u << lane) - 1u;
    unsigned long long key[ITEMS];
    unsigned place[ITEMS];
    int val[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const int idx = base + 32 * k;
        key[k] = idx < n ? kin[idx] : 0ull;
        val[k] = idx < n && vin ? vin[idx] : idx;
    }
    // place among the warp's earlier equal digits
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const bool ok = base + 32 * k < n;
        const unsigned d = (unsigned)(key[k] >> shift) & 255u;
        const unsigned peers = __match_any_sync(0xffffffffu, ok ? d : 256u);
        const unsigned before = ok ? cnt[w][d] : 0u;
        __syncwarp();
        place[k] = before + __popc(peers & lt);
        if (ok && (peers & lt) == 0) cnt[w][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // thread t owns digit t: the tile's count, the warps' places in it, and the
    // count of the tiles before
    unsigned sum = 0;
#pragma unroll
    for (int k = 0; k < SORT_WARPS; k++) {
        const unsigned c = cnt[k][t];
        cnt[k][t] = sum;
        sum += c;
    }
    cuda::atomic_ref<unsigned, cuda::thread_scope_device> mine(state[(size_t)tile * 256 + t]);
    mine.store((tile == 0 ? TOTAL : LOCAL) | sum, cuda::memory_order_relaxed);
    const unsigned start = scan256(tot[t], tmp);  // where digit t begins
    unsigned prev = 0;
    if (tile > 0) {
        int b = tile - 1, left = polls;
        bool end = false;
        while (b >= 0 && !end && left > 0) {
            // up to LOOK earlier tiles at a time
            unsigned v[LOOK];
#pragma unroll
            for (int q = 0; q < LOOK; q++)
                v[q] = b - q >= 0 ? cuda::atomic_ref<unsigned, cuda::thread_scope_device>(
                                        state[(size_t)(b - q) * 256 + t])
                                        .load(cuda::memory_order_relaxed)
                                  : (unsigned)TOTAL;
            bool stall = false;
#pragma unroll
            for (int q = 0; q < LOOK; q++) {
                if (!end && !stall) {
                    if (v[q] == 0u) {
                        stall = true;
                    } else {
                        prev += v[q] & VALUE;
                        end = (v[q] & TOTAL) != 0u;
                        b--;
                    }
                }
            }
            left -= stall;
        }
        if (b >= 0 && !end) {
            const int before = (b + 1) * SORT_THREADS * ITEMS;
            for (int k = 0; k < before; k++) prev += ((unsigned)(kin[k] >> shift) & 255u) == (unsigned)t;
            if (polls) status_add(status, SPH_S_WAIT_TIMEOUT, 1);
        }
        mine.store(TOTAL | (prev + sum), cuda::memory_order_relaxed);
    }
    const unsigned at = start + prev;
    if constexpr (EXCHANGE) {
        const unsigned in_tile = scan256(sum, tmp2);
        to[t] = at - in_tile;
#pragma unroll
        for (int k = 0; k < SORT_WARPS; k++) cnt[k][t] += in_tile;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            if (base + 32 * k < n) {
                const unsigned p = cnt[w][(unsigned)(key[k] >> shift) & 255u] + place[k];
                xkey[p] = key[k];
                xval[p] = val[k];
            }
        }
        __syncthreads();
        const int in = min(n - tile * SORT_THREADS * ITEMS, SORT_THREADS * ITEMS);
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const int p = k * SORT_THREADS + t;
            if (p < in) {
                const unsigned long long v = xkey[p];
                const unsigned pos = to[(unsigned)(v >> shift) & 255u] + (unsigned)p;
                if (pos < (unsigned)n) {
                    kout[pos] = v;
                    vout[pos] = xval[p];
                }
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < SORT_WARPS; k++) cnt[k][t] += at;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            if (base + 32 * k < n) {
                const unsigned pos = cnt[w][(unsigned)(key[k] >> shift) & 255u] + place[k];
                if (pos < (unsigned)n) {
                    kout[pos] = key[k];
                    vout[pos] = val[k];
                }
            }
        }
    }
}

// origin of each cloud's FP32 walk coordinates: the centre of its box (0
// for a cloud without a finite box)
__global__ void k_origin(const unsigned long long *__restrict__ box, int ncloud,
                         double *__restrict__ corg) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncloud) return;
    for (int d = 0; d < 3; d++) {
        const double lo = ord_to_dbl(box[6 * c + d]), hi = ord_to_dbl(box[6 * c + 3 + d]);
        corg[3 * c + d] = lo <= hi ? 0.5 * (lo + hi) : 0.0;
    }
}

struct PermTab {
    const double *src[ST_N];
    double *dst[ST_N];
};

template <class R>
__global__ void k_permute(int n, const int *__restrict__ perm, const PermTab tab, const int *__restrict__ id_in,
                          const int *__restrict__ cl_in, int *__restrict__ id_out,
                          int *__restrict__ cl_out, double4 *__restrict__ p0,
                          typename R4<R>::T *__restrict__ p1, typename R4<R>::T *__restrict__ pw,
                          const double *__restrict__ corg) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    int o = perm[s];
    double v[ST_N];
#pragma unroll
    for (int k = 0; k < ST_N; k++) v[k] = tab.src[k][o];
#pragma unroll
    for (int k = 0; k < ST_N; k++) tab.dst[k][s] = v[k];
    const int cl = cl_in[o];
    id_out[s] = id_in[o];
    cl_out[s] = cl;
    p0[s] = make_double4(v[ST_X], v[ST_Y], v[ST_Z], v[ST_H]);
    typename R4<R>::T a, b;
    a.x = (R)v[ST_VX]; a.y = (R)v[ST_VY]; a.z = (R)v[ST_VZ]; a.w = (R)v[ST_M];
    const double *org = corg + 3 * cl;
    b.x = (R)(v[ST_X] - WalkOrigin<R>::off(org, 0));
    b.y = (R)(v[ST_Y] - WalkOrigin<R>::off(org, 1));
    b.z = (R)(v[ST_Z] - WalkOrigin<R>::off(org, 2));
    b.w = (R)v[ST_M];
    p1[s] = a;
    pw[s] = b;
}

}  // namespace

// Elements per thread of a pass, by the number of particles: a cloud that would
// leave SMs without a tile takes small ones, and putting a tile in digit order
// first pays where the chip's writes and not a tile's latency bound the pass.
// us per pass with 2 / 4 / 8 elements, the last exchanging:  3k 4.0 / 4.8 / -;
// 30k 5.9 / 6.4 / -;  65k 7.1 / 7.1 / 7.7;  100k 8.7 / 7.7 / 8.1;  200k 12.6 /
// 10.9 / 9.0;  1M - / 29 / 24.8
constexpr int SORT_N2 = 50000, SORT_N4 = 130000;
static int sort_items(int n) { return n <= SORT_N2 ? 2 : n <= SORT_N4 ? 4 : 8; }
static int sort_tiles(int n) { return div_up(n, SORT_THREADS * sort_items(n)); }

// words of sort scratch for up to n particles: counts of the eight digits, a
// ticket counter and tile states per pass
size_t sort_scratch(size_t n) {
    int tiles = sort_tiles((int)n);
    if (n > SORT_N2) tiles = std::max(tiles, sort_tiles(SORT_N2));
    if (n > SORT_N4) tiles = std::max(tiles, sort_tiles(SORT_N4));
    return SORT_PASSES * 257 + (size_t)SORT_PASSES * 256 * tiles;
}

static int morton_bits_for(int ncloud) {
    int cb = 0;
    while ((1 << cb) < ncloud) cb++;
    return (63 - cb) / 3;
}

// The first phase of a refit step: the per-cloud boxes (non-finite check and
// the origin of the FP32 walk coordinates) and the packed records of the
// drifted particles, in the storage order of the last sort.
int launch_sort_refit(sph_ctx *ctx) {
    ctx->cand_ok = false;
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    cudaStream_t s = ctx->stream;
    double *const *st = ctx->st[ctx->cur];
    k_box_reset<<<div_up(6 * ctx->ncloud, 256), 256, 0, s>>>(ctx->box, ctx->ncloud);
    k_box<<<div_up(n, 256), 256, 0, s>>>(st[ST_X], st[ST_Y], st[ST_Z], ctx->cloud[ctx->cur], n,
                                         ctx->box, ctx->status);
    k_origin<<<div_up(ctx->ncloud, 128), 128, 0, s>>>(ctx->box, ctx->ncloud, ctx->corg);
    // same order: the drift is added to the distances moved
    int rc = launch_pack_p1(ctx, true);
    if (rc) return rc;
    return ctx_check_launch(ctx, "sort refit");
}

int launch_sort(sph_ctx *ctx) {
    ctx->cand_ok = false;
    ctx->topo_ok = false;  // the next tree build splits the new order
    // the candidate rows hold storage indices of the old order
    int rc0 = launch_rows_invalidate(ctx);
    if (rc0) return rc0;
    const int n = ctx->n;
    if (n <= 0) return SPH_OK;
    cudaStream_t s = ctx->stream;
    const int c = ctx->cur;
    double *const *st = ctx->st[c];
    k_box_reset<<<div_up(6 * ctx->ncloud, 256), 256, 0, s>>>(ctx->box, ctx->ncloud);
    k_box<<<div_up(n, 256), 256, 0, s>>>(st[ST_X], st[ST_Y], st[ST_Z], ctx->cloud[c], n, ctx->box,
                                         ctx->status);
    k_origin<<<div_up(ctx->ncloud, 128), 128, 0, s>>>(ctx->box, ctx->ncloud, ctx->corg);
    const int tiles = sort_tiles(n);
    unsigned *tot = ctx->hist, *ticket = tot + SORT_PASSES * 256, *state = ticket + SORT_PASSES;
    CK(cudaMemsetAsync(ctx->hist, 0,
                       sizeof(unsigned) * (SORT_PASSES * 257 + (size_t)SORT_PASSES * 256 * tiles), s));
    k_keys<<<std::min(div_up(n, SORT_THREADS), 4 * ctx->num_sms), SORT_THREADS, 0, s>>>(
        st[ST_X], st[ST_Y], st[ST_Z], ctx->cloud[c], n, ctx->box, morton_bits_for(ctx->ncloud),
        ctx->key_in, tot);
    const auto pass = sort_items(n) == 2   ? k_radix_pass<2, false>
                      : sort_items(n) == 4 ? k_radix_pass<4, false>
                                           : k_radix_pass<8, true>;
    const int polls = ctx->cfg.flags & SPH_FLAG_SORT_COUNT ? 0 : LOOK_LIMIT;
    const unsigned long long *kin = ctx->key_in;
    const int *vin = nullptr;
    for (int p = 0; p < SORT_PASSES; p++) {
        const int o = (p + 1) & 1;
        pass<<<tiles, SORT_THREADS, 0, s>>>(kin, vin, ctx->key[o], ctx->val[o], n, 8 * p, tot + 256 * p,
                                            state + (size_t)p * 256 * tiles, ticket + p, polls, ctx->status);
        kin = ctx->key[o];
        vin = ctx->val[o];
    }
    ctx->perm = ctx->val[0];
    const int d = c ^ 1;
    PermTab tab;
    for (int k = 0; k < ST_N; k++) {
        tab.src[k] = ctx->st[c][k];
        tab.dst[k] = ctx->st[d][k];
    }
    if (ctx->cfg.precision == SPH_PREC_MIXED)
        k_permute<float><<<div_up(n, 256), 256, 0, s>>>(n, ctx->perm, tab, ctx->id[c],
                                                        ctx->cloud[c], ctx->id[d], ctx->cloud[d],
                                                        ctx->p0, (float4 *)ctx->p1, (float4 *)ctx->pw,
                                                        ctx->corg);
    else
        k_permute<double><<<div_up(n, 256), 256, 0, s>>>(n, ctx->perm, tab, ctx->id[c],
                                                         ctx->cloud[c], ctx->id[d], ctx->cloud[d],
                                                         ctx->p0, (double4 *)ctx->p1,
                                                         (double4 *)ctx->pw, ctx->corg);
    ctx->cur = d;
    return ctx_check_launch(ctx, "sort");
}
