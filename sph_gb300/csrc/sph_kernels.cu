// sph_kernels.cu -- the step kernels of libsph_cuda (sm_103a).
//
// One step (fluid.c:273-348) is nine kernels on one stream, captured as a
// CUDA graph:
//
//   viscosity_predict   gravity + viscosity gather + predict + BCs + cell key   (A -> B)
//   cell_starts         exclusive scan of the cell histogram -> cell starts      (C cells)
//   scatter, permute    counting-sort scatter, then in-cell order by id          (B -> C)
//   density             density / near-density gather                           (C)
//   relax_update        relaxation gather + BCs + velocity update + cell key     (C -> B)
//   cell_starts         cell starts of the relaxed positions                     (A cells)
//   scatter, permute    back into (cell, id) order                              (B -> A)
//
// A handle holds one scene or many (an ensemble): every kernel runs over the
// particles of all scenes at once, each particle reading its own scene's
// grid and tunables from the scene table.
//
// Every pass is a gather: a thread owns one particle (in sorted order) and
// reads its 3x3 cell stencil, so no floating-point atomics exist and every
// sum is taken in a fixed order: the results are deterministic.  The only
// atomics are the integer cell-histogram increments, whose arrival rank is
// used solely to give each particle a distinct scratch slot; the final
// in-cell order is by id, recomputed deterministically in `permute`.
#include <algorithm>
#include <type_traits>
#include <utility>
#include <cstdio>

#include "sph_device.cuh"
#include "sph_learned.h"

namespace sph {
// Particles whose stencil rows have up to kShortRow candidates have their hits
// marked first and then walked, the others are gathered in one loop over the
// candidates (density_one and viscosity_cold say why; with the line at 20 to 28
// the dam break's 1,048,576 particles lost 2-8% of the viscosity pass and the
// other states stayed within 1%).
constexpr int kShortRow = 32;
// Handles of up to this many particles run the viscosity pass in the form that
// marks and walks rows of up to kMaskRow candidates: with so few warps a pass
// takes as long as its longest warp, and one of both short and long rows runs
// the walk and then the loop over the long ones.  Steps of a dam break (early)
// / a fluid at rest with rows of about 28, some above kShortRow / the same of
// 18, one form and the other: 100,000 particles 67.7 and 59.1 us / 71.1 and
// 60.0 / 43.7 and 45.4, 300,000 84.7 and 76.4 / 112 and 101 / 73.0 and 72.8,
// 500,000 95.5 and 93.8 / 150 and 141 / 102.6 and 102.5, where larger handles
// keep what compressed states of 4,194,304 particles gain by the loop.
constexpr int kFewParticles = 300000;
// Unroll factors of the candidate loops (tuned on GB300): the blocks of a
// mark-then-walk scan (hit_mask32), and the single-phase loops of the density
// and viscosity passes' long rows.
constexpr int kMarkUnroll = 8;
constexpr int kDensLongUnroll = 4;
constexpr int kViscLongUnroll = 8;
// The learned step's fallback pass: CTAs resident per SM, and how many times
// over its grid fills the GPU (it knows its particles on the device only; with
// one filling a list a little longer than the grid had threads left most of
// them idle in the second turn: 94 -> 78 us at 130,000 particles).
constexpr int kFallbackCtas = 4;
constexpr int kFallbackWaves = 2;
}  // namespace sph

namespace sph {

// ---------------------------------------------------------------------------
// block-wide helpers
// ---------------------------------------------------------------------------

template <class T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ unsigned warp_max(unsigned v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Counts one particle with cell key `key` into its build tile: the lanes of
// the warp that reach this call together and share a tile add with one
// atomic (the particles of a warp are neighbours in cell order, so almost
// every warp issues one).
__device__ __forceinline__ void add_tile_count(unsigned *tile_cnt, unsigned key)
{
    if (!tile_cnt) return;
    const unsigned active = __activemask();
    const unsigned t = key / (unsigned)kBuildTile;
    const unsigned lane = threadIdx.x & 31;
    const int first = __ffs(active) - 1;
    // nearly every warp's particles share one tile: a broadcast and a vote
    // settle it; the rest group their lanes by tile
    const unsigned t0 = __shfl_sync(active, t, first);
    if (__all_sync(active, t == t0)) {
        if (lane == (unsigned)first) atomicAdd(tile_cnt + t0, (unsigned)__popc(active));
        return;
    }
    const unsigned peers = __match_any_sync(active, t);
    if (lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(tile_cnt + t, (unsigned)__popc(peers));
}

// The same count for a whole CTA, called once by every thread of it (t: the
// build tile of the key the thread made, -1 for none): warps whose keys
// share one tile report it to thread 0, which adds runs of equal tiles with
// one atomic each.  The particles a CTA advances lie in one or two tiles,
// and the CTAs running at any moment in a narrow range of them: in a light
// kernel (the learned relaxation) one atomic per warp makes those few
// counters a hot spot, one per CTA does not.  The gathers keep the warp
// form: the barrier here would hold each CTA until its slowest warp.
__device__ __forceinline__ void cta_tile_count(unsigned *tile_cnt, int t)
{
    __shared__ int s_t[kMaxBlock / 32];
    __shared__ unsigned s_c[kMaxBlock / 32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned made = __ballot_sync(0xffffffffu, t >= 0);
    int t0 = -1;
    bool uniform = true;
    if (made) {
        t0 = __shfl_sync(0xffffffffu, t, __ffs(made) - 1);
        uniform = __all_sync(0xffffffffu, t < 0 || t == t0);
    }
    if (!uniform && t >= 0) {
        const unsigned peers = __match_any_sync(made, t);
        if (lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(tile_cnt + t, (unsigned)__popc(peers));
    }
    if (lane == 0) {
        s_t[warp] = (made && uniform) ? t0 : -1;
        s_c[warp] = (unsigned)__popc(made);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int cur = -1;
        unsigned acc = 0u;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            const int tw = s_t[w];
            if (tw < 0) continue;
            if (tw != cur) {
                if (cur >= 0) atomicAdd(tile_cnt + cur, acc);
                cur = tw;
                acc = 0u;
            }
            acc += s_c[w];
        }
        if (cur >= 0) atomicAdd(tile_cnt + cur, acc);
    }
}

// Exclusive scan over the block; returns the thread's exclusive prefix and
// the block total.  `sh` holds one word per warp.
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned *sh, unsigned &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned w = lane < nw ? sh[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) sh[lane] = w;
    }
    __syncthreads();
    total = sh[nw - 1];
    const unsigned before = warp ? sh[warp - 1] : 0u;
    __syncthreads();
    return before + x - v;
}

// ---------------------------------------------------------------------------
// cell build: histogram scan, scatter, permute
// ---------------------------------------------------------------------------

// Per-tile sums.
__global__ void __launch_bounds__(kScanThreads)
k_scan_reduce(const unsigned *__restrict__ in, int M, int *__restrict__ tile_sums)
{
    pdl_enter();
    __shared__ unsigned sh_s[kScanThreads / 32];
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    unsigned s = 0;
    if (base + kScanItems <= M) {
        const uint4 *p = reinterpret_cast<const uint4 *>(in + base);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q) {
            const uint4 t = p[q];
            s += t.x + t.y + t.z + t.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < kScanItems; ++e) s += base + e < M ? in[base + e] : 0u;
    }
    s = warp_sum(s);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh_s[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned ts = 0;
        for (int w = 0; w < kScanThreads / 32; ++w) ts += sh_s[w];
        tile_sums[blockIdx.x] = (int)ts;
    }
}

// Exclusive scan: out[i] = sum(in[0..i)), out[M] = total, which goes to
// total_out too (if any).
__global__ void __launch_bounds__(kScanThreads)
k_scan_apply(const unsigned *__restrict__ in, int M, const int *__restrict__ tile_sums,
             int *__restrict__ out, int *__restrict__ total_out)
{
    pdl_enter();
    __shared__ unsigned sh[kScanThreads / 32];
    __shared__ unsigned sh_prefix;
    // prefix of all earlier tiles
    unsigned acc = 0;
    for (int t = threadIdx.x; t < (int)blockIdx.x; t += blockDim.x) acc += (unsigned)tile_sums[t];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned p = 0;
        for (int w = 0; w < kScanThreads / 32; ++w) p += sh[w];
        sh_prefix = p;
    }
    __syncthreads();
    const unsigned prefix = sh_prefix;
    __syncthreads();

    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    unsigned v[kScanItems];
    const bool full = base + kScanItems <= M;
    if (full) {
        const uint4 *p = reinterpret_cast<const uint4 *>(in + base);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q) {
            const uint4 t = p[q];
            v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < kScanItems; ++e) v[e] = base + e < M ? in[base + e] : 0u;
    }
    unsigned local = 0;
#pragma unroll
    for (int e = 0; e < kScanItems; ++e) local += v[e];
    unsigned total;
    unsigned run = prefix + block_exclusive_scan(local, sh, total);
    if (full) {
        int4 *o = reinterpret_cast<int4 *>(out + base);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q) {
            int4 t;
            t.x = (int)run; run += v[4 * q];
            t.y = (int)run; run += v[4 * q + 1];
            t.z = (int)run; run += v[4 * q + 2];
            t.w = (int)run; run += v[4 * q + 3];
            o[q] = t;
        }
    } else {
#pragma unroll
        for (int e = 0; e < kScanItems; ++e) {
            if (base + e < M) {
                out[base + e] = (int)run;
                run += v[e];
            }
        }
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) {
        out[M] = (int)(prefix + total);
        if (total_out) *total_out = (int)(prefix + total);
    }
}

// Cell starts of a step's build in one pass over the counters: the key
// producers of a step (viscosity_predict, the relaxations) also count their
// particles per build tile (add_tile_count), so each CTA takes the prefix of
// the tiles before it from those counts, scans its own tile of counters
// into starts, zeroes the counters and gathers the occupancy statistics of
// k_scan_reduce -- with one barrier, so that a CTA's life is one round of
// loads and one of stores.  It checks its tile's total against the
// producers' count (DevState::tile_count_mismatch); the build's scatter
// zeroes the counts afterwards.
__global__ void __launch_bounds__(kBuildThreads, 1536 / kBuildThreads)
k_cell_starts(unsigned *__restrict__ in, int M, const unsigned *__restrict__ nocell,
              const unsigned *__restrict__ tile_cnt, int *__restrict__ out, DevState *st,
              unsigned *occ, int max_bucket, int max_neighbors)
{
    constexpr int ITEMS = kBuildItems, NW = ITEMS >= 32 ? ITEMS / 32 : 1;
    constexpr int WARPS = kBuildThreads / 32;
    static_assert(ITEMS % 4 == 0 && (ITEMS == 16 || ITEMS % 32 == 0), "items per thread");
    __shared__ unsigned sh_sum[WARPS], sh_pre[WARPS], sh_m[WARPS];
    __shared__ unsigned long long sh_e[WARPS], sh_o[WARPS];
    pdl_enter();
    const int tile = blockIdx.x;
    const int base = tile * kBuildTile + threadIdx.x * ITEMS;
    // prefix of all earlier tiles, from the producers' counts: the loads go
    // out together with the tile's own counters
    unsigned acc = 0;
    {
        constexpr int kBatch = 4;
        for (int t0 = 0; t0 < tile; t0 += kBatch * kBuildThreads) {
            unsigned x[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int t = t0 + j * kBuildThreads + threadIdx.x;
                x[j] = t < tile ? __ldcg(tile_cnt + t) : 0u;
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) acc += x[j];
        }
    }
    // a tile no producer counted a particle into holds only zero counters:
    // its counters are neither read nor zeroed again (most tiles of a
    // sparse scene); the others check their total against the count below
    const unsigned expect = __ldcg(tile_cnt + tile);
    unsigned v[ITEMS];
    const bool full = base + ITEMS <= M;
    if (expect == 0u) {
#pragma unroll
        for (int e = 0; e < ITEMS; ++e) v[e] = 0u;
    } else if (full) {
        const uint4 *p = reinterpret_cast<const uint4 *>(in + base);
#pragma unroll
        for (int q = 0; q < ITEMS / 4; ++q) {
            const uint4 t = p[q];
            v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < ITEMS; ++e) v[e] = base + e < M ? in[base + e] : 0u;
    }
    // the thread's counters in the no-cell bitmap
    unsigned bits[NW];
#pragma unroll
    for (int j = 0; j < NW; ++j)
        bits[j] = (nocell && base + 32 * j < M) ? __ldg(nocell + (base >> 5) + j) : 0u;
    if (ITEMS < 32) bits[0] >>= (base & 31);
    unsigned local = 0, mx = 0;
    unsigned long long excess = 0, outside = 0;
#pragma unroll
    for (int e = 0; e < ITEMS; ++e) {
        local += v[e];
        if ((bits[e >> 5] >> (e & 31)) & 1u) {
            outside += v[e];
        } else {
            mx = max(mx, v[e]);
            if (v[e] > (unsigned)max_bucket) excess += v[e] - max_bucket;
        }
    }
    // warp-level: inclusive scan of the thread sums, reductions of the rest
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned x = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    acc = warp_sum(acc);
    mx = warp_max(mx);
    excess = warp_sum(excess);
    outside = warp_sum(outside);
    if (lane == 31) sh_sum[warp] = x;
    if (lane == 0) { sh_pre[warp] = acc; sh_m[warp] = mx; sh_e[warp] = excess; sh_o[warp] = outside; }
    __syncthreads();
    // every thread combines the per-warp words itself (no second barrier)
    unsigned before = 0, total = 0, prefix = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
        const unsigned sw = sh_sum[w];
        before += w < warp ? sw : 0u;
        total += sw;
        prefix += sh_pre[w];
    }
    unsigned run = prefix + before + x - local;
    if (full) {
        int4 *o = reinterpret_cast<int4 *>(out + base);
        uint4 *z = reinterpret_cast<uint4 *>(in + base);
#pragma unroll
        for (int q = 0; q < ITEMS / 4; ++q) {
            int4 t;
            t.x = (int)run; run += v[4 * q];
            t.y = (int)run; run += v[4 * q + 1];
            t.z = (int)run; run += v[4 * q + 2];
            t.w = (int)run; run += v[4 * q + 3];
            o[q] = t;
            if (expect != 0u) z[q] = make_uint4(0, 0, 0, 0);
        }
    } else {
#pragma unroll
        for (int e = 0; e < ITEMS; ++e) {
            if (base + e < M) {
                out[base + e] = (int)run;
                run += v[e];
                if (expect != 0u) in[base + e] = 0u;
            }
        }
    }
    if (tile == (int)gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[M] = (int)(prefix + total);
    if (threadIdx.x == 0) {
        if (total != expect) atomicOr(&st->tile_count_mismatch, 1u);
        if (occ) {
            unsigned tm = 0;
            unsigned long long te = 0, to = 0;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                tm = max(tm, sh_m[w]); te += sh_e[w]; to += sh_o[w];
            }
            atomicMax(occ, tm);
            atomicMax(&st->max_occ, tm);
            if (te) atomicAdd(&st->bucket_overflow, te);
            if (to) atomicAdd(&st->out_of_grid, to);
            const unsigned m = tm < (unsigned)max_bucket ? tm : (unsigned)max_bucket;
            if (m > 0 && 5u * m - 1u > (unsigned)max_neighbors) atomicOr(&st->list_cap_risk, 1u);
        }
    }
}

// Scatter and permutation of a build.  The scatter puts each particle's id
// into its scratch slot (cell start + arrival rank); the permutation's slot is
// the cell start + the number of cell members with a smaller id, so that each
// cell holds its particles in id order -- the order hash.c:153-163 inserts
// them into a bucket (pointer-array order).  K particles per thread (strided
// by the block size, so the loads stay coalesced), their loads issued
// together, so that each thread has K dependent chains (key -> cell start ->
// slot) in flight instead of one.
//
// What a kernel reads of kernels before its predecessor it requests ahead of
// the wait for the predecessor (their results are complete: the predecessor
// waited for them before this kernel could start), past L1 (ld.cg), so that
// its first loads overlap the predecessor's tail.
template <int K>
__global__ void __launch_bounds__(kBlock)
k_scatter_ids_x(int n, const uint2 *__restrict__ kr, const int *__restrict__ id_src,
                const int *__restrict__ start, int *__restrict__ tmp, unsigned *tile_cnt,
                int ntiles)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int i0 = blockIdx.x * blockDim.x * K + threadIdx.x;
    uint2 k[K];
    int id[K], st[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int i = i0 + j * blockDim.x;
        if (i < n) {
            k[j] = __ldcg(kr + i);
            id[j] = id_src ? __ldcg(id_src + i) : i;
        }
    }
    pdl_enter();
    // the build's tile counts have been read (k_cell_starts): zero them for
    // the next build
    for (int t = g; t < ntiles; t += gridDim.x * blockDim.x) tile_cnt[t] = 0u;
#pragma unroll
    for (int j = 0; j < K; ++j)
        if (i0 + j * (int)blockDim.x < n) st[j] = __ldg(start + k[j].x);
#pragma unroll
    for (int j = 0; j < K; ++j) {
        if (i0 + j * (int)blockDim.x >= n) continue;
        const int d = st[j] + (int)k[j].y;
        if (in_bounds(d, n, kBadScatter)) tmp[d] = id[j];
    }
}

template <int K>
__global__ void __launch_bounds__(kBlock)
k_permute_x(int n, const uint2 *__restrict__ kr, const int *__restrict__ start,
            const int *__restrict__ tmp, const int *__restrict__ id_src,
            const float2 *__restrict__ a_src, const float2 *__restrict__ b_src,
            int *__restrict__ id_dst, float2 *__restrict__ a_dst, float2 *__restrict__ b_dst,
            DevState *__restrict__ end_step)
{
    const int i0 = blockIdx.x * blockDim.x * K + threadIdx.x;
    uint2 k[K];
    int id[K], s0[K], s1[K];
    float2 a[K], b[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int i = i0 + j * blockDim.x;
        if (i < n) {
            k[j] = __ldcg(kr + i);
            id[j] = id_src ? __ldcg(id_src + i) : i;
            a[j] = __ldcg(a_src + i);
            if (b_src) b[j] = __ldcg(b_src + i);
        }
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
        if (i0 + j * (int)blockDim.x < n) {
            s0[j] = __ldcg(start + k[j].x);
            s1[j] = __ldcg(start + k[j].x + 1);
        }
    pdl_enter();
    if (end_step && blockIdx.x == 0 && threadIdx.x == 0) {
        // last kernel of a step: the neighbour relation of the new positions
        // now exists (viscosity is on from the next step), one more step done
        end_step->lists_valid = 1u;
        end_step->steps += 1ull;
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        if (i0 + j * (int)blockDim.x >= n) continue;
        int r;
        if (s1[j] - s0[j] <= kRankScanMax) {
            r = 0;
            for (int q = s0[j]; q < s1[j]; ++q)
                if (in_bounds(q, n, kBadScatter)) r += __ldg(tmp + q) < id[j];
        } else {
            r = (int)k[j].y;  // pathological cell: arrival order
        }
        const int d = s0[j] + r;
        if (!in_bounds(d, n, kBadScatter)) continue;
        id_dst[d] = id[j];
        a_dst[d] = a[j];
        if (b_src) b_dst[d] = b[j];
    }
}

// ---------------------------------------------------------------------------
// pass 1: gravity + viscosity (gather) + predict + boundary + cell key
// ---------------------------------------------------------------------------

// What the viscosity pass reads and writes.
struct ViscArrays {
    Ctx c;
    const DevState *st;
    const float2 *pos, *vel;
    const int *start;
    const unsigned *occ_in;  // the build's largest cell population
    float2 *pos_out, *prev_out;
    uint2 *kr_out;
    unsigned *cnt;
    float2 *probe_out;
};

// The end of a particle's viscosity pass: gravity and the impulses' sum dv on
// its velocity v0, predict_positions with boundaryConditions, and the
// predicted position's cell key counted into its build.
template <bool PROBE>
__device__ __forceinline__ void viscosity_finish(int i, const ViscArrays &A, const Scene *S,
                                                 const SG &g, float2 p, float2 v0, float2 dv)
{
    if (PROBE) {
        A.probe_out[i] = dv;
        return;
    }
    const float dt = __ldg(&S->P.time_step);
    const float gdt = __fmul_rn(-__ldg(&S->P.g), dt);
    const float vx = __fadd_rn(v0.x, dv.x);
    const float vy = __fadd_rn(__fadd_rn(v0.y, gdt), dv.y);
    float nx = __fadd_rn(p.x, __fmul_rn(vx, dt));
    float ny = __fadd_rn(p.y, __fmul_rn(vy, dt));
    boundary_of(nx, ny, S);
    const unsigned k2 = cell_key(nx, ny, g);
    unsigned rank = 0u;
    if (in_bounds(k2, A.c.M, kBadKey)) {
        rank = atomicAdd(A.cnt + k2, 1u);
        add_tile_count(A.c.tile_cnt, k2);
    }
    A.pos_out[i] = make_float2(nx, ny);
    A.prev_out[i] = p;
    A.kr_out[i] = make_uint2(k2, rank);
}

// The scene constants of a pair's viscosity impulse, and the impulse itself.
struct ViscConsts {
    float h2, dt, dt_h, sigma, beta;
};

__device__ __forceinline__ ViscConsts visc_consts(const Scene *S)
{
    ViscConsts c;
    c.dt = __ldg(&S->P.time_step);
    const float hh = __ldg(&S->P.smoothing_radius);
    c.h2 = __fmul_rn(hh, hh);
    c.dt_h = c.dt * __fdiv_rn(1.0f, hh);
    c.sigma = __ldg(&S->P.sigma);
    c.beta = __ldg(&S->P.beta);
    return c;
}

// One neighbour's impulse on the particle at -mp with velocity v0, added to
// dv; d = (position, velocity), r2 <= h2 known, velocities before gravity
// (which adds the same amount to both).  Self (and any coincident particle)
// has r2 == 0 and gives none, as u is NaN in the reference for r == 0
// (fluid.c:446-451).
__device__ __forceinline__ void visc_impulse(const ViscConsts &c, float2 e, float r2, float2 v0,
                                             float2 dvel, float2 &dv)
{
    float r_recip = rsqrt_normal(r2);
    if (r2 < kMinNormal) {
        if (r2 == 0.0f) return;
        r_recip = rsqrtf(r2);
    }
    const float r = r2 * r_recip;
    const float2 w = __fadd2_rn(v0, make_float2(-dvel.x, -dvel.y));
    const float u0 = __fmaf_rn(w.x, e.x, __fmul_rn(w.y, e.y)) * r_recip;
    // only approaching pairs (u > 0) push; the others run the same
    // instructions with u = 0, whose impulse is +-0 and leaves dv's bits
    // as they are (no divergent branch: about half the pairs of every
    // warp approach)
    const float u = fmaxf(u0, 0.0f);  // 0 for a NaN
    // dt (1 - r/h) (sigma u + beta u^2) = (dt - (dt/h) r) u (sigma + beta u)
    const float imp = fmaf(-c.dt_h, r, c.dt) * u * fmaf(c.beta, u, c.sigma);
    // per component imp * q * r_recip, clamped, halved and subtracted
    // (packed FP32x2, each operation rounded as the scalar form)
    const float2 t = __fmul2_rn(__fmul2_rn(make_float2(imp, imp), e),
                                make_float2(r_recip, r_recip));
    dv = __ffma2_rn(make_float2(-0.5f, -0.5f), make_float2(clamp5(t.x), clamp5(t.y)), dv);
}

// The sum of a particle with a stencil row of more than kShortRow candidates,
// or with an overflowing bucket somewhere, in one loop over the candidates:
// the lanes of a warp are then mostly of one cell and read the same candidate
// at a time, which a walk over each lane's own hits does not (the dam break's
// 1,048,576 particles, compressed: all rows marked and walked 218 us, this 187
// us; 64 compressed scenes 231 and 217 us).  Out of line and to the end of
// the particle's pass: nothing of the short rows' walk lives across the call.
template <bool PROBE>
__device__ __noinline__ void viscosity_cold(int i, const ViscArrays &A)
{
    const Scene *S = A.c.scenes + scene_of(A.c, i);
    const float2 *pos = A.pos, *vel = A.vel;
    const bool capped = *A.occ_in > (unsigned)A.c.max_bucket;
    const int n = A.c.n;
    const SG g = load_grid(S);
    const ViscConsts vc = visc_consts(S);
    const float2 p = __ldg(pos + i), v0 = __ldg(vel + i);
    const float2 mp = make_float2(-p.x, -p.y);
    const unsigned key = cell_key(p.x, p.y, g);
    float2 dv = make_float2(0.0f, 0.0f);
    if (capped) {
        for_each_candidate(key, A.start, g, true, A.c.max_bucket, n, [&](int j) {
            const float2 q = __ldg(pos + j);
            float2 e;
            const float r2 = dist2_packed(mp, q, e);
            if (!(r2 > vc.h2)) visc_impulse(vc, e, r2, v0, __ldg(vel + j), dv);
        });
        viscosity_finish<PROBE>(i, A, S, g, p, v0, dv);
        return;
    }
    auto one = [&](int j) {
        const float2 q = __ldg(pos + j), w = __ldg(vel + j);
        float2 e;
        const float r2 = dist2_packed(mp, q, e);
        if (r2 <= vc.h2) visc_impulse(vc, e, r2, v0, w, dv);
    };
    int ra[3], rl[3];
    stencil_rows(p, key, A.start, g, ra, rl, n);
#pragma unroll 1
    for (int r = 0; r < 3; ++r) {
        const int a = ra[r], l = rl[r];
#pragma unroll kViscLongUnroll
        for (int j = a; j < a + l; ++j) one(j);
    }
    viscosity_finish<PROBE>(i, A, S, g, p, v0, dv);
}

// apply_gravity (fluid.c:398-413), viscosity_impluses (fluid.c:416-478) in
// gather form, predict_positions (fluid.c:507-523) with boundaryConditions.
// Gather form of the viscosity: dv_i = -1/2 sum_j clamp5(I_ij),
// I_ij = dt (1 - r/h)(sigma u + beta u^2) (x_j - x_i)/r for u > 0,
// u = ((v_i - v_j).(x_j - x_i))/r, all from the velocities after gravity.
// PROBE writes dv instead of advancing.
// FEW (kFewParticles): rows of up to kMaskRow candidates are marked and walked,
// except in a warp that has a longer one and takes the loop for it anyway.
template <bool PROBE, bool FEW>
__device__ __forceinline__ void viscosity_predict_one(int i, const ViscArrays &A)
{
    const Scene *S = A.c.scenes + scene_of(A.c, i);
    const SG g = load_grid(S);
    const float2 *pos = A.pos, *vel = A.vel;
    const bool capped = *A.occ_in > (unsigned)A.c.max_bucket;
    const float2 p = pos[i];
    const float2 v0 = vel[i];  // before gravity
    float2 dv = make_float2(0.0f, 0.0f);
    const unsigned key = cell_key(p.x, p.y, g);
    if ((PROBE || A.st->lists_valid) && searchable(key, i, A.start, g, capped, A.c.max_bucket)) {
        int ra[3] = {0, 0, 0}, rl[3] = {0, 0, 0};
        if (!capped) stencil_rows(p, key, A.start, g, ra, rl, A.c.n);
        const int longest = max(rl[0], max(rl[1], rl[2]));
        int marked = kShortRow;
        if (FEW && !__any_sync(__activemask(), longest > kMaskRow)) marked = kMaskRow;
        if (!capped && longest <= marked) {
            // two phases: a cheap scan marks the neighbours of the stencil
            // rows, then only they pay for the impulse (less SIMT waste)
            const ViscConsts vc = visc_consts(S);
            const float2 mp = make_float2(-p.x, -p.y);
            auto load = [&](int j) {
                const float2 q = __ldg(pos + j), w = __ldg(vel + j);
                return make_float4(q.x, q.y, w.x, w.y);
            };
            auto visit = [&](int, const float4 &d) {
                float2 e;
                const float r2 = dist2_packed(mp, make_float2(d.x, d.y), e);
                visc_impulse(vc, e, r2, v0, make_float2(d.z, d.w), dv);
            };
            if (FEW) {
                unsigned long long m[3];
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const float2 *row = pos + ra[r];
                    const unsigned lo = hit_mask32<kMarkUnroll>(row, min(rl[r], 32), mp, vc.h2);
                    const unsigned hi = hit_mask32<kMarkUnroll>(row + 32, max(rl[r] - 32, 0), mp, vc.h2);
                    m[r] = (unsigned long long)hi << 32 | lo;
                }
                m[1] &= ~(1ull << (i - ra[1]));  // not the particle itself
                walk_rows<float4>(m, ra, A.c.n, load, visit);
            } else {
                const unsigned b0 = hit_mask32<kMarkUnroll>(pos + ra[0], rl[0], mp, vc.h2);
                const unsigned b1 = hit_mask32<kMarkUnroll>(pos + ra[1], rl[1], mp, vc.h2) &
                                    ~(1u << (i - ra[1]));  // not the particle itself
                const unsigned b2 = hit_mask32<kMarkUnroll>(pos + ra[2], rl[2], mp, vc.h2);
                walk_three<float4>(b0, ra[0], b1, ra[1], b2, ra[2], A.c.n, load, visit);
            }
        } else {
            viscosity_cold<PROBE>(i, A);
            return;
        }
    }
    viscosity_finish<PROBE>(i, A, S, g, p, v0, dv);
}

// 40 registers (48 resident warps per SM): 4,194,304 particles 189 -> 184 us
// early in the dam break and 237 -> 230 us compressed against 48 registers,
// 200 and 253 with 56.
template <bool PROBE, bool PERSIST, bool FEW>
__device__ __forceinline__ void viscosity_predict(const ViscArrays &A, unsigned *occ_reset)
{
    pdl_enter();
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (!PROBE && i0 == 0) *occ_reset = 0u;
    for (int i = i0; i < A.c.n; i += gridDim.x * blockDim.x) {
        viscosity_predict_one<PROBE, FEW>(i, A);
        if (!PERSIST) break;
    }
}

template <bool PROBE, bool PERSIST = false>
__global__ void __maxnreg__(40)
k_viscosity_predict(const __grid_constant__ ViscArrays A, unsigned *occ_reset)
{
    viscosity_predict<PROBE, PERSIST, false>(A, occ_reset);
}

// 48 registers: no spills (40 and 64 take the same time, within 2%).
template <bool PROBE, bool PERSIST = false>
__global__ void __maxnreg__(48)
k_viscosity_predict_few(const __grid_constant__ ViscArrays A, unsigned *occ_reset)
{
    viscosity_predict<PROBE, PERSIST, true>(A, occ_reset);
}

// ---------------------------------------------------------------------------
// pass 2: density and near density (gather)
// ---------------------------------------------------------------------------

// rho_i = sum_j (1 - r/h)^2, rho_near_i = sum_j (1 - r/h)^3 over neighbours
// j != i with r/h < 1 (calculate_density, fluid.c:527-539; the pairs of
// hash_fluid, hash.c:185/221: r2 <= h2 inclusive).
// Writes xr = (x, y, rho, rho_near) and, per stencil row, the bit mask of the
// candidates that are neighbours (r2 <= h2, self excluded), which the
// relaxation pass of the same positions walks instead of the whole stencil.
// Where a density pass by itself puts its results: by particle id.
struct DensityById {
    const int *ids = nullptr;
    float *rho = nullptr, *rho_near = nullptr;
    __device__ __forceinline__ void put(int i, float2 ab) const
    {
        const int id = __ldg(ids + i);
        rho[id] = ab.x;
        rho_near[id] = ab.y;
    }
};

// What a density pass reads and writes: the densities alone to by_id, or the
// records, masks and rows.
struct DensArrays {
    Ctx c;
    const float2 *pos;
    const int *start;
    const unsigned *occ_in;  // the build's largest cell population
    float4 *xr_out;
    ulonglong2 *mask01;
    unsigned long long *mask2;
    int4 *rows_out;
    DensityById by_id;
};

template <bool BY_ID>
__device__ __forceinline__ void density_finish(int i, const DensArrays &A, float2 p, float2 ab,
                                               unsigned long long m0, unsigned long long m1,
                                               unsigned long long m2, int4 rec)
{
    if (BY_ID) {
        A.by_id.put(i, ab);
        return;
    }
    A.xr_out[i] = make_float4(p.x, p.y, ab.x, ab.y);
    A.mask01[i] = make_ulonglong2(m0, m1);
    A.mask2[i] = m2;
    A.rows_out[i] = rec;
}

// A particle with a stencil row of more than kShortRow candidates, or with an
// overflowing bucket somewhere, in one loop over the candidates: the lanes of
// a warp are then mostly of one cell and read the same candidate at a time,
// which a walk over each lane's own hits does not.  The candidates come in
// blocks without a remainder (as hit_mask32; four at a time 135 us early in the
// dam break of 4,194,304 particles, with a remainder loop 141).  To the end of
// the particle's pass, so that the short rows' walk shares no values with it;
// out of line it was 5-10% slower in compressed states.
// LM: long-row masks (rows of up to 2 kMaskRow candidates recorded as
// kRowsMasked2, the hit bits of their candidates kMaskRow.. in c.maskx).
template <bool LM, bool BY_ID>
__device__ __forceinline__ void density_long_rows(int i, const DensArrays &A)
{
    const Ctx &c = A.c;
    const Scene *S = c.scenes + scene_of(c, i);
    const SG g = load_grid(S);
    const float hh = __ldg(&S->P.smoothing_radius);
    const float h2 = __fmul_rn(hh, hh);
    const float h_recip = __fdiv_rn(1.0f, hh);
    const float2 *pos = A.pos;
    const float2 p = __ldg(pos + i), mp = make_float2(-p.x, -p.y);
    const unsigned key = cell_key(p.x, p.y, g);
    const bool capped = *A.occ_in > (unsigned)c.max_bucket;
    float2 ab = make_float2(0.0f, 0.0f);  // (rho, rho_near)
    unsigned long long m[3] = {0ull, 0ull, 0ull};
    int4 rec = make_int4(0, 0, 0, kRowsNone);
    if (searchable(key, i, A.start, g, capped, c.max_bucket)) {
        rec.w = kRowsFull;
        if (!capped) {
            int ra[3], rl[3];
            stencil_rows(p, key, A.start, g, ra, rl, c.n);
            unsigned long long *mx = nullptr;
            if (rl[0] <= kMaskRow && rl[1] <= kMaskRow && rl[2] <= kMaskRow) {
                rec = make_int4(ra[0], ra[1], ra[2], kRowsMasked);
            } else if (LM && c.maskx && rl[0] <= 2 * kMaskRow && rl[1] <= 2 * kMaskRow &&
                       rl[2] <= 2 * kMaskRow) {
                rec = make_int4(ra[0], ra[1], ra[2], kRowsMasked2);
                mx = c.maskx + 3 * (size_t)i;
                mx[0] = mx[1] = mx[2] = 0ull;  // rows of kMaskRow or fewer leave theirs
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int len = rl[r];
                const float2 *row = pos + ra[r];
                const int self = r == 1 ? i - ra[1] : -1;
                unsigned long long w0 = 0ull, w1 = 0ull;
#pragma unroll 1
                for (int c0 = 0; c0 < len; c0 += kDensLongUnroll) {
                    float2 q[kDensLongUnroll];
#pragma unroll
                    for (int k = 0; k < kDensLongUnroll; ++k) q[k] = __ldg(row + c0 + k);
                    unsigned b = 0u;
#pragma unroll
                    for (int k = 0; k < kDensLongUnroll; ++k) {
                        float2 e;
                        const float r2 = dist2_packed(mp, q[k], e);
                        if (r2 <= h2 && c0 + k < len && c0 + k != self) {
                            b |= 1u << k;
                            add_density(ab, r2, h_recip);
                        }
                    }
                    if (c0 < kMaskRow) w0 |= (unsigned long long)b << c0;
                    else if (c0 < 2 * kMaskRow) w1 |= (unsigned long long)b << (c0 - kMaskRow);
                }
                m[r] = w0;
                if (LM && mx != nullptr && len > kMaskRow) mx[r] = w1;
            }
        } else {
            for_each_candidate(key, A.start, g, true, c.max_bucket, c.n, [&](int j) {
                if (j == i) return;
                const float2 q = __ldg(pos + j);
                const float r2 = dist2(p.x - q.x, p.y - q.y);
                if (r2 > h2) return;
                add_density(ab, r2, h_recip);
            });
        }
    }
    density_finish<BY_ID>(i, A, p, ab, m[0], m[1], m[2], rec);
}

// Particles whose rows have up to kShortRow candidates have their hits marked
// first and the marked ones walked: the terms are run for the hits alone,
// where one loop over the candidates runs them for nearly every candidate of a
// warp (some lane hits).  4,194,304 particles: one loop for every row 182 us
// early in the dam break and 201 us compressed, this 135 and 172 us; two
// phases for rows of any length 162 and 197 us.
template <bool LM = false, bool BY_ID = false>
__device__ __forceinline__ void density_one(int i, const DensArrays &A)
{
    const Scene *S = A.c.scenes + scene_of(A.c, i);
    const SG g = load_grid(S);
    const float2 *pos = A.pos;
    const float2 p = pos[i];
    const unsigned key = cell_key(p.x, p.y, g);
    const bool capped = *A.occ_in > (unsigned)A.c.max_bucket;
    int ra[3] = {0, 0, 0}, rl[3] = {0, 0, 0};
    int4 rec = make_int4(0, 0, 0, kRowsNone);
    if (!capped && searchable(key, i, A.start, g, false, A.c.max_bucket)) {
        stencil_rows(p, key, A.start, g, ra, rl, A.c.n);
        rec = make_int4(ra[0], ra[1], ra[2], kRowsMasked);
    }
    if (capped || max(rl[0], max(rl[1], rl[2])) > kShortRow) {
        density_long_rows<LM, BY_ID>(i, A);
        return;
    }
    const float hh = __ldg(&S->P.smoothing_radius);
    const float h2 = __fmul_rn(hh, hh);
    const float h_recip = __fdiv_rn(1.0f, hh);
    const float2 mp = make_float2(-p.x, -p.y);
    float2 ab = make_float2(0.0f, 0.0f);  // (rho, rho_near)
    const unsigned m0 = hit_mask32<kMarkUnroll>(pos + ra[0], rl[0], mp, h2);
    const unsigned m1 = hit_mask32<kMarkUnroll>(pos + ra[1], rl[1], mp, h2) &
                        ~(1u << ((i - ra[1]) & 31));  // not the particle itself
    const unsigned m2 = hit_mask32<kMarkUnroll>(pos + ra[2], rl[2], mp, h2);
    // walk_three without the record in flight, for which this pass has no
    // registers
    unsigned b0 = m0, b1 = m1, b2 = m2;
    int a0 = ra[0], a1 = ra[1], a2 = ra[2];
    if (!b1) { b1 = b2; a1 = a2; b2 = 0u; }
    if (!b0) { b0 = b1; a0 = a1; b1 = b2; a1 = a2; b2 = 0u; }
    while (b0) {
        const int j = a0 + __ffs(b0) - 1;
        b0 &= b0 - 1u;
        if (!b0) { b0 = b1; a0 = a1; b1 = b2; a1 = a2; b2 = 0u; }
        if (!in_bounds(j, A.c.n, kBadSlot)) continue;
        float2 e;
        add_density(ab, dist2_packed(mp, __ldg(pos + j), e), h_recip);
    }
    density_finish<BY_ID>(i, A, p, ab, m0, m1, m2, rec);
}

// 32 registers (four 512-thread CTAs' worth per SM): full occupancy for this
// issue-bound pass outweighs the few spilled values of its rare paths.
template <bool PERSIST, bool LM = false>
__global__ void __launch_bounds__(kMaxBlock, 4)
k_density_t(const __grid_constant__ DensArrays A)
{
    pdl_enter();
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = i0; i < A.c.n; i += gridDim.x * blockDim.x) {
        density_one<LM>(i, A);
        if (!PERSIST) break;
    }
}

// One density launch per block (the form other translation units call).
__global__ void __launch_bounds__(kMaxBlock)
k_density(const __grid_constant__ DensArrays A)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.c.n) density_one(i, A);
}

// ---------------------------------------------------------------------------
// pass 3: relaxation (gather) + boundary + velocity update + cell key
// ---------------------------------------------------------------------------

// Whether particle (slot i, id_i, cell ki) holds the pair with (slot j) in
// its own half list in the reference: same cell and smaller id
// (hash.c:178-199), or j's cell is one of i's forward cells
// (0,+1), (+1,-1), (+1,0), (+1,+1) (hash.c:203-234).
__device__ __noinline__ bool owns_pair(unsigned ki, int id_i, float2 qj, int id_j, const SG &g)
{
    const unsigned kj = cell_key(qj.x, qj.y, g);
    if (kj == ki) return id_i < id_j;
    const int li = (int)ki - g.c_off, lj = (int)kj - g.c_off;
    const int yi = li / g.size_x, xi = li - yi * g.size_x;
    const int yj = lj / g.size_x, xj = lj - yj * g.size_x;
    const int dx = xj - xi, dy = yj - yi;
    return (dx == 0 && dy == 1) || (dx == 1 && dy >= -1 && dy <= 1);
}

struct RelaxConsts {
    float h2, hh, h_recip, dt2, k, k_near, rest, half_spring;
};

// One neighbour's contribution to the displacement (r2 <= h2 known), with
// the constants pre-multiplied by dt^2; the rare r <= 1e-6 path computes
// the grid and cell key it needs itself, so that they are not live across
// the neighbour walk.
struct WalkConsts {
    float h_recip, kd, knd, hsd, hshd, Pd, Pnd;
};

// The scene's relaxation constants, and the walk's for particle record me =
// (x, y, rho, rho_near): P = k (rho - rest), Pn = k_near rho_near
// (fluid.c:563-564), pre-multiplied by dt^2.  One definition for every
// relaxation path, so that their pair terms round identically.
__device__ __forceinline__ RelaxConsts relax_consts(const Scene *__restrict__ S)
{
    RelaxConsts c;
    c.hh = __ldg(&S->P.smoothing_radius);
    c.h2 = __fmul_rn(c.hh, c.hh);
    c.h_recip = __fdiv_rn(1.0f, c.hh);
    const float dt = __ldg(&S->P.time_step);
    c.dt2 = __fmul_rn(dt, dt);
    c.k = __ldg(&S->P.k);
    c.k_near = __ldg(&S->P.k_near);
    c.rest = __ldg(&S->P.rest_density);
    c.half_spring = __fmul_rn(0.5f, __ldg(&S->P.k_spring));
    return c;
}

__device__ __forceinline__ WalkConsts walk_consts(const RelaxConsts &c, float4 me)
{
    const float Pi = __fmul_rn(c.k, __fsub_rn(me.z, c.rest));
    const float Pni = __fmul_rn(c.k_near, me.w);
    WalkConsts wc;
    wc.h_recip = c.h_recip;
    wc.kd = __fmul_rn(c.dt2, c.k);
    wc.knd = __fmul_rn(c.dt2, c.k_near);
    wc.hsd = __fmul_rn(c.dt2, c.half_spring);
    wc.hshd = __fmul_rn(wc.hsd, c.hh);
    wc.Pd = __fmul_rn(c.dt2, __fsub_rn(Pi, __fmul_rn(c.k, c.rest)));
    wc.Pnd = __fmul_rn(c.dt2, Pni);
    return wc;
}

// The largest float whose correctly rounded root is at most 1e-6.
constexpr float kNudgeR2 = 0x1.19799ap-40f;

// Whether particle i at `p` (cell `key`) is nudged by its pair with slot j at
// `q` (fluid.c:583-586): r <= 1e-6 and i holds the pair.
__device__ __forceinline__ bool is_nudge(int i, int j, float2 p, unsigned key, float2 q, const SG &g,
                                         const int *__restrict__ ids)
{
    float2 e;
    return dist2_packed(make_float2(-p.x, -p.y), q, e) <= kNudgeR2 && j != i &&
           owns_pair(key, __ldg(ids + i), q, __ldg(ids + j), g);
}

// The pair term of one neighbour (r2 <= h2 known, not the particle itself):
// returns whether it displaces the particle, by s (p - q) with d = q - p (the
// caller adds -s d with one packed FMA); `rare` is set by a pair that may be
// a nudge (r <= 1e-6).
__device__ __forceinline__ bool relax_pair_term(const WalkConsts &c, float2 p, float4 q, float &s,
                                                float2 &d, bool &rare)
{
    // d = q - p: the negated pair offset, rounded as p - q is
    const float r2 = dist2_packed(make_float2(-p.x, -p.y), make_float2(q.x, q.y), d);
    float r_recip = rsqrt_normal(r2);
    if (r2 <= 2e-12f) {
        rare = true;
        if (!(r2 > 0.0f)) return false;
        r_recip = rsqrtf(r2);
    }
    const float r = r2 * r_recip;
    const float ratio = __fmul_rn(r, c.h_recip);
    if (!(ratio < 1.0f)) return false;
    // rounded step by step: the same bits wherever this is compiled into
    const float omr = __fsub_rn(1.0f, ratio);
    const float near = __fmul_rn(__fmaf_rn(c.knd, q.w, c.Pnd), omr);
    const float X = __fmaf_rn(__fmaf_rn(c.kd, q.z, c.Pd), omr, __fmul_rn(near, omr));
    const float D = __fadd_rn(X, __fmaf_rn(-c.hsd, r, c.hshd));
    s = D * r_recip;
    return true;
}

__device__ __forceinline__ void relax_pair_walk(const WalkConsts &c, float2 p, float4 q, float2 &a,
                                                bool &rare)
{
    float s;
    float2 d;
    if (relax_pair_term(c, p, q, s, d, rare))
        a = __ffma2_rn(make_float2(-s, -s), d, a);  // += s (p - q), per component
}

// double_density_relaxation (fluid.c:541-611) in gather form:
//   dx_i = sum_{j: 0 < r < h} D_ij (x_i - x_j)/r,
//   D_ij = dt^2 [(P_i + P_j)(1 - r/h) + (Pn_i + Pn_j)(1 - r/h)^2 + k_spring (h - r)/2],
//   P = k (rho - rest_density), Pn = k_near rho_near (fluid.c:560-565),
// plus the reference's (1e-6, 1e-6) nudge for each pair with r <= 1e-6 that
// the particle owns (fluid.c:583-586).  Then updateVelocities
// (fluid.c:642-653): boundaryConditions, v = (x - x_prev)/dt clamped to +-5.
// Walks the density pass's hit masks; rows longer than kMaskRow (or
// overflowing buckets) fall back to the whole stencil.
// PROBE writes the displacement instead of advancing.
// The network's output for a learned step: particle i takes the displacement
// (net.x, net.y) * s, s = h dt^2 (k + k_near + k_spring), when it has at most
// max_nb neighbours (counts of 65535 mark particles the network must not
// take) and the predicted density error net.z (percent of rest density) is
// at most thr_pct; every other particle runs the plain relaxation.
struct LearnedIn {
    const float4 *net = nullptr;
    const unsigned short *nbc = nullptr;
    float thr_pct = 0.0f;
    int max_nb = 0;
    bool defer = false;  // leave the fallback particles to a second pass
};

// What a relaxation reads and writes.
struct RelaxArrays {
    Ctx c;
    const float4 *xr;
    const ulonglong2 *mask01;
    const unsigned long long *mask2;
    const int4 *rows;
    const float2 *prev;
    const int *ids, *start;
    const unsigned *occ_in;  // the build's largest cell population
    float2 *pos_out, *vel_out;
    uint2 *kr_out;
    unsigned *cnt;
    float2 *probe_out;
};

// The end of a particle's relaxation: x += the displacement and the owner's
// nudges, boundaryConditions, then updateVelocity (fluid.c:627-653):
// v = (x - x_prev)/dt clamped to +-5, and the new position's cell key
// counted into the build of the relaxed positions.
__device__ __forceinline__ void relax_finish(int i, const RelaxArrays &A, const Scene *S, float2 p,
                                             float2 acc, int nudges, int *tile_made)
{
    const float nd = (float)nudges * 0.000001f;
    float nx = __fadd_rn(__fadd_rn(p.x, acc.x), nd);
    float ny = __fadd_rn(__fadd_rn(p.y, acc.y), nd);
    boundary_of(nx, ny, S);
    const float2 pv = A.prev[i];
    const float dt_end = __ldg(&S->P.time_step);
    const float vx = clamp5(__fdiv_rn(__fsub_rn(nx, pv.x), dt_end));
    const float vy = clamp5(__fdiv_rn(__fsub_rn(ny, pv.y), dt_end));
    const unsigned k2 = cell_key(nx, ny, load_grid(S));
    unsigned rank = 0u;
    if (in_bounds(k2, A.c.M, kBadKey)) {
        rank = atomicAdd(A.cnt + k2, 1u);
        if (tile_made)
            *tile_made = (int)(k2 / (unsigned)kBuildTile);
        else
            add_tile_count(A.c.tile_cnt, k2);
    }
    A.pos_out[i] = make_float2(nx, ny);
    A.vel_out[i] = make_float2(vx, vy);
    A.kr_out[i] = make_uint2(k2, rank);
}

// The end of a relaxation in a function of its own (relax_cold).
template <bool PROBE>
__device__ __forceinline__ void relax_end_cold(int i, const RelaxArrays &A, const Scene *S, float2 p,
                                               float2 acc, int nudges)
{
    if (PROBE) {
        const float nd = (float)nudges * 0.000001f;
        A.probe_out[i] = make_float2(acc.x + nd, acc.y + nd);
        return;
    }
    relax_finish(i, A, S, p, acc, nudges, nullptr);
}

// The nudges of a particle whose walk has met a pair that may be one (r2 <=
// 2e-12): such pairs are searched for again.  Hardly any particle has one,
// but early in the dam break of 41,000 to 200,000 particles a step waits for
// the warp of the one that does, and most of that wait is the fetch of code
// that nothing else runs: so there is little of it (relax_update 20.5 us
// with the search and the rest of the relaxation out of line, 14.3 so).
template <bool LM>
__device__ __forceinline__ int masked_nudges(int i, const RelaxArrays &A, const Scene *S, float2 p,
                                             const int4 &rw)
{
    const SG g = load_grid(S);
    const unsigned key = cell_key(p.x, p.y, g);
    int nudges = 0;
    // the rows' masks, then (LM) those of their candidates beyond kMaskRow
#pragma unroll 1
    for (int w = 0; w < (LM && rw.w == kRowsMasked2 ? 6 : 3); ++w) {
        const int r = w < 3 ? w : w - 3;
        const int base = (r == 0 ? rw.x : r == 1 ? rw.y : rw.z) + (w < 3 ? 0 : kMaskRow);
        const unsigned long long *at = w >= 3 ? A.c.maskx + 3 * (size_t)i + r
                                       : r < 2 ? &A.mask01[i].x + r : A.mask2 + i;
#pragma unroll 1
        for (unsigned long long m = __ldg(at); m; m &= m - 1ull) {
            const int j = base + __ffsll(m) - 1;
            const float4 q = __ldg(A.xr + j);
            nudges += is_nudge(i, j, p, key, make_float2(q.x, q.y), g, A.ids);
        }
    }
    return nudges;
}

// The same over the whole stencil, for particles without hit masks.
__device__ __noinline__ int nudges_of(int i, const RelaxArrays &A)
{
    const Scene *S = A.c.scenes + scene_of(A.c, i);
    const SG g = load_grid(S);
    const float hh = __ldg(&S->P.smoothing_radius), h2 = __fmul_rn(hh, hh);
    const float4 me = __ldg(A.xr + i);
    const float2 p = make_float2(me.x, me.y), mp = make_float2(-me.x, -me.y);
    const unsigned key = cell_key(p.x, p.y, g);
    const bool capped = *A.occ_in > (unsigned)A.c.max_bucket;
    int nudges = 0;
    if (searchable(key, i, A.start, g, capped, A.c.max_bucket))
        for_each_candidate(key, A.start, g, capped, A.c.max_bucket, A.c.n, [&](int j) {
            const float4 q = __ldg(A.xr + j);
            float2 e;
            if (dist2_packed(mp, make_float2(q.x, q.y), e) <= h2)
                nudges += is_nudge(i, j, p, key, make_float2(q.x, q.y), g, A.ids);
        });
    return nudges;
}

// A particle whose rows have no hit masks (a row too long for them, or an
// overflowing bucket), in slot order as everywhere.  MARK: 96 candidates
// marked and their hits walked at a time, where the lanes of a warp are of
// different cells (the fallback list: 106 us for 219,000 particles, 32 at a
// time 117, in one loop over the candidates 129); one loop where they are mostly of one
// (4,194,304 particles, compressed further: 475 -> 355 us; 64 compressed
// scenes 206 -> 174 us).  No calls inside the loops, which would cost them
// registers.
template <bool PROBE, bool MARK>
__device__ __noinline__ void relax_cold(int i, const RelaxArrays &A)
{
    const Ctx &cx = A.c;
    const Scene *S = cx.scenes + scene_of(cx, i);
    const SG g = load_grid(S);
    const RelaxConsts c = relax_consts(S);
    const float4 *xr = A.xr;
    const float4 me = __ldg(xr + i);
    const WalkConsts wc = walk_consts(c, me);
    const float2 p = make_float2(me.x, me.y), mp = make_float2(-me.x, -me.y);
    const bool capped = *A.occ_in > (unsigned)cx.max_bucket;
    const int n = cx.n;
    float2 acc = make_float2(0.0f, 0.0f);
    bool rare = false;
    auto visit = [&](int, const float4 &q) { relax_pair_walk(wc, p, q, acc, rare); };
    const unsigned key = cell_key(p.x, p.y, g);
    if (searchable(key, i, A.start, g, capped, cx.max_bucket)) {
        if (!capped) {
            int ra[3], rl[3];
            stencil_rows(p, key, A.start, g, ra, rl, n);
#pragma unroll 1
            for (int r = 0; r < 3; ++r) {
                const int a = ra[r], l = rl[r];
                if (MARK) {
#pragma unroll 1
                    for (int c0 = 0; c0 < l; c0 += 96) {
                        unsigned b[3];
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            const int o = c0 + 32 * k, m = min(l - o, 32);
                            b[k] = 0u;
#pragma unroll 4
                            for (int t = 0; t < m; ++t) {
                                const float4 q = __ldg(xr + a + o + t);
                                float2 e;
                                if (dist2_packed(mp, make_float2(q.x, q.y), e) <= c.h2) b[k] |= 1u << t;
                            }
                            if (r == 1 && (unsigned)(i - a - o) < 32u) b[k] &= ~(1u << (i - a - o));
                        }
                        walk_three<float4>(b[0], a + c0, b[1], a + c0 + 32, b[2], a + c0 + 64, n,
                                           [&](int j) { return __ldg(xr + j); }, visit);
                    }
                } else {
#pragma unroll 4
                    for (int j = a; j < a + l; ++j) {
                        const float4 q = __ldg(xr + j);
                        float2 e;
                        if (dist2_packed(mp, make_float2(q.x, q.y), e) <= c.h2 && j != i) visit(j, q);
                    }
                }
            }
        } else {
            for_each_candidate(key, A.start, g, true, cx.max_bucket, n, [&](int j) {
                if (j == i) return;
                const float4 q = __ldg(xr + j);
                if (dist2(p.x - q.x, p.y - q.y) > c.h2) return;
                visit(j, q);
            });
        }
    }
    relax_end_cold<PROBE>(i, A, S, p, acc, rare ? nudges_of(i, A) : 0);
}

// MARK: as in relax_cold.
template <bool PROBE, bool LEARNED = false, bool LM = false, bool MARK = false>
__device__ __forceinline__ void relax_update_one(int i, const RelaxArrays &A,
                                                 const LearnedIn &L = LearnedIn(),
                                                 bool *used_net = nullptr, int *tile_made = nullptr)
{
    const Ctx &cx = A.c;
    const Scene *S = cx.scenes + scene_of(cx, i);
    const float4 *xr = A.xr;
    const float4 me = xr[i];
    // the plain pass requests the hit masks with the record and prefetches
    // the previous position, so that their DRAM latencies overlap instead of
    // following one another (the record decides whether the masks are used;
    // relax_finish reads the previous position): 7% off this latency-bound
    // pass
    constexpr bool kHoist = !LEARNED;
    ulonglong2 m01 = make_ulonglong2(0ull, 0ull);
    unsigned long long m2 = 0ull;
    if (kHoist) {
        m01 = __ldg(A.mask01 + i);
        m2 = __ldg(A.mask2 + i);
        if (!PROBE) asm volatile("prefetch.global.L1 [%0];" ::"l"(A.prev + i));
    }
    const float2 p = make_float2(me.x, me.y);
    float2 acc = make_float2(0.0f, 0.0f);  // the displacement
    int nudges = 0;
    bool net = false;
    if (LEARNED) {
        // the network's output requested with the count (not after it), and
        // the previous position prefetched for relax_finish: one DRAM latency
        // for a network particle instead of three in a row
        const float4 y = __ldg(L.net + i);
        if (!PROBE) asm volatile("prefetch.global.L1 [%0];" ::"l"(A.prev + i));
        if ((int)__ldg(L.nbc + i) <= L.max_nb && y.z <= L.thr_pct) {
            const RelaxConsts c = relax_consts(S);
            const float s = c.hh * c.dt2 * (c.k + c.k_near + 2.0f * c.half_spring);
            acc = make_float2(y.x * s, y.y * s);
            net = true;
        }
    }
    if (LEARNED && used_net) *used_net = net;
    if (LEARNED && !net && L.defer) return;
    if (!net) {
        // the density pass's row record: the stencil rows' first slots, so
        // the walk needs neither the cell key nor the cell starts
        const int4 rw = __ldg(A.rows + i);
        const int ra[3] = {rw.x, rw.y, rw.z};
        bool rare = false;
        if (rw.w == kRowsMasked || (LM && rw.w == kRowsMasked2)) {
            const WalkConsts wc = walk_consts(relax_consts(S), me);
            if (!kHoist) {
                m01 = __ldg(A.mask01 + i);
                m2 = __ldg(A.mask2 + i);
            }
            const unsigned long long mm[3] = {m01.x, m01.y, m2};
            auto load = [&](int j) { return __ldg(xr + j); };
            auto visit = [&](int, const float4 &q) { relax_pair_walk(wc, p, q, acc, rare); };
            if (!LM || rw.w == kRowsMasked) {
                walk_rows<float4>(mm, ra, cx.n, load, visit);
            } else {
                // rows of up to 2 kMaskRow candidates: each row's two masks in
                // slot order (the visiting order of the whole-stencil walk)
                const unsigned long long *mx = cx.maskx + 3 * (size_t)i;
                const unsigned long long mh[3] = {__ldg(mx), __ldg(mx + 1), __ldg(mx + 2)};
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    walk_mask<float4>(mm[r], ra[r], cx.n, load, visit);
                    walk_mask<float4>(mh[r], ra[r] + kMaskRow, cx.n, load, visit);
                }
            }
        } else {
            relax_cold<PROBE, MARK>(i, A);
            return;
        }
        if (rare) nudges = masked_nudges<LM>(i, A, S, p, rw);
    }
    if (PROBE) {
        const float nd = (float)nudges * 0.000001f;
        A.probe_out[i] = make_float2(acc.x + nd, acc.y + nd);
        return;
    }
    relax_finish(i, A, S, p, acc, nudges, tile_made);
}

// 40 registers: 48 resident warps per SM instead of 32 (64 registers) for
// this latency-bound pass; what the rare paths would need is out of line
// (4,194,304 particles: 64 registers 178 us early in the dam break and 227 us
// compressed, 48 with the long rows' sum alone out of line 152 and 199, this
// 138 and 172).
template <bool PROBE, bool PERSIST = false, bool LM = false>
__global__ void __maxnreg__(40)
k_relax_update(const __grid_constant__ RelaxArrays A, unsigned *occ_reset)
{
    pdl_enter();
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (!PROBE && i0 == 0) *occ_reset = 0u;
    for (int i = i0; i < A.c.n; i += gridDim.x * blockDim.x) {
        relax_update_one<PROBE, false, LM>(i, A);
        if (!PERSIST) break;
    }
}

// The relaxation pass of a learned step (one particle per thread).  PROBE:
// every particle's displacement, fallback included.  Otherwise the particles
// that take the network are advanced here and the others are appended to
// fb_list (one atomic per warp that has any) for k_relax_fallback, so that
// the rare plain gathers do not hold up whole warps.  Block 0 counts the step.
template <bool PROBE, bool LM = false>
__global__ void __launch_bounds__(kBlock, 4)
k_relax_learned(const __grid_constant__ RelaxArrays A, unsigned *occ_reset, LearnedIn L,
                DevState *st, int *__restrict__ fb_list)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (!PROBE && i == 0) {
        *occ_reset = 0u;
        atomicAdd(&st->learned_steps, 1ull);
    }
    bool used = true;
    L.defer = !PROBE;
    int t = -1;
    if (i < A.c.n) relax_update_one<PROBE, true, LM>(i, A, L, &used, &t);
    if (PROBE) return;
    if (A.c.tile_cnt) cta_tile_count(A.c.tile_cnt, t);
    // fallback particles: those whose stencil rows fit the hit masks go to
    // the front of fb_list (one thread each in k_relax_fallback), those with
    // a row too long for a mask to the back (one warp each)
    const bool longrow = !used && __ldg(A.rows + i).w == kRowsFull;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned fbs = __ballot_sync(0xffffffffu, !used && !longrow);
    const unsigned fbl = __ballot_sync(0xffffffffu, longrow);
    if (fbs) {
        const int leader = __ffs(fbs) - 1;
        unsigned base = 0;
        if (lane == (unsigned)leader) base = atomicAdd(&st->fb_count, (unsigned)__popc(fbs));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (!used && !longrow) fb_list[base + __popc(fbs & ((1u << lane) - 1u))] = i;
    }
    if (fbl) {
        const int leader = __ffs(fbl) - 1;
        unsigned base = 0;
        if (lane == (unsigned)leader) base = atomicAdd(&st->fb_long, (unsigned)__popc(fbl));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (longrow) fb_list[A.c.n - 1 - (int)(base + __popc(fbl & ((1u << lane) - 1u)))] = i;
    }
}

// ---------------------------------------------------------------------------
// the gathers with G lanes per particle (small handles)
// ---------------------------------------------------------------------------

// One thread per particle leaves the GPU nearly idle where there are few
// particles: a pass then takes as long as one thread needs for its densest
// particle's candidates, one after another (3,000 particles, dense: 16-30 us
// a gather at 1-2% of the issue slots).  Here G lanes of a warp share a
// particle: they load and test G candidates of a stencil row at once and
// evaluate the hits' terms side by side; the terms are then added in slot
// order from shuffles, by every lane, with the very operations of the
// one-thread passes -- bit for bit the same sums.  A lane whose candidate
// is no hit takes no part in the additions.
//
// All lanes of a warp run the same loops (bounds are maxima over its
// groups), so that every shuffle and vote is converged; groups past the last
// particle have empty rows.
template <int G>
struct Group {
    static_assert(G == 4 || G == 8 || G == 16 || G == 32, "lanes per particle");
    static constexpr unsigned kFull = 0xffffffffu;
    int lane, gl, base;
    __device__ __forceinline__ Group()
    {
        lane = threadIdx.x & 31;
        gl = lane & (G - 1);
        base = lane & ~(G - 1);
    }
    // the group's bits of a warp vote
    __device__ __forceinline__ unsigned ballot(bool p) const
    {
        const unsigned b = __ballot_sync(kFull, p);
        return G == 32 ? b : (b >> base) & ((1u << (G & 31)) - 1u);
    }
    __device__ __forceinline__ static int max_over_warp(int v) { return __reduce_max_sync(kFull, v); }
    // visits the set bits of `hits` (the group's lanes) in increasing order:
    // f(source lane, whether this group still has one)
    template <class F>
    __device__ __forceinline__ void ordered(unsigned hits, F &&f) const
    {
        const int iters = G == 32 ? __popc(hits) : max_over_warp(__popc(hits));
#pragma unroll 4
        for (int k = 0; k < iters; ++k) {
            const bool on = hits != 0u;
            const int src = base + (on ? __ffs(hits) - 1 : 0);
            hits &= hits - 1u;
            f(src, on);
        }
    }
};

// Whether a group kernel shares its particles among lanes: where a cell is
// populated enough for it (min_occ, from lanes_min_occ) and no bucket
// overflows.  Else its first n threads take a particle each and the other
// warps leave.
template <class Arrays>
__device__ __forceinline__ bool shared_by_lanes(const Arrays &A, unsigned min_occ)
{
    const unsigned occ = *A.occ_in;
    return occ >= min_occ && occ <= (unsigned)A.c.max_bucket;
}

// Particle i's viscosity pass by the group (every lane of the warp calls it;
// `valid` per group; no overflowing buckets).
template <int G>
__device__ __forceinline__ void viscosity_group_one(const Group<G> &g, int i, bool valid,
                                                    const ViscArrays &A)
{
    const Ctx &c = A.c;
    const float2 *pos = A.pos, *vel = A.vel;
    const Scene *S = c.scenes + scene_of(c, i);
    const SG sg = load_grid(S);
    const float2 p = __ldg(pos + i), v0 = __ldg(vel + i);
    const float dt = __ldg(&S->P.time_step);
    const float hh = __ldg(&S->P.smoothing_radius);
    const float h2 = __fmul_rn(hh, hh);
    const float dt_h = dt * __fdiv_rn(1.0f, hh);
    const float sigma = __ldg(&S->P.sigma), beta = __ldg(&S->P.beta);
    const unsigned key = cell_key(p.x, p.y, sg);
    int ra[3] = {0, 0, 0}, rl[3] = {0, 0, 0};
    if (valid && A.st->lists_valid && searchable(key, i, A.start, sg, false, c.max_bucket))
        stencil_rows(p, key, A.start, sg, ra, rl, c.n);
    const float2 mp = make_float2(-p.x, -p.y);
    float2 dv = make_float2(0.0f, 0.0f);
    // the rows' first candidates, requested together
    float2 q0[3], w0[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        q0[r] = w0[r] = make_float2(0.0f, 0.0f);
        if (g.gl < rl[r]) {
            q0[r] = __ldg(pos + ra[r] + g.gl);
            w0[r] = __ldg(vel + ra[r] + g.gl);
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int len = Group<G>::max_over_warp(rl[r]);
        for (int t0 = 0; t0 < len; t0 += G) {
            const int t = t0 + g.gl;
            float2 q = q0[r], w = w0[r];
            if (t0 > 0 && t < rl[r]) {
                q = __ldg(pos + ra[r] + t);
                w = __ldg(vel + ra[r] + t);
            }
            float2 e;
            const float r2 = dist2_packed(mp, q, e);
            float cx = 0.0f, cy = 0.0f;
            bool push = false;
            if (t < rl[r] && r2 <= h2 && r2 != 0.0f) {
                // as visc_impulse: a pair that does not approach has u = 0 and
                // adds +-0 there and nothing here (or a NaN in both, with
                // tunables without bounds)
                const float r_recip = rsqrtf(r2);
                const float rr = r2 * r_recip;
                const float2 dw = __fadd2_rn(v0, make_float2(-w.x, -w.y));
                const float u = fmaxf(__fmaf_rn(dw.x, e.x, __fmul_rn(dw.y, e.y)) * r_recip, 0.0f);
                const float imp = fmaf(-dt_h, rr, dt) * u * fmaf(beta, u, sigma);
                const float2 m = __fmul2_rn(__fmul2_rn(make_float2(imp, imp), e),
                                            make_float2(r_recip, r_recip));
                cx = clamp5(m.x);
                cy = clamp5(m.y);
                push = cx != 0.0f || cy != 0.0f;
            }
            g.ordered(g.ballot(push), [&](int src, bool on) {
                const float sx = __shfl_sync(Group<G>::kFull, cx, src);
                const float sy = __shfl_sync(Group<G>::kFull, cy, src);
                if (on) dv = __ffma2_rn(make_float2(-0.5f, -0.5f), make_float2(sx, sy), dv);
            });
        }
    }
    if (valid && g.gl == 0)
        viscosity_finish<false>(i, A, S, sg, p, v0, dv);
}

template <int G>
__global__ void __launch_bounds__(kBlock)
k_viscosity_group(const __grid_constant__ ViscArrays A, unsigned *occ_reset, unsigned min_occ)
{
    pdl_enter();
    const int th = blockIdx.x * blockDim.x + threadIdx.x;
    if (th == 0) *occ_reset = 0u;
    if (!shared_by_lanes(A, min_occ)) {
        if (th < A.c.n) viscosity_predict_one<false, true>(th, A);
        return;
    }
    const Group<G> g;
    const bool valid = th / G < A.c.n;
    const int i = valid ? th / G : A.c.n - 1;
    viscosity_group_one<G>(g, i, valid, A);
}

template <int G, bool LM, bool BY_ID = false>
__device__ __forceinline__ void density_group_one(const Group<G> &g, int i, bool valid,
                                                  const DensArrays &A)
{
    const Ctx &c = A.c;
    const float2 *pos = A.pos;
    const Scene *S = c.scenes + scene_of(c, i);
    const SG sg = load_grid(S);
    const float2 p = __ldg(pos + i);
    const float hh = __ldg(&S->P.smoothing_radius);
    const float h2 = __fmul_rn(hh, hh);
    const float h_recip = __fdiv_rn(1.0f, hh);
    const float2 mp = make_float2(-p.x, -p.y);
    const unsigned key = cell_key(p.x, p.y, sg);
    const bool search = valid && searchable(key, i, A.start, sg, false, c.max_bucket);
    int ra[3] = {0, 0, 0}, rl[3] = {0, 0, 0};
    if (search) stencil_rows(p, key, A.start, sg, ra, rl, c.n);
    float2 ab = make_float2(0.0f, 0.0f);
    unsigned long long m[3] = {0ull, 0ull, 0ull}, mx[3] = {0ull, 0ull, 0ull};
    float2 q0[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        q0[r] = g.gl < rl[r] ? __ldg(pos + ra[r] + g.gl) : make_float2(0.0f, 0.0f);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int len = Group<G>::max_over_warp(rl[r]);
        for (int t0 = 0; t0 < len; t0 += G) {
            const int t = t0 + g.gl;
            float2 q = q0[r];
            if (t0 > 0 && t < rl[r]) q = __ldg(pos + ra[r] + t);
            float2 e;
            const float r2 = dist2_packed(mp, q, e);
            const bool hit = t < rl[r] && r2 <= h2 && ra[r] + t != i;
            float2 term = make_float2(0.0f, 0.0f);
            if (hit) add_density(term, r2, h_recip);  // 0 + x: the term itself
            const unsigned bits = g.ballot(hit);
            if (t0 < kMaskRow) m[r] |= (unsigned long long)bits << t0;
            else if (LM && t0 < 2 * kMaskRow) mx[r] |= (unsigned long long)bits << (t0 - kMaskRow);
            g.ordered(bits, [&](int src, bool on) {
                const float ta = __shfl_sync(Group<G>::kFull, term.x, src);
                const float tb = __shfl_sync(Group<G>::kFull, term.y, src);
                if (on) ab = __fadd2_rn(ab, make_float2(ta, tb));
            });
        }
    }
    if (!valid || g.gl != 0) return;
    int4 rec = make_int4(0, 0, 0, kRowsNone);
    if (search && !BY_ID) {
        rec.w = kRowsFull;
        if (rl[0] <= kMaskRow && rl[1] <= kMaskRow && rl[2] <= kMaskRow) {
            rec = make_int4(ra[0], ra[1], ra[2], kRowsMasked);
        } else if (LM && c.maskx && rl[0] <= 2 * kMaskRow && rl[1] <= 2 * kMaskRow &&
                   rl[2] <= 2 * kMaskRow) {
            rec = make_int4(ra[0], ra[1], ra[2], kRowsMasked2);
            unsigned long long *x = c.maskx + 3 * (size_t)i;
            x[0] = mx[0]; x[1] = mx[1]; x[2] = mx[2];
        }
    }
    density_finish<BY_ID>(i, A, p, ab, m[0], m[1], m[2], rec);
}

template <int G, bool LM>
__global__ void __launch_bounds__(kBlock)
k_density_group(const __grid_constant__ DensArrays A, unsigned min_occ)
{
    pdl_enter();
    const int th = blockIdx.x * blockDim.x + threadIdx.x;
    if (!shared_by_lanes(A, min_occ)) {
        if (th < A.c.n) density_one<LM>(th, A);
        return;
    }
    const Group<G> g;
    const bool valid = th / G < A.c.n;
    const int i = valid ? th / G : A.c.n - 1;
    density_group_one<G, LM>(g, i, valid, A);
}

template <int G, bool LM>
__device__ __forceinline__ void relax_group_one(const Group<G> &g, int i, bool valid,
                                                const RelaxArrays &A)
{
    const Ctx &c = A.c;
    const float4 *xr = A.xr;
    // the particle's record, masks and rows, requested together
    const float4 me = __ldg(xr + i);
    const int4 rw = __ldg(A.rows + i);
    const ulonglong2 m01 = __ldg(A.mask01 + i);
    const unsigned long long m2 = __ldg(A.mask2 + i);
    asm volatile("prefetch.global.L1 [%0];" ::"l"(A.prev + i));
    const Scene *S = c.scenes + scene_of(c, i);
    const RelaxConsts rc = relax_consts(S);
    const float2 p = make_float2(me.x, me.y);
    const WalkConsts wc = walk_consts(rc, me);
    // the rows to visit: with hit masks only the hits are loaded (the
    // distance test below holds for exactly those), else every candidate
    int ra[3] = {rw.x, rw.y, rw.z}, rl[3] = {0, 0, 0};
    unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {~0ull, ~0ull, ~0ull};
    const int mode = valid ? rw.w : kRowsNone;
    if (mode == kRowsMasked || (LM && mode == kRowsMasked2)) {
        lo[0] = m01.x; lo[1] = m01.y; lo[2] = m2;
        hi[0] = hi[1] = hi[2] = 0ull;
        if (LM && mode == kRowsMasked2) {
            const unsigned long long *x = c.maskx + 3 * (size_t)i;
#pragma unroll
            for (int r = 0; r < 3; ++r) hi[r] = __ldg(x + r);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) rl[r] = hi[r] ? 128 - __clzll(hi[r]) : lo[r] ? 64 - __clzll(lo[r]) : 0;
    } else if (mode != kRowsNone) {
        const SG sg = load_grid(S);
        const unsigned key = cell_key(p.x, p.y, sg);
        ra[0] = ra[1] = ra[2] = 0;
        if (searchable(key, i, A.start, sg, false, c.max_bucket))
            stencil_rows(p, key, A.start, sg, ra, rl, c.n);
    }
    const bool masked = mode != kRowsFull;
    auto wanted = [&](int r, int t) {
        if (t >= rl[r]) return false;
        if (!masked) return ra[r] + t != i;
        return t < 64 ? ((lo[r] >> t) & 1ull) != 0ull : LM && ((hi[r] >> (t - 64)) & 1ull) != 0ull;
    };
    float4 q0[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        q0[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (wanted(r, g.gl) && in_bounds(ra[r] + g.gl, c.n, kBadSlot)) q0[r] = __ldg(xr + ra[r] + g.gl);
    }
    float2 acc = make_float2(0.0f, 0.0f);
    int nudges = 0;
    const float2 mp = make_float2(-p.x, -p.y);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const int len = Group<G>::max_over_warp(rl[r]);
        for (int t0 = 0; t0 < len; t0 += G) {
            const int t = t0 + g.gl, j = ra[r] + t;
            float s = 0.0f;
            float2 d = make_float2(0.0f, 0.0f);
            bool apply = false;
            if (wanted(r, t) && in_bounds(j, c.n, kBadSlot)) {
                const float4 q = t0 > 0 ? __ldg(xr + j) : q0[r];
                float2 e;
                if (dist2_packed(mp, make_float2(q.x, q.y), e) <= rc.h2) {
                    bool rare = false;
                    apply = relax_pair_term(wc, p, q, s, d, rare);
                    if (rare) {
                        const SG sg = load_grid(S);
                        nudges += is_nudge(i, j, p, cell_key(p.x, p.y, sg), make_float2(q.x, q.y), sg, A.ids);
                    }
                }
            }
            g.ordered(g.ballot(apply), [&](int src, bool on) {
                const float ss = __shfl_sync(Group<G>::kFull, s, src);
                const float dx = __shfl_sync(Group<G>::kFull, d.x, src);
                const float dy = __shfl_sync(Group<G>::kFull, d.y, src);
                if (on) acc = __ffma2_rn(make_float2(-ss, -ss), make_float2(dx, dy), acc);
            });
        }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) nudges += __shfl_xor_sync(Group<G>::kFull, nudges, o);
    if (valid && g.gl == 0)
        relax_finish(i, A, S, p, acc, nudges, nullptr);
}

// Left to itself the compiler takes 64 registers and spills; 75 to 80 without
// spills (frames of the dam break of 3,000 / 7,000 / 15,000 particles 134 ->
// 132, 192 -> 188 and 261 -> 257 us; 86 with the long-row masks: 5% slower).
template <int G, bool LM>
__global__ void __launch_bounds__(kBlock, G == 8 || LM ? 3 : 1)
k_relax_group(const __grid_constant__ RelaxArrays A, unsigned *occ_reset, unsigned min_occ)
{
    pdl_enter();
    const int th = blockIdx.x * blockDim.x + threadIdx.x;
    if (th == 0) *occ_reset = 0u;
    if (!shared_by_lanes(A, min_occ)) {
        if (th < A.c.n) relax_update_one<false, false, LM>(th, A);
        return;
    }
    const Group<G> g;
    const bool valid = th / G < A.c.n;
    const int i = valid ? th / G : A.c.n - 1;
    relax_group_one<G, LM>(g, i, valid, A);
}

// The fallback particles of a learned step: the plain relaxation + update for
// each slot on fb_list (those with hit masks from its front, those with a row
// too long for them from its back).  They are the densest particles, with the
// longest walks of all, and mostly too few to fill the GPU with a thread
// each: 32 or 4 lanes a particle while the grid holds them in one pass, else
// a thread each (at two passes of 4 lanes the threads are the faster).  The
// same bits either way.  The dam break's 1,048,576 particles: 26,000 on the
// list 61 -> 35 us, 90,000 72 -> 53 us.  Grid-stride loops: the counts are
// known on the device only.  Block 0 adds them to the fallback statistics.
template <bool LM>
__global__ void __launch_bounds__(kBlock, kFallbackCtas)
k_relax_fallback(const __grid_constant__ RelaxArrays A, DevState *st,
                 const int *__restrict__ fb_list)
{
    const unsigned front = st->fb_count, total = front + st->fb_long;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(&st->learned_fallback, (unsigned long long)total);
    const bool capped = *A.occ_in > (unsigned)A.c.max_bucket;
    const unsigned t0 = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nt = gridDim.x * blockDim.x, resident = nt / kFallbackWaves;
    auto slot_of = [&](unsigned k) { return fb_list[k < front ? (int)k : A.c.n - 1 - (int)(k - front)]; };
    auto by_groups = [&](auto G) {
        const Group<G.value> g;
        const unsigned k = t0 / G.value, k0 = (t0 & ~31u) / G.value;
        if (k0 >= total) return;  // the whole warp
        const bool valid = k < total;
        relax_group_one<G.value, LM>(g, slot_of(valid ? k : k0), valid, A);
    };
    if (!capped && total <= resident / 32) {
        by_groups(std::integral_constant<int, 32>());
    } else if (!capped && total <= resident / 4) {
        by_groups(std::integral_constant<int, 4>());
    } else {
        for (unsigned k = t0; k < total; k += nt) relax_update_one<false, false, LM, true>(slot_of(k), A);
    }
}

// ---------------------------------------------------------------------------
// state I/O, diagnostics, neighbour lists
// ---------------------------------------------------------------------------

// Sorted state -> id order: out = [pos | vel | prev | rho | pressure] (5 n float2).
__global__ void __launch_bounds__(kBlock)
k_unpermute(Ctx c, const int *__restrict__ id_a, const float2 *__restrict__ pos_a,
            const float2 *__restrict__ vel_a, const int *__restrict__ id_c,
            const float2 *__restrict__ prev_c, const float4 *__restrict__ xr_c,
            float2 *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const size_t n = (size_t)c.n;
    const int ia = id_a[i], ic = id_c[i];
    out[ia] = pos_a[i];
    out[n + ia] = vel_a[i];
    out[2 * n + ic] = prev_c[i];
    const float4 x4 = xr_c[i];
    const float2 r = make_float2(x4.z, x4.w);
    out[3 * n + ic] = r;
    // pressure and near pressure, fluid.c:563-564, with the scene's tunables
    const Scene *S = c.scenes + scene_of(c, i);
    const float k = __ldg(&S->P.k), rest = __ldg(&S->P.rest_density), kn = __ldg(&S->P.k_near);
    out[4 * n + ic] = make_float2(__fmul_rn(k, __fsub_rn(r.x, rest)), __fmul_rn(kn, r.y));
}

// (rho, rho_near) of the (x, y, rho, rho_near) records.
__global__ void __launch_bounds__(kBlock)
k_xr_density(int n, const float4 *__restrict__ xr, float2 *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = xr[i];
    out[i] = make_float2(v.z, v.w);
}

// Sorted per-particle values -> id order.
__global__ void __launch_bounds__(kBlock)
k_by_id(int n, const int *__restrict__ ids, const float2 *__restrict__ in, float2 *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[ids[i]] = in[i];
}

// Pixel-space shorts for the render rank (fluid.c:360-361), by id.
__global__ void __launch_bounds__(kBlock)
k_pack_coords(Ctx c, const int *__restrict__ id_a, const float2 *__restrict__ pos_a,
              short2 *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const Scene *S = c.scenes + scene_of(c, i);
    const float max_x = __ldg(&S->max_x), max_y = __ldg(&S->max_y);
    const float2 p = pos_a[i];
    const float cx = __fmul_rn(__fsub_rn(__fdiv_rn(__fmul_rn(2.0f, p.x), max_x), 1.0f), 32767.0f);
    const float cy = __fmul_rn(__fsub_rn(__fdiv_rn(__fmul_rn(2.0f, p.y), max_y), 1.0f), 32767.0f);
    out[id_a[i]] = make_short2((short)__float2int_rz(cx), (short)__float2int_rz(cy));
}

// FP64 sums of density, near density and 0.5|v|^2, per block (fixed order).
__global__ void __launch_bounds__(kBlock)
k_diag_partial(int n, const float4 *__restrict__ xr_c, const float2 *__restrict__ vel_a,
               double *__restrict__ partials)
{
    __shared__ double sh[3][kBlock / 32];
    double a = 0.0, b = 0.0, c = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 r = xr_c[i];
        const float2 v = vel_a[i];
        a += r.z;
        b += r.w;
        c += 0.5 * ((double)v.x * v.x + (double)v.y * v.y);
    }
    a = warp_sum(a); b = warp_sum(b); c = warp_sum(c);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sh[0][warp] = a; sh[1][warp] = b; sh[2][warp] = c; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s0 = 0, s1 = 0, s2 = 0;
        for (int w = 0; w < kBlock / 32; ++w) { s0 += sh[0][w]; s1 += sh[1][w]; s2 += sh[2][w]; }
        partials[3 * blockIdx.x] = s0;
        partials[3 * blockIdx.x + 1] = s1;
        partials[3 * blockIdx.x + 2] = s2;
    }
}

__global__ void k_diag_final(int nparts, int n, const double *__restrict__ partials, double *out)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double s0 = 0, s1 = 0, s2 = 0;
    for (int b = 0; b < nparts; ++b) {
        s0 += partials[3 * b];
        s1 += partials[3 * b + 1];
        s2 += partials[3 * b + 2];
    }
    out[0] = n ? s0 / n : 0.0;
    out[1] = n ? s1 / n : 0.0;
    out[2] = n ? s2 / n : 0.0;
}

constexpr int kDiagPiece = 2048;

// Per-scene FP64 sums, each scene cut into gridDim.y pieces (fixed order: the
// pieces' sums are added in theirs by k_diag_scenes_final).  One block a
// scene left the whole pass to the largest scene's block (64 scenes of 1,024
// to 65,536 particles: 200 us, so 45 us).  Where no scene is large enough to
// be cut its block writes the means itself (a call for two scenes of 2,048: 28
// us, 30 with the second kernel).  The density records are in C order and the
// velocities in A order; both keep every scene in its own slot range.
__global__ void __launch_bounds__(kBlock)
k_diag_scenes(Ctx c, const float4 *__restrict__ xr_c, const float2 *__restrict__ vel_a,
              double *__restrict__ partials, double *__restrict__ out)
{
    pdl_enter();
    __shared__ double sh[3][kBlock / 32];
    const int s = blockIdx.x;
    const int s0 = __ldg(c.p_off + s), s1 = __ldg(c.p_off + s + 1);
    // at least kDiagPiece particles a block: the block's own reduction is FP64
    // arithmetic too, which is what this pass is made of
    const int piece = max(kDiagPiece, (s1 - s0 + (int)gridDim.y - 1) / (int)gridDim.y);
    const bool whole = gridDim.y == 1;
    const int b0 = (int)min((long long)s1, s0 + (long long)blockIdx.y * piece), b1 = whole ? s1 : min(s1, b0 + piece);
    double *const at = whole ? out + 3 * s : partials + 3 * ((size_t)s * gridDim.y + blockIdx.y);
    if (b0 >= s1) {
        if (threadIdx.x < 3) at[threadIdx.x] = 0.0;
        return;
    }
    double a = 0.0, b = 0.0, k = 0.0;
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
        const float4 r = xr_c[i];
        const float2 v = vel_a[i];
        a += r.z;
        b += r.w;
        k += 0.5 * ((double)v.x * v.x + (double)v.y * v.y);
    }
    a = warp_sum(a); b = warp_sum(b); k = warp_sum(k);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sh[0][warp] = a; sh[1][warp] = b; sh[2][warp] = k; }
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[threadIdx.x][w];
        at[threadIdx.x] = whole ? t / (s1 - s0) : t;
    }
}

__global__ void __launch_bounds__(kBlock)
k_diag_scenes_final(Ctx c, int pieces, const double *__restrict__ partials, double *__restrict__ out)
{
    pdl_enter();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * c.nscenes) return;
    const int s = t / 3, q = t - 3 * s;
    double sum = 0.0;
    for (int p = 0; p < pieces; ++p) sum += partials[3 * ((size_t)s * pieces + p) + q];
    const int m = __ldg(c.p_off + s + 1) - __ldg(c.p_off + s);
    out[t] = m ? sum / m : 0.0;
}

// The reference's half list of one particle, in its order (hash.c:169-234):
// later members of its own cell, then the forward cells (0,+1), (+1,-1),
// (+1,0), (+1,+1), each in id order, r2 <= h2, cut at max_neighbors.
// WRITE = false counts, WRITE = true writes the entries at off[id], those of
// them in [lo, lo + m), to out[entry - lo] (and the counts, if asked, in the
// order of their ids, as suits host memory).
template <bool WRITE>
__global__ void __launch_bounds__(kBlock)
k_half_lists(Ctx c, const float2 *__restrict__ pos, const int *__restrict__ ids,
             const int *__restrict__ start, const unsigned *__restrict__ occ_in,
             unsigned *__restrict__ counts, const int *__restrict__ off, int *__restrict__ out,
             long long lo, long long m)
{
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    if (WRITE && counts) counts[i] = (unsigned)(off[i + 1] - off[i]);
    const Scene *S = c.scenes + scene_of(c, i);
    const SG g = load_grid(S);
    const float hh = __ldg(&S->P.smoothing_radius);
    const int max_neighbors = __ldg(&S->max_neighbors);
    const float h2 = __fmul_rn(hh, hh);
    const bool capped = *occ_in > (unsigned)c.max_bucket;
    const float2 p = pos[i];
    const unsigned key = cell_key(p.x, p.y, g);
    const int myid = ids[i];
    int cnum = 0;
    const long long first = WRITE ? off[myid] - lo : 0;
    if (WRITE && (first >= m || off[myid + 1] - lo <= 0)) return;
    if (searchable(key, i, start, g, capped, c.max_bucket)) {
        const int lk = (int)key - g.c_off;
        const int gy = lk / g.size_x, gx = lk - gy * g.size_x;
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const int x = gx + (f >= 2 ? 1 : 0);
            const int y = gy + (f == 0 ? 0 : (f == 1 ? 1 : f - 3));
            if (x < 0 || y < 0 || x >= g.size_x || y >= g.size_y) continue;
            const int cell = g.c_off + y * g.size_x + x;
            const int a = start[cell], e = start[cell + 1];
            const int b = capped && e - a > c.max_bucket ? a + c.max_bucket : e;
            for (int j = f == 0 ? i + 1 : a; j < b; ++j) {
                const float2 q = pos[j];
                if (dist2(p.x - q.x, p.y - q.y) > h2) continue;
                if (cnum < max_neighbors) {
                    if (WRITE && first + cnum >= 0 && first + cnum < m) out[first + cnum] = ids[j];
                    ++cnum;
                }
            }
        }
    }
    if (!WRITE) counts[myid] = (unsigned)cnum;
}

// ---------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------

static inline int blocks_for(int n, int bs = kBlock) { return (n + bs - 1) / bs; }

// Grid of a gather launch for shape s.
static inline dim3 gather_grid(const sph_cuda *h, const Shape &s)
{
    const int tiles = blocks_for(h->n, s.block);
    if (s.persistent <= 0) return dim3(tiles);
    const int p = h->num_sms * s.persistent;
    return dim3(p < tiles ? p : tiles);
}

// Exclusive scan of `in` (M entries) into out (M + 1 entries).  Both arrays
// must be 16-byte aligned: the scan kernels move 16-byte vectors.
int launch_prefix(sph_cuda *h, unsigned *in, int M, int *out, int *total)
{
    if (((uintptr_t)in | (uintptr_t)out) & 15u) {
        set_error("internal: scan arrays not 16-byte aligned");
        return SPH_ERR_INVALID;
    }
    const int tiles = (M + kScanTile - 1) / kScanTile;
    if (tiles > h->ntiles) {
        set_error("internal: scan of %d items exceeds the tile buffer", M);
        return SPH_ERR_INVALID;
    }
    launch_step(k_scan_reduce, tiles, kScanThreads, 0, h->stream, (const unsigned *)in, M,
                h->tile_sums);
    launch_step(k_scan_apply, tiles, kScanThreads, 0, h->stream, (const unsigned *)in, M,
                (const int *)h->tile_sums, out, total);
    return SPH_OK;
}

// The cell starts of a step's build (all M counters, zeroed after) into
// `out` (M + 1 entries); the build's key producer counted its particles per
// build tile into build_tiles, which the build's scatter zeroes again.
static int build_tiles_of(const sph_cuda *h) { return (h->M + kBuildTile - 1) / kBuildTile; }
// particles per thread of the step's scatter and permute
constexpr int kBuildPerThread = 2;

static void enqueue_cell_starts(sph_cuda *h, int *out, unsigned *occ)
{
    launch_step(k_cell_starts, build_tiles_of(h), kBuildThreads, 0, h->stream, h->cnt, h->M,
                (const unsigned *)h->d_nocell, (const unsigned *)h->build_tiles, out, h->d_state,
                occ, h->max_bucket, h->max_neighbors);
}

// Scatter and permutation of pos_b / vel_b (ids id_c, keys kr_b) into the A
// order by start_a; `end_step`: they end a step.  between() comes between.
template <class F>
static void enqueue_a_order(sph_cuda *h, DevState *end_step, F &&between)
{
    const int n = h->n, nbx = blocks_for(n, kBlock * kBuildPerThread);
    launch_step(k_scatter_ids_x<kBuildPerThread>, nbx, kBlock, 0, h->stream, n,
                (const uint2 *)h->kr_b, (const int *)h->id_c, (const int *)h->start_a, h->tmp_id,
                h->build_tiles, build_tiles_of(h));
    between();
    launch_step(k_permute_x<kBuildPerThread>, nbx, kBlock, 0, h->stream, n,
                (const uint2 *)h->kr_b, (const int *)h->start_a, (const int *)h->tmp_id,
                (const int *)h->id_c, (const float2 *)h->pos_b, (const float2 *)h->vel_b,
                h->id_a, h->pos_a, h->vel_a, end_step);
}

static const char *const kKernelNames[] = {
    "viscosity_predict", "cell_starts_1", "cell_scatter_1", "cell_permute_1", "density",
    "relax_update",      "cell_starts_2", "cell_scatter_2", "cell_permute_2"};
static const int kStepKernels = 9;
// A step with a learned model: density becomes the feature pass, then the
// network, then the relaxation with fallback.
static const char *const kLearnedKernelNames[] = {
    "viscosity_predict", "cell_starts_1",  "cell_scatter_1", "cell_permute_1",
    "features",          "mlp",            "relax_learned",  "relax_fallback",
    "cell_starts_2",     "cell_scatter_2", "cell_permute_2"};
static const int kLearnedStepKernels = 11;

// Lanes per particle of a handle's gathers, for states dense enough
// (lanes_min_occ): the fewer the particles, the more lanes it takes to fill
// the GPU.  The lines lie where two neighbouring choices cross over a dam
// break, in microseconds a step early / compressed: 32 and 16 lanes at 5,000
// particles 38.2 / 43.3 and 35.0 / 43.8, 16 and 8 at 12,500 45.2 / 66.5 and 41.5
// / 70.7 (at step 200 50.7 and 59.7), 8 and one thread at 40,000 59.8 / 95.1
// and 54.0 / 135, at 55,000 73 / 117 and 54 / 136.
static int lanes_for(int n)
{
    return n <= 5000 ? 32 : n <= 14000 ? 16 : n <= 40000 ? 8 : 1;
}

// The largest cell population from which gather k shares a particle among
// lanes: with one thread a particle a pass takes as long as its longest rows,
// with lanes as long as there are particles.  Below it the lanes' votes and
// shuffles cost more than the walk that they share, in the relaxation, which
// does the least per neighbour, first.  From a population whose rows may be
// too long for a hit mask on the rows are longest by far, and lanes pay in
// every handle that has them.  Microseconds a step with lanes and with one
// thread a particle, 14,000 / 28,000 / 40,000 particles at rest with a largest
// cell of 9 39.6 and 37.2 / 55.6 and 38.1 / 64.1 and 39.3, of 16 53.8 and 74.0 /
// 78.7 and 74.0 / 97.5 and 78.2; dam break at step 40 (18) 41.8 and 53.0 / 50.6
// and 52.7 / 59.8 and 54.0, at step 100 (28) 52.4 and 87.6 / 55.6 and 87.5 /
// 63.7 and 89.2.
static unsigned lanes_min_occ(int n, int k)
{
    constexpr int per[kGathers] = {1400, 2200, 800};
    return (unsigned)std::min(kMaskRow / 3 + 1, (n + per[k] - 1) / per[k]);
}

// A launch shape other than the default asks for the one-thread kernels.
static int gather_lanes(const sph_cuda *h, int k)
{
    if (h->shape[k].block != kBlock || h->shape[k].persistent != 0) return 1;
    return lanes_for(h->n);
}

// f(std::integral_constant<int, G>) for the G lanes of a group kernel.
template <class F>
static void with_lanes(int lanes, F &&f)
{
    switch (lanes) {
    case 32: f(std::integral_constant<int, 32>()); break;
    case 16: f(std::integral_constant<int, 16>()); break;
    default: f(std::integral_constant<int, 8>()); break;
    }
}

// Viscosity + prediction, the rebuild into the C order (kernels 0-3 of a step).
template <class Mark>
static void enqueue_predict_sort(sph_cuda *h, Mark &mark)
{
    const int n = h->n;
    const int nb = blocks_for(n);
    const Ctx c = make_ctx(h);
    DevState *st = h->d_state;
    const ViscArrays arrays{c, st, h->pos_a, h->vel_a, h->start_a, &st->build_max_occ[SLOT_RELAXED],
                            h->pos_b, h->prev_b, h->kr_b, h->cnt, nullptr};
    const int lanes = gather_lanes(h, 0);
    if (lanes > 1) {
        with_lanes(lanes, [&](auto G) {
            launch_step(k_viscosity_group<G.value>, blocks_for(n * G.value), kBlock, 0, h->stream, arrays,
                        &st->build_max_occ[SLOT_PREDICTED], lanes_min_occ(n, 0));
        });
    } else {
        auto kv = n <= kFewParticles ? (h->shape[0].persistent ? k_viscosity_predict_few<false, true>
                                                               : k_viscosity_predict_few<false, false>)
                                     : (h->shape[0].persistent ? k_viscosity_predict<false, true>
                                                               : k_viscosity_predict<false, false>);
        launch_step(kv, gather_grid(h, h->shape[0]), h->shape[0].block, 0, h->stream, arrays,
                    &st->build_max_occ[SLOT_PREDICTED]);
    }
    mark();
    enqueue_cell_starts(h, h->start_c, &st->build_max_occ[SLOT_PREDICTED]);
    mark();
    const int nbx = blocks_for(n, kBlock * kBuildPerThread);
    launch_step(k_scatter_ids_x<kBuildPerThread>, nbx, kBlock, 0, h->stream, n,
                (const uint2 *)h->kr_b, (const int *)h->id_a, (const int *)h->start_c, h->tmp_id,
                h->build_tiles, build_tiles_of(h));
    mark();
    launch_step(k_permute_x<kBuildPerThread>, nbx, kBlock, 0, h->stream, n,
                (const uint2 *)h->kr_b, (const int *)h->start_c, (const int *)h->tmp_id,
                (const int *)h->id_a, (const float2 *)h->pos_b, (const float2 *)h->prev_b,
                h->id_c, h->pos_c, h->prev_c, (DevState *)nullptr);
    mark();
}

static void enqueue_density(sph_cuda *h)
{
    const DensArrays arrays{make_ctx(h), h->pos_c, h->start_c,
                            &h->d_state->build_max_occ[SLOT_PREDICTED], h->xr_c, h->mask01_c,
                            h->mask2_c, h->rows_c, DensityById()};
    const int lanes = gather_lanes(h, 1);
    if (lanes > 1) {
        with_lanes(lanes, [&](auto G) {
            launch_step(h->long_masks ? k_density_group<G.value, true> : k_density_group<G.value, false>,
                        blocks_for(h->n * G.value), kBlock, 0, h->stream, arrays, lanes_min_occ(h->n, 1));
        });
        return;
    }
    auto kd = h->shape[1].persistent
                  ? (h->long_masks ? k_density_t<true, true> : k_density_t<true, false>)
                  : (h->long_masks ? k_density_t<false, true> : k_density_t<false, false>);
    launch_step(kd, gather_grid(h, h->shape[1]), h->shape[1].block, 0, h->stream, arrays);
}

// The density pass of a step (the learned step's features start with it).
int launch_density_pass(sph_cuda *h)
{
    if (h->n == 0) return SPH_OK;
    enqueue_density(h);
    return cuda_fail(cudaGetLastError(), "density");
}

// The C-order state of the next step's relaxation -- predicted positions,
// their cell starts, density records and hit masks -- without advancing:
// the A state is left as it is (the last step's density record in xr_c is
// replaced).
int enqueue_predicted_state(sph_cuda *h)
{
    if (h->n == 0) return SPH_OK;
    auto none = []() {};
    enqueue_predict_sort(h, none);
    enqueue_density(h);
    const int rc = cuda_fail(cudaGetLastError(), "predicted state");
    h->cells_dirty |= rc != SPH_OK;
    return rc;
}

// The relaxation of a step: the C order's density records to the B arrays.
static RelaxArrays relax_arrays(const sph_cuda *h, float2 *probe_out = nullptr)
{
    return RelaxArrays{make_ctx(h), h->xr_c, h->mask01_c, h->mask2_c, h->rows_c, h->prev_c,
                       h->id_c, h->start_c, &h->d_state->build_max_occ[SLOT_PREDICTED], h->pos_b,
                       h->vel_b, h->kr_b, h->cnt, probe_out};
}

// The relaxation passes of a learned step (network particles, then the
// fallback list); with probe_out, one pass writes every particle's
// displacement (C order) instead of advancing.  `events` (two) are recorded
// after each pass.
int launch_learned_relax(sph_cuda *h, float2 *probe_out, cudaEvent_t *events)
{
    const Ctx c = make_ctx(h);
    DevState *st = h->d_state;
    LearnedIn L;
    L.net = h->net_c;
    L.nbc = h->nbc_c;
    L.thr_pct = h->learned_thr * 100.0f;
    // a negative threshold sends every particle to the plain relaxation
    L.max_nb = h->learned_thr < 0.0f ? -1 : SPH_LEARNED_MAX_NEIGHBORS;
    const int nb = blocks_for(h->n);
    const bool lm = h->long_masks;
    const RelaxArrays arrays = relax_arrays(h, probe_out);
    if (probe_out) {
        (lm ? k_relax_learned<true, true>
            : k_relax_learned<true, false>)<<<nb, kBlock, 0, h->stream>>>(arrays, nullptr, L, st, nullptr);
        return cuda_fail(cudaGetLastError(), "learned relaxation probe");
    }
    (lm ? k_relax_learned<false, true> : k_relax_learned<false, false>)<<<nb, kBlock, 0, h->stream>>>(
        arrays, &st->build_max_occ[SLOT_RELAXED], L, st, h->fb_list);
    if (events) cudaEventRecord(events[0], h->stream);
    const int fb_blocks = kFallbackWaves * kFallbackCtas * h->num_sms;
    (lm ? k_relax_fallback<true> : k_relax_fallback<false>)<<<fb_blocks, kBlock, 0, h->stream>>>(
        arrays, st, h->fb_list);
    if (events) cudaEventRecord(events[1], h->stream);
    return cuda_fail(cudaGetLastError(), "learned relaxation");
}

// Queues one step.  With `events` (one per kernel + 1) each kernel is
// bracketed for timing.  With `mid_tp`, the scene's tunables are replaced
// by *mid_tp after the first half (gravity, viscosity, prediction and the
// cell build of the predicted positions) and before the density pass, the
// relaxation and the velocity update -- where the reference's compute rank
// receives new tunables inside a step (fluid.c:293-294, between
// predict_positions at :279 and hash_fluid at :315).  Single-scene handles.
static int enqueue_step_kernels(sph_cuda *h, cudaEvent_t *events, int *nkernels,
                                const tunable_parameters *mid_tp)
{
    const int n = h->n;
    const int nb = blocks_for(n);
    const Ctx c = make_ctx(h);
    DevState *st = h->d_state;
    int e = 0;
    auto mark = [&]() {
        if (events) cudaEventRecord(events[e], h->stream);
        ++e;
    };
    mark();
    enqueue_predict_sort(h, mark);
    if (mid_tp) {
        const int rc = set_scene_params(h, 0, mid_tp);
        if (rc != SPH_OK) return rc;
    }
    if (h->learned) {
        int rc = launch_learned_passes(h, events ? events + e : nullptr);
        if (rc != SPH_OK) return rc;
        e += 2;
        rc = launch_learned_relax(h, nullptr, events ? events + e : nullptr);
        if (rc != SPH_OK) return rc;
        e += 2;
    } else {
        enqueue_density(h);
        mark();
        const int lanes = gather_lanes(h, 2);
        if (lanes > 1) {
            with_lanes(lanes, [&](auto G) {
                launch_step(h->long_masks ? k_relax_group<G.value, true> : k_relax_group<G.value, false>,
                            blocks_for(n * G.value), kBlock, 0, h->stream, relax_arrays(h),
                            &st->build_max_occ[SLOT_RELAXED], lanes_min_occ(n, 2));
            });
        } else {
            auto kr = h->shape[2].persistent
                          ? (h->long_masks ? k_relax_update<false, true, true>
                                           : k_relax_update<false, true, false>)
                          : (h->long_masks ? k_relax_update<false, false, true>
                                           : k_relax_update<false, false, false>);
            launch_step(kr, gather_grid(h, h->shape[2]), h->shape[2].block, 0, h->stream, relax_arrays(h),
                        &st->build_max_occ[SLOT_RELAXED]);
        }
        mark();
    }
    enqueue_cell_starts(h, h->start_a, &st->build_max_occ[SLOT_RELAXED]);
    mark();
    enqueue_a_order(h, st, mark);
    mark();
    if (nkernels) *nkernels = e - 1;
    return cuda_fail(cudaGetLastError(), "step launch");
}

int enqueue_step(sph_cuda *h, cudaEvent_t *events, int *nkernels, const tunable_parameters *mid_tp)
{
    const int rc = enqueue_step_kernels(h, events, nkernels, mid_tp);
    h->cells_dirty |= rc != SPH_OK;
    return rc;
}

unsigned bounds_flags_kernels() { return read_bounds_flag(); }

const char *kernel_name(int k)
{
    return (k >= 0 && k < kStepKernels) ? kKernelNames[k] : "";
}
const char *step_kernel_name(const sph_cuda *h, int k)
{
    if (h && h->learned) return (k >= 0 && k < kLearnedStepKernels) ? kLearnedKernelNames[k] : "";
    return kernel_name(k);
}
int step_kernel_count() { return kStepKernels; }
int step_kernel_count(const sph_cuda *h)
{
    return (h && h->learned) ? kLearnedStepKernels : kStepKernels;
}

// Particles to upload -> the upload arrays in id order (pos_b, vel_b, prev_c
// and xr_c = (x, y, rho, rho_near)), from structure-of-arrays (vx, vy may be
// null: zero), from the reference's fluid_particle records, or in place
// already, with their cell keys counted into the build that sorts them, in
// one kernel (layout, ids and keys were three, and the sort that followed
// four more without programmatic launch).
__global__ void __launch_bounds__(kBlock)
k_upload(Ctx c, UploadSource src, float2 *__restrict__ pos, float2 *__restrict__ vel,
         float2 *__restrict__ prev, float4 *__restrict__ xr, int *__restrict__ id,
         uint2 *__restrict__ kr, unsigned *__restrict__ cnt, unsigned *occ_reset)
{
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *occ_reset = 0u;
    int t = -1;
    if (i < c.n) {
        float2 p;
        if (src.x) {
            p = make_float2(src.x[i], src.y[i]);
            pos[i] = p;
            vel[i] = make_float2(src.vx ? src.vx[i] : 0.0f, src.vy ? src.vy[i] : 0.0f);
            prev[i] = p;
            xr[i] = make_float4(p.x, p.y, 0.0f, 0.0f);
        } else if (src.recs) {
            const fluid_particle &q = src.recs[i];
            p = make_float2(q.x, q.y);
            pos[i] = p;
            vel[i] = make_float2(q.v_x, q.v_y);
            prev[i] = make_float2(q.x_prev, q.y_prev);
            xr[i] = make_float4(q.x, q.y, q.density, q.density_near);
        } else {
            p = pos[i];
        }
        id[i] = i;
        const unsigned key = cell_key(p.x, p.y, load_grid(c.scenes + scene_of(c, i)));
        unsigned rank = 0u;
        if (in_bounds(key, c.M, kBadKey)) {
            rank = atomicAdd(cnt + key, 1u);
            t = (int)(key / (unsigned)kBuildTile);
        }
        kr[i] = make_uint2(key, rank);
    }
    cta_tile_count(c.tile_cnt, t);
}

// The id-order records of k_unpermute (pos, vel, prev, (rho, rho_near),
// pressures; n float2 each) -> six float arrays x, y, vx, vy, rho, rho_near
// (n each; null: not wanted), which may be the caller's own.
__global__ void __launch_bounds__(kBlock)
k_split_soa(int n, const float2 *__restrict__ rec, SoaColumns out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t m = (size_t)n;
    const float2 p = rec[i], v = rec[m + i], r = rec[3 * m + i];
    const float f[6] = {p.x, p.y, v.x, v.y, r.x, r.y};
#pragma unroll
    for (int k = 0; k < 6; ++k)
        if (out.c[k]) out.c[k][i] = f[k];
}

int launch_split_soa(sph_cuda *h, int n, const float2 *rec, const SoaColumns &out)
{
    if (n == 0) return SPH_OK;
    k_split_soa<<<blocks_for(n), kBlock, 0, h->stream>>>(n, rec, out);
    return cuda_fail(cudaGetLastError(), "split");
}

__global__ void k_enable_lists(DevState *st) { st->lists_valid = 1u; }

int launch_enable_lists(sph_cuda *h)
{
    k_enable_lists<<<1, 1, 0, h->stream>>>(h->d_state);
    return cuda_fail(cudaGetLastError(), "neighbour lists");
}

// Uploaded particles -> sorted A state; prev_c / xr_c hold the uploaded values
// in id order.
int upload_device(sph_cuda *h, int n, const UploadSource &src)
{
    if (n == 0) return SPH_OK;
    DevState *st = h->d_state;
    // a fresh state starts every build from zero tile counts and cell
    // counters, whatever an interrupted step left: k_cell_starts looks at the
    // counters of the counted tiles alone, and zeroes them itself
    cudaMemsetAsync(h->build_tiles, 0, (size_t)h->ntiles * sizeof(unsigned), h->stream);
    if (h->cells_dirty) cudaMemsetAsync(h->cnt, 0, (size_t)h->M * sizeof(unsigned), h->stream);
    launch_step(k_upload, blocks_for(n), kBlock, 0, h->stream, make_ctx(h), src, h->pos_b, h->vel_b,
                h->prev_c, h->xr_c, h->id_c, h->kr_b, h->cnt, &st->build_max_occ[SLOT_RELAXED]);
    cudaEventRecord(h->host_ev, h->stream);  // the source has been read
    enqueue_cell_starts(h, h->start_a, &st->build_max_occ[SLOT_RELAXED]);
    enqueue_a_order(h, nullptr, [] {});
    const int rc = cuda_fail(cudaGetLastError(), "upload kernels");
    h->cells_dirty = rc != SPH_OK;
    return rc;
}

int launch_unpermute(sph_cuda *h, float2 *out)
{
    if (h->n == 0) return SPH_OK;
    k_unpermute<<<blocks_for(h->n), kBlock, 0, h->stream>>>(make_ctx(h), h->id_a, h->pos_a,
                                                            h->vel_a, h->id_c, h->prev_c, h->xr_c,
                                                            out);
    return cuda_fail(cudaGetLastError(), "unpermute");
}

int launch_pack(sph_cuda *h, short2 *out)
{
    if (h->n == 0) return SPH_OK;
    k_pack_coords<<<blocks_for(h->n), kBlock, 0, h->stream>>>(make_ctx(h), h->id_a, h->pos_a, out);
    return cuda_fail(cudaGetLastError(), "pack coords");
}

int launch_diagnostics(sph_cuda *h, double *d_out)
{
    const int parts = h->npartials;
    k_diag_partial<<<parts, kBlock, 0, h->stream>>>(h->n, h->xr_c, h->vel_a, h->d_partials);
    k_diag_final<<<1, 32, 0, h->stream>>>(parts, h->n, h->d_partials, d_out);
    return cuda_fail(cudaGetLastError(), "diagnostics");
}

// Pieces a scene is summed in at most: of kDiagPiece particles of the largest
// scene, a few waves of the GPU in all.
int scene_diagnostic_pieces(const sph_cuda *h)
{
    int largest = 1;
    for (const Scene &s : h->scenes) largest = std::max(largest, s.n);
    const int fill = std::max(1, 16 * h->num_sms / h->nscenes);
    return std::min({64, fill, (largest + kDiagPiece - 1) / kDiagPiece});
}

// out: 3 nscenes means; partials: 3 nscenes x scene_diagnostic_pieces.
int launch_scene_diagnostics(sph_cuda *h, double *d_out, double *partials)
{
    if (h->nscenes == 0) return SPH_OK;
    const Ctx c = make_ctx(h);
    const int pieces = scene_diagnostic_pieces(h);
    launch_step(k_diag_scenes, dim3(h->nscenes, pieces), kBlock, 0, h->stream, c, (const float4 *)h->xr_c,
                (const float2 *)h->vel_a, partials, d_out);
    if (pieces > 1)
        launch_step(k_diag_scenes_final, blocks_for(3 * h->nscenes), kBlock, 0, h->stream, c, pieces,
                    (const double *)partials, d_out);
    return cuda_fail(cudaGetLastError(), "scene diagnostics");
}

// Probes on the A state.  which: 0 density, 1 relaxation displacement,
// 2 viscosity velocity change.  `scratch` (probe_scratch_bytes(n), 256-byte
// aligned) holds the sorted records; out: n float2 by id (device).
size_t probe_scratch_bytes(int n)
{
    const size_t a = ((size_t)n * 16 + 255) & ~(size_t)255;
    return 4 * a + (((size_t)n * 8 + 255) & ~(size_t)255);
}

int launch_probe(sph_cuda *h, int which, void *scratch, float2 *out)
{
    const int n = h->n;
    if (n == 0) return SPH_OK;
    const int nb = blocks_for(n);
    const Ctx c = make_ctx(h);
    DevState *st = h->d_state;
    const unsigned *occ = &st->build_max_occ[SLOT_RELAXED];
    const size_t a = ((size_t)n * 16 + 255) & ~(size_t)255;
    char *base = (char *)scratch;
    float4 *xr = (float4 *)base;
    ulonglong2 *m01 = (ulonglong2 *)(base + a);
    unsigned long long *m2 = (unsigned long long *)(base + 2 * a);
    int4 *rw = (int4 *)(base + 3 * a);
    float2 *sorted = (float2 *)(base + 4 * a);
    if (which == 0 || which == 1) {
        k_density<<<nb, kBlock, 0, h->stream>>>(
            DensArrays{c, h->pos_a, h->start_a, occ, xr, m01, m2, rw, DensityById()});
        if (which == 1)
            k_relax_update<true><<<nb, kBlock, 0, h->stream>>>(
                RelaxArrays{c, xr, m01, m2, rw, nullptr, h->id_a, h->start_a, occ, nullptr, nullptr,
                            nullptr, nullptr, sorted},
                nullptr);
        else
            k_xr_density<<<nb, kBlock, 0, h->stream>>>(n, xr, sorted);
    } else {
        (n <= kFewParticles ? k_viscosity_predict_few<true> : k_viscosity_predict<true>)<<<nb, kBlock, 0, h->stream>>>(
            ViscArrays{c, st, h->pos_a, h->vel_a, h->start_a, occ, nullptr, nullptr, nullptr, nullptr, sorted},
            nullptr);
    }
    k_by_id<<<nb, kBlock, 0, h->stream>>>(n, h->id_a, sorted, out);
    return cuda_fail(cudaGetLastError(), "probe");
}

// Half lists in the reference's order on the A state: the counts by id and
// their prefix sums (d_counts: n words, d_off: n + 1 ints, both 16-byte
// aligned; total_out: as launch_prefix), or the entries [lo, lo + m) of the
// lists (and, with counts_out, the counts once more, for host memory).
int launch_half_list_counts(sph_cuda *h, unsigned *d_counts, int *d_off, int *total_out)
{
    const int n = h->n;
    if (n == 0) return SPH_OK;
    k_half_lists<false><<<blocks_for(n), kBlock, 0, h->stream>>>(
        make_ctx(h), h->pos_a, h->id_a, h->start_a, &h->d_state->build_max_occ[SLOT_RELAXED], d_counts,
        nullptr, nullptr, 0, 0);
    const int rc = launch_prefix(h, d_counts, n, d_off, total_out);
    return rc != SPH_OK ? rc : cuda_fail(cudaGetLastError(), "half list counts");
}

int launch_half_lists(sph_cuda *h, const int *d_off, int *d_ids, long long lo, long long m,
                      unsigned *counts_out)
{
    if (h->n == 0) return SPH_OK;
    launch_step(k_half_lists<true>, blocks_for(h->n), kBlock, 0, h->stream, make_ctx(h),
                (const float2 *)h->pos_a, (const int *)h->id_a, (const int *)h->start_a,
                (const unsigned *)&h->d_state->build_max_occ[SLOT_RELAXED], counts_out, d_off,
                d_ids, lo, m);
    return cuda_fail(cudaGetLastError(), "half lists");
}

// ---------------------------------------------------------------------------
// the density of caller-owned arrays (sph_cuda_density_static)
// ---------------------------------------------------------------------------

// Everything a call starts from: zero counters and tile counts, a fresh
// state, the scene table and its no-cell bitmap.
__global__ void __launch_bounds__(kBlock)
k_static_init(Scene s, StaticArrays a, int ntiles)
{
    pdl_trigger();  // the keys may fetch the caller's positions meanwhile
    const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const int M = s.ncells + 1;
    for (int i = t; i < M; i += nt) a.cnt[i] = 0u;
    for (int i = t; i < ntiles; i += nt) a.tile_cnt[i] = 0u;
    for (int i = t; i < (M + 31) / 32; i += nt)
        a.nocell[i] = i == s.ncells >> 5 ? 1u << (s.ncells & 31) : 0u;
    if (t == 0) {
        *a.scene = s;
        a.p_off[0] = 0;
        a.p_off[1] = s.n;
        *a.state = DevState{};
    }
}

// Positions and cell keys of the caller's arrays.
__global__ void __launch_bounds__(kBlock)
k_static_keys(Ctx c, SG g, const float *__restrict__ x, const float *__restrict__ y,
              float2 *__restrict__ pos, uint2 *__restrict__ kr, unsigned *__restrict__ cnt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float2 p = make_float2(0.0f, 0.0f);
    if (i < c.n) p = make_float2(__ldg(x + i), __ldg(y + i));  // the caller's: complete before the call
    pdl_enter();
    if (i >= c.n) return;
    const unsigned key = cell_key(p.x, p.y, g);
    unsigned rank = 0u;
    if (in_bounds(key, c.M, kBadKey)) {
        rank = atomicAdd(cnt + key, 1u);
        add_tile_count(c.tile_cnt, key);
    }
    pos[i] = p;
    kr[i] = make_uint2(key, rank);
}

template <int G>
__global__ void __launch_bounds__(kBlock)
k_density_static(const __grid_constant__ DensArrays A, unsigned min_occ)
{
    pdl_enter();
    const int th = blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (G > 1) {
        if (!shared_by_lanes(A, min_occ)) {
            if (th < A.c.n) density_one<false, true>(th, A);
            return;
        }
        const Group<G> g;
        const bool valid = th / G < A.c.n;
        const int i = valid ? th / G : A.c.n - 1;
        density_group_one<G, false, true>(g, i, valid, A);
    } else if (th < A.c.n) {
        density_one<false, true>(th, A);
    }
}

// Six kernels, the first launched as usual, each of the others while its
// predecessor still runs (programmatic launch): zeroing, keys, cell starts,
// scatter, permute, density by id.  With three memsets, nine kernels and a
// full drain between each two, 65,521 particles took 58 us, so 23 us.
int launch_static_density(const Scene &sc, const StaticArrays &a, const float *x, const float *y,
                          float *rho, float *rho_near, cudaStream_t st)
{
    Ctx c;
    c.scenes = a.scene;
    c.p_off = a.p_off;
    c.nscenes = 1;
    c.n = sc.n;
    c.max_bucket = sc.max_bucket;
    c.M = sc.ncells + 1;
    c.tile_cnt = a.tile_cnt;
    SG g;
    g.spacing = sc.spacing;
    g.inv = exact_reciprocal(sc.spacing);
    g.size_x = sc.size_x;
    g.size_y = sc.size_y;
    g.ncells = sc.ncells;
    g.c_off = 0;
    const int n = sc.n, nb = blocks_for(n), nbx = blocks_for(n, kBlock * kBuildPerThread);
    const int ntiles = (c.M + kBuildTile - 1) / kBuildTile;
    unsigned *occ = &a.state->build_max_occ[SLOT_PROBE];
    k_static_init<<<blocks_for(c.M, kBlock * 4), kBlock, 0, st>>>(sc, a, ntiles);
    launch_step(k_static_keys, nb, kBlock, 0, st, c, g, x, y, a.pos_in, a.kr, a.cnt);
    launch_step(k_cell_starts, ntiles, kBuildThreads, 0, st, a.cnt, c.M, (const unsigned *)a.nocell,
                (const unsigned *)a.tile_cnt, a.start, a.state, occ, sc.max_bucket, sc.max_neighbors);
    launch_step(k_scatter_ids_x<kBuildPerThread>, nbx, kBlock, 0, st, n, (const uint2 *)a.kr,
                (const int *)nullptr, (const int *)a.start, a.tmp, a.tile_cnt, ntiles);
    launch_step(k_permute_x<kBuildPerThread>, nbx, kBlock, 0, st, n, (const uint2 *)a.kr,
                (const int *)a.start, (const int *)a.tmp, (const int *)nullptr,
                (const float2 *)a.pos_in, (const float2 *)nullptr, a.id_s, a.pos_s,
                (float2 *)nullptr, (DevState *)nullptr);
    const DensArrays arrays{c, a.pos_s, a.start, occ, nullptr, nullptr, nullptr, nullptr,
                            DensityById{a.id_s, rho, rho_near}};
    const int lanes = lanes_for(n);
    if (lanes > 1) {
        with_lanes(lanes, [&](auto G) {
            launch_step(k_density_static<G.value>, blocks_for(n * G.value), kBlock, 0, st, arrays,
                        lanes_min_occ(n, 1));
        });
    } else {
        launch_step(k_density_static<1>, nb, kBlock, 0, st, arrays, 0u);
    }
    return cuda_fail(cudaGetLastError(), "sph_cuda_density_static launch");
}

}  // namespace sph
