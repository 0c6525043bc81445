// sph_learned.cu -- learned relaxation (include/sph_learned.h).
//
//   k_messages   after the plain density pass: a walk of its hit masks that
//                aggregates the neighbour messages (offsets, velocities,
//                densities and near densities) -> 32-wide BF16 feature rows
//                and neighbour counts
//   k_mlp        fused 2-layer width-128 GELU MLP on the tcgen05 tensor cores:
//                one CTA per SM of four 256-thread pipelines, weights
//                resident in shared memory, FP32 accumulators in tensor memory
//   (k_relax_learned then applies the network's displacement and lists the
//    particles that take the plain relaxation for k_relax_fallback)
//
// Training: k_train, the forward and backward pass of a batch on the tensor
// cores (a tile of 128 samples at a time), k_grad, the weight gradients in the
// samples' order, k_adam on FP32 master weights; sample collection and the
// calibration of the error output.
#include <algorithm>
#include <cstddef>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda_bf16.h>

#include "sph_device.cuh"
#include "sph_learned.h"
#include "sph_tc.cuh"


namespace sph {

int launch_probe(sph_cuda *h, int which, void *scratch, float2 *out);
size_t probe_scratch_bytes(int n);
int ensure_scratch(sph_cuda *h, size_t bytes);

namespace ml {

constexpr int IN = SPH_LEARNED_IN, HID = SPH_LEARNED_HIDDEN, OUT = SPH_LEARNED_OUT;
constexpr int MAXNB = SPH_LEARNED_MAX_NEIGHBORS;

// Flat parameter layout: W1 [HID x IN], b1, W2 [HID x HID], b2, W3 [OUT x HID], b3.
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + HID * IN;
constexpr int OFF_W2 = OFF_B1 + HID;
constexpr int OFF_B2 = OFF_W2 + HID * HID;
constexpr int OFF_W3 = OFF_B2 + HID;
constexpr int OFF_B3 = OFF_W3 + OUT * HID;
constexpr int NPARAM = OFF_B3 + OUT;

// Outputs used: 0, 1 displacement / s; 2 predicted density error in % of rho0.

// Derivative of the activation 2 GELU (tanh form).
__device__ __forceinline__ float act_grad(float x)
{
    float t;
    const float u = 0.7978845608f * (x + 0.044715f * x * x * x);
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
    return (1.0f + t) + x * (1.0f - t * t) * 0.7978845608f * (1.0f + 0.134145f * x * x);
}

// Output scale of a scene: s = h dt^2 (k + k_near + k_spring).
__device__ __forceinline__ float out_scale(const Scene *__restrict__ S)
{
    const float dt = __ldg(&S->P.time_step), h = __ldg(&S->P.smoothing_radius);
    return h * dt * dt * (__ldg(&S->P.k) + __ldg(&S->P.k_near) + __ldg(&S->P.k_spring));
}

// ---------------------------------------------------------------------------
// message pass
// ---------------------------------------------------------------------------

// A neighbour's record for the message walk: (x, y, rho, rho_near) and its
// previous position.
struct NbRec {
    float4 q;
    float2 qp;
};

// Whether a particle has more than max_nb neighbours: the hits of its masks,
// or, where a row is too long for them, its candidates counted until there
// are more.  A step asks first: the relaxation does not look at the network's
// output for such a particle, and these are the longest walks of all (the dam
// break's 1,048,576 particles: density and messages 154 -> 131 us with 9% of
// them, 299 -> 184 us with 29%).
__device__ __forceinline__ bool more_hits_than(int max_nb, int i, const Ctx &c, const Scene *S,
                                               bool lm, float2 p, float h2,
                                               const float4 *__restrict__ xr,
                                               const int *__restrict__ start, const int4 &rw,
                                               const ulonglong2 &m01, unsigned long long m2)
{
    if (rw.w != kRowsFull) {
        int count = __popcll(m01.x) + __popcll(m01.y) + __popcll(m2);
        if (lm && rw.w == kRowsMasked2) {
            const unsigned long long *mx = c.maskx + 3 * (size_t)i;
            count += __popcll(__ldg(mx)) + __popcll(__ldg(mx + 1)) + __popcll(__ldg(mx + 2));
        }
        return count > max_nb;
    }
    const SG g = load_grid(S);
    int ra[3], rl[3], count = -1;  // not the particle itself
    stencil_rows(p, cell_key(p.x, p.y, g), start, g, ra, rl, c.n);
#pragma unroll 1
    for (int r = 0; r < 3; ++r)
#pragma unroll 4
        for (int j = ra[r]; j < ra[r] + rl[r]; ++j) {
            const float4 q = __ldg(xr + j);
            float2 e;
            if (dist2_packed(make_float2(-p.x, -p.y), make_float2(q.x, q.y), e) <= h2 &&
                ++count > max_nb)
                return true;
        }
    return false;
}

// The particle's feature row, from the plain density pass's records (its
// (x, y, rho, rho_near), hit masks and stencil-row record, all in C order):
// messages of the neighbours j with r/h < 1 (self excluded),
// u = unit offset towards the neighbour, w = 1 - r/h,
// dv = (v_j - v_i) dt / h with v = (x - x_prev) / dt:
//   V1 = sum w u, V2 = sum w^2 u, M = sum w, T = sum w u u^T, D = sum w dv,
//   R1 = sum w (rho_j - rest) u, R2 = sum w^2 rho_near_j u
// (the neighbours' densities and near densities, as the relaxation's pair
// term uses them, fluid.c:588-608), with the particle's rho, rho_near,
// neighbour count (r2 <= h2), its scene's stiffness ratios a_k, a_n, a_s
// (k, k_near, k_spring over their sum) and the "own" terms of the
// relaxation formula a_k (rho - rest) V1, a_n rho_near V2, a_s V1.  A
// particle with a coincident neighbour (r2 <= 2e-12, where the reference
// nudges) or in an overflowing bucket gets count 65535: it always takes the
// plain relaxation.  Block 0 resets the step's fallback-list counters.
template <bool LM>
__global__ void __maxnreg__(56)
k_messages(Ctx c, const float4 *__restrict__ xr, const ulonglong2 *__restrict__ mask01,
           const unsigned long long *__restrict__ mask2, const int4 *__restrict__ rows,
           const float2 *__restrict__ prev, const int *__restrict__ start,
           const unsigned *__restrict__ occ_in, __nv_bfloat16 *__restrict__ feat,
           unsigned short *__restrict__ nbcount, unsigned *__restrict__ fb_count, int max_nb)
{
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 && fb_count) {  // both fallback counters of the step (fb_count, fb_long)
        fb_count[0] = 0u;
        fb_count[1] = 0u;
    }
    if (i >= c.n) return;
    // the particle's streams, requested together
    const float4 me = xr[i];
    const int4 rw = __ldg(rows + i);
    const ulonglong2 m01 = __ldg(mask01 + i);
    const unsigned long long m2 = __ldg(mask2 + i);
    const float2 pp = prev[i];
    const Scene *S = c.scenes + scene_of(c, i);
    const float hh = __ldg(&S->P.smoothing_radius);
    const float h2 = __fmul_rn(hh, hh);
    const float h_recip = __fdiv_rn(1.0f, hh);
    const float dt = __ldg(&S->P.time_step);
    const float inv_dt = 1.0f / dt;
    const float vscale = dt * h_recip;
    const float rest = __ldg(&S->P.rest_density);
    const bool capped = *occ_in > (unsigned)c.max_bucket;
    const float2 p = make_float2(me.x, me.y);
    const float vix = (p.x - pp.x) * inv_dt, viy = (p.y - pp.y) * inv_dt;
    const float2 mp = make_float2(-p.x, -p.y);
    if (max_nb < INT_MAX && !capped && rw.w != kRowsNone &&
        more_hits_than(max_nb, i, c, S, LM, p, h2, xr, start, rw, m01, m2)) {
        nbcount[i] = 65535;  // the plain relaxation takes it: no row of features
        return;
    }
    float2 V1 = make_float2(0.0f, 0.0f), V2 = V1, Tdiag = V1, Dsum = V1, R1 = V1, R2 = V1;
    float Ms = 0.0f, Txy = 0.0f;
    int count = 0;
    bool degenerate = capped;
    // one neighbour (r2 <= h2 known, never the particle itself)
    auto visit = [&](int, const NbRec &d) {
        float2 e;  // q - p
        const float r2 = dist2_packed(mp, make_float2(d.q.x, d.q.y), e);
        float rinv = rsqrt_normal(r2);
        ++count;
        if (r2 <= 2e-12f) {
            degenerate = true;
            rinv = rsqrtf(r2);
        }
        const float ratio = r2 * rinv * h_recip;
        if (ratio < 1.0f) {
            const float omr = 1.0f - ratio;
            const float omr2 = omr * omr;
            // message sums in packed FP32x2 arithmetic
            const float2 u = __fmul2_rn(e, make_float2(rinv, rinv));
            const float2 w2 = make_float2(omr, omr);
            const float2 wu = __fmul2_rn(w2, u);
            V1 = __fadd2_rn(V1, wu);
            V2 = __ffma2_rn(make_float2(omr2, omr2), u, V2);
            Ms += omr;
            Tdiag = __ffma2_rn(wu, u, Tdiag);
            Txy += wu.x * u.y;
            const float pr = d.q.z - rest, prn = omr2 * d.q.w;
            R1 = __ffma2_rn(make_float2(pr, pr), wu, R1);
            R2 = __ffma2_rn(make_float2(prn, prn), u, R2);
            // sum w (x_j - x_prev_j); the velocities follow at the end
            Dsum = __ffma2_rn(w2, __fadd2_rn(make_float2(d.q.x, d.q.y),
                                             make_float2(-d.qp.x, -d.qp.y)), Dsum);
        }
    };
    auto load = [&](int j) {
        NbRec d;
        d.q = __ldg(xr + j);
        d.qp = __ldg(prev + j);
        return d;
    };
    if (!capped && rw.w == kRowsMasked) {
        const int ra[3] = {rw.x, rw.y, rw.z};
        const unsigned long long mm[3] = {m01.x, m01.y, m2};
        walk_rows<NbRec>(mm, ra, c.n, load, visit);
    } else if (LM && !capped && rw.w == kRowsMasked2) {
        // long-row masks: each row's two masks in slot order
        const int ra[3] = {rw.x, rw.y, rw.z};
        const unsigned long long mm[3] = {m01.x, m01.y, m2};
        const unsigned long long *mx = c.maskx + 3 * (size_t)i;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            walk_mask<NbRec>(mm[r], ra[r], c.n, load, visit);
            walk_mask<NbRec>(__ldg(mx + r), ra[r] + kMaskRow, c.n, load, visit);
        }
    } else if (!capped && rw.w == kRowsFull) {
        // a stencil row longer than a hit mask: the whole stencil, in slot
        // order
        const SG g = load_grid(S);
        const unsigned key = cell_key(p.x, p.y, g);
        for_each_candidate(key, start, g, false, c.max_bucket, c.n, [&](int j) {
            if (j == i) return;
            const NbRec d = load(j);
            float2 e;
            if (dist2_packed(mp, make_float2(d.q.x, d.q.y), e) > h2) return;
            visit(j, d);
        });
    }
    nbcount[i] = degenerate ? (unsigned short)65535 : (unsigned short)(count < 65534 ? count : 65534);
    const float a = me.z, b = me.w;
    const float V1x = V1.x, V1y = V1.y, V2x = V2.x, V2y = V2.y;
    const float Txx = Tdiag.x, Tyy = Tdiag.y;
    // sum w (v_j - v_i) = (sum w (x_j - x_prev_j)) / dt - v_i sum w
    const float Dx = Dsum.x * inv_dt - vix * Ms, Dy = Dsum.y * inv_dt - viy * Ms;

    const float k = __ldg(&S->P.k), kn = __ldg(&S->P.k_near), ks = __ldg(&S->P.k_spring);
    const float ksum = k + kn + ks;
    const float ak = k / ksum, an = kn / ksum, as = ks / ksum;
    const float ds = vscale * 2.5f;
    float f[IN];
    f[0] = a * 0.25f;
    f[1] = b * 0.5f;
    f[2] = V1x * 0.25f;
    f[3] = V1y * 0.25f;
    f[4] = V2x * 0.5f;
    f[5] = V2y * 0.5f;
    f[6] = Ms * 0.125f;
    f[7] = (float)min(count, MAXNB) * (1.0f / MAXNB);
    f[8] = Dx * ds;
    f[9] = Dy * ds;
    f[10] = Txx * 0.25f;
    f[11] = Txy * 0.25f;
    f[12] = Tyy * 0.25f;
    f[13] = ak;
    f[14] = an;
    f[15] = as;
    f[16] = rest * 0.25f;
    f[17] = ak * (a - rest) * V1x * 0.25f;
    f[18] = ak * (a - rest) * V1y * 0.25f;
    f[19] = an * b * V2x * 0.5f;
    f[20] = an * b * V2y * 0.5f;
    f[21] = as * V1x * 0.5f;
    f[22] = as * V1y * 0.5f;
    f[23] = ak * R1.x * 0.25f;
    f[24] = ak * R1.y * 0.25f;
    f[25] = an * R2.x * 0.5f;
    f[26] = an * R2.y * 0.5f;
#pragma unroll
    for (int e = 27; e < IN - 1; ++e) f[e] = 0.0f;
    f[IN - 1] = 1.0f;  // constant input: the first layer's bias
    uint4 *row = reinterpret_cast<uint4 *>(feat + (size_t)i * IN);
#pragma unroll
    for (int q = 0; q < IN / 8; ++q) {
        uint4 v;
        v.x = tc::pack_bf16x2(f[8 * q + 0], f[8 * q + 1]);
        v.y = tc::pack_bf16x2(f[8 * q + 2], f[8 * q + 3]);
        v.z = tc::pack_bf16x2(f[8 * q + 4], f[8 * q + 5]);
        v.w = tc::pack_bf16x2(f[8 * q + 6], f[8 * q + 7]);
        row[q] = v;
    }
}

// ---------------------------------------------------------------------------
// fused MLP inference (tcgen05)
// ---------------------------------------------------------------------------

// Inference layout.  The first layer's bias is folded into the weight of
// the constant feature 31 (= 1); the second layer's bias enters as one more
// K = 16 MMA of a ones column against the bias column; the activation is
// 2 GELU (the factor 2 is absorbed by the weights that follow it, in
// training and inference alike).
struct alignas(128) MlpWeights {
    unsigned char w1[HID * IN * 2];    // W1, column 31 + b1
    unsigned char w2[HID * HID * 2];   // W2
    unsigned char w2b[HID * 16 * 2];   // column 0 = b2 (BF16), the rest 0
    unsigned char w3[OUT * HID * 2];   // W3
    unsigned char ones[128 * 16 * 2];  // column 0 = 1, the rest 0
    float b3[OUT];
    uint32_t taddr;
};

struct alignas(128) MlpPipe {
    unsigned char x[128 * IN * 2];
    unsigned char hbuf[128 * HID * 2];
    uint64_t mbar;
};

// One CTA per SM of four independent pipelines of 256 threads (8 warps);
// pipeline p owns TMEM columns [128 p, 128 p + 128) (all three layers of a
// tile accumulate there in turn), its own operand tiles, mbarrier and named
// barrier.  The pipelines share the weights; their tensor-core work and
// epilogues interleave.
constexpr int kPipes = 4;
constexpr int kPipeThreads = 256;
constexpr int kMlpThreads = kPipes * kPipeThreads;
constexpr uint32_t kTmemCols = 128 * kPipes;
constexpr int kTurnBar = 1 + kPipes;  // named barriers of the pipelines' turns at the epilogues

struct MlpSmem {
    MlpWeights w;
    MlpPipe pipe[kPipes];
};
// operand tiles start on 128-byte boundaries (descriptors and 16-byte stores)
static_assert(offsetof(MlpWeights, w2) % 128 == 0 && offsetof(MlpWeights, w2b) % 128 == 0 &&
                  offsetof(MlpWeights, w3) % 128 == 0 && offsetof(MlpWeights, ones) % 128 == 0,
              "weight tiles aligned");
static_assert(offsetof(MlpSmem, pipe) % 128 == 0 && sizeof(MlpPipe) % 128 == 0 &&
                  offsetof(MlpPipe, hbuf) % 128 == 0,
              "pipeline tiles aligned");
static_assert(sizeof(MlpSmem) + 1024 <= 227 * 1024, "fits the shared memory of one CTA");

// A row-major BF16 matrix of `cols` columns into a K-major tile, 16 bytes
// at a time.
__device__ __forceinline__ void stage_matrix(unsigned char *tile, const __nv_bfloat16 *__restrict__ w,
                                             int rows, int cols)
{
    const int chunks = cols >> 3;
    const uint4 *src = reinterpret_cast<const uint4 *>(w);
    for (int e = threadIdx.x; e < rows * chunks; e += blockDim.x) {
        const int r = e / chunks, k = e % chunks;
        *reinterpret_cast<uint4 *>(tile + tc::kmajor_offset(r, 8 * k, cols)) = __ldcg(src + e);
    }
}

// The inference weights, in 16-byte pieces (with 2-byte ones this prologue
// was 9 of the 13 us that a few rows took).
__device__ __forceinline__ void stage_weights(MlpWeights &s, const __nv_bfloat16 *__restrict__ w,
                                              const float *__restrict__ wf)
{
    const int t = threadIdx.x;
    stage_matrix(s.w2, w + OFF_W2, HID, HID);
    stage_matrix(s.w1, w + OFF_W1, HID, IN);
    stage_matrix(s.w3, w + OFF_W3, OUT, HID);
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (int e = t; e < HID * 2; e += blockDim.x) {
        const int r = e >> 1, k = 8 * (e & 1);
        uint4 b = zero, o = zero;
        if (k == 0) {
            b.x = (uint32_t)__bfloat16_as_ushort(__float2bfloat16(__ldcg(wf + OFF_B2 + r)));
            o.x = 0x3F80u;  // 1
        }
        *reinterpret_cast<uint4 *>(s.w2b + tc::kmajor_offset(r, k, 16)) = b;
        *reinterpret_cast<uint4 *>(s.ones + tc::kmajor_offset(r, k, 16)) = o;
    }
    for (int e = t; e < OUT; e += blockDim.x) s.b3[e] = __ldcg(wf + OFF_B3 + e);
    __syncthreads();  // column 31 of W1, staged above, takes the first bias
    for (int r = t; r < HID; r += blockDim.x)
        *reinterpret_cast<__nv_bfloat16 *>(s.w1 + tc::kmajor_offset(r, IN - 1, IN)) =
            __float2bfloat16(__ldcg(wf + OFF_W1 + r * IN + IN - 1) + __ldcg(wf + OFF_B1 + r));
}

// Epilogue of a hidden layer in a pipeline: warp w (0..7 within it) takes
// TMEM lanes 32 (w % 4) .. + 31 (one row per thread) and columns
// 64 (w / 4) .. + 63 of the pipeline's accumulator; activation in BF16 into
// the K-major activation tile (16-byte stores).
__device__ __forceinline__ void hidden_epilogue(unsigned char *hbuf, uint32_t tacc, int tp)
{
    const int w = tp >> 5;
    const int row = 32 * (w & 3) + (tp & 31);
    const int c0 = 64 * (w >> 2);
    const uint32_t lane = (uint32_t)(32 * (w & 3)) << 16;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int c = c0 + 32 * h;
        float v[32];
        tc::tmem_ld32(tacc + lane + (uint32_t)c, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint4 o;
            o.x = tc::act_bf16x2(v[8 * q + 0], v[8 * q + 1]);
            o.y = tc::act_bf16x2(v[8 * q + 2], v[8 * q + 3]);
            o.z = tc::act_bf16x2(v[8 * q + 4], v[8 * q + 5]);
            o.w = tc::act_bf16x2(v[8 * q + 6], v[8 * q + 7]);
            *reinterpret_cast<uint4 *>(hbuf + tc::kmajor_offset(row, c + 8 * q, HID)) = o;
        }
    }
}

// Half a feature row (16 values) of row tile*128 + (tp >> 1) as BF16: from
// the step's BF16 rows, or (HOST_ROWS) from a caller's float rows.
template <bool HOST_ROWS>
__device__ __forceinline__ void load_feat(const void *__restrict__ feat, int n, int tile, int tp,
                                          uint4 &a, uint4 &b)
{
    const int gi = tile * 128 + (tp >> 1);
    a = make_uint4(0, 0, 0, 0);
    b = a;
    if (gi >= n) return;
    if (!HOST_ROWS) {
        const uint4 *src = reinterpret_cast<const uint4 *>(
                               reinterpret_cast<const __nv_bfloat16 *>(feat) + (size_t)gi * IN) +
                           2 * (tp & 1);
        a = __ldcs(src);
        b = __ldcs(src + 1);
    } else {
        const float4 *src = reinterpret_cast<const float4 *>(
                                reinterpret_cast<const float *>(feat) + (size_t)gi * IN) +
                            4 * (tp & 1);
        const float4 f0 = __ldcs(src), f1 = __ldcs(src + 1), f2 = __ldcs(src + 2), f3 = __ldcs(src + 3);
        a = make_uint4(tc::pack_bf16x2(f0.x, f0.y), tc::pack_bf16x2(f0.z, f0.w),
                       tc::pack_bf16x2(f1.x, f1.y), tc::pack_bf16x2(f1.z, f1.w));
        b = make_uint4(tc::pack_bf16x2(f2.x, f2.y), tc::pack_bf16x2(f2.z, f2.w),
                       tc::pack_bf16x2(f3.x, f3.y), tc::pack_bf16x2(f3.z, f3.w));
    }
}

__device__ __forceinline__ void store_feat(unsigned char *x, int tp, const uint4 &a, const uint4 &b)
{
    const int r = tp >> 1, k = 16 * (tp & 1);
    *reinterpret_cast<uint4 *>(x + tc::kmajor_offset(r, k, IN)) = a;
    *reinterpret_cast<uint4 *>(x + tc::kmajor_offset(r, k + 8, IN)) = b;
}

// out[i] = (y0, y1, y2, 0) for n feature rows; tiles of 128 rows, pipeline
// p of CTA b takes tiles (p gridDim.x + b) + k gridDim.x kPipes: a few tiles
// spread over as many SMs before a second pipeline of any starts.  The next
// tile's features are fetched while the current one runs.  The weights are
// staged before the wait for the predecessor: no kernel of a step writes
// them.  HOST_ROWS: float rows in, rows of OUT floats (zeros after the
// third) out.
template <bool HOST_ROWS>
__global__ void __launch_bounds__(kMlpThreads, 1)
k_mlp(int n, const void *__restrict__ feat, const __nv_bfloat16 *__restrict__ wbf,
      const float *__restrict__ wf, float4 *__restrict__ out, unsigned *__restrict__ err)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    MlpSmem &S = *reinterpret_cast<MlpSmem *>(smem_raw);
    const int t = threadIdx.x;
    const int p = t / kPipeThreads, tp = t % kPipeThreads, w = tp >> 5;
    MlpPipe &P = S.pipe[p];
    const int bar = 1 + p;
    if (t < 32) {
        tc::tmem_alloc(&S.w.taddr, kTmemCols);
        tc::tmem_relinquish();
    }
    if (tp == 0) {
        tc::mbar_init(&P.mbar, 1);
        tc::mbar_fence_init();
    }
    stage_weights(S.w, wbf, wf);
    const int ntiles = (n + 127) / 128;
    const int stride = gridDim.x * kPipes;
    int tile = p * gridDim.x + blockIdx.x;
    pdl_enter();
    {
        uint4 a, b;
        load_feat<HOST_ROWS>(feat, n, tile, tp, a, b);
        store_feat(P.x, tp, a, b);
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tacc = S.w.taddr + (uint32_t)(128 * p);
    const uint32_t sx = tc::smem_u32(P.x), sh = tc::smem_u32(P.hbuf);
    uint32_t phase = 0;
    bool ok = true;
    // A wait that gives up clears `ok`, which stays uniform across the
    // pipeline (every barrier after a wait is a vote): the pipeline then issues
    // and waits for no more MMAs, but goes through its barriers to the end, so
    // that its partner's turns come.
    auto rounds_of = [&](int q) {
        const int first = q * (int)gridDim.x + (int)blockIdx.x;
        return first < ntiles ? (ntiles - 1 - first) / stride + 1 : 0;
    };
    // Turns at the epilogues: pipelines p and p + 2 have them alternately,
    // pipeline p's first (turn e is the e-th of either).  Left to themselves
    // the four pipelines fall into step -- they share the activation units
    // fairly, so they end their epilogues together and then wait for the
    // tensor core together (1,048,576 rows: 94 -> 84 us).
    const int partner = p ^ 2;
    const int partner_turns = 2 * rounds_of(partner);
    int turn = 0;
    auto epilogue = [&] {
        // pipeline p + 2 follows turn e of pipeline p, which follows turn e - 1
        const int before = p < partner ? turn - 1 : turn;
        if (before >= 0 && before < partner_turns) tc::named_sync(kTurnBar + p, 2 * kPipeThreads);
        hidden_epilogue(P.hbuf, tacc, tp);
        const int after = p < partner ? turn : turn + 1;
        if (after < partner_turns) tc::named_arrive(kTurnBar + partner, 2 * kPipeThreads);
        ++turn;
    };
    for (; tile < ntiles; tile += stride) {
        // layer 1: x (128 x 32) . W1'^T
        if (tp == 0 && ok) {
            tc::mma_tile(tacc, sx, tc::smem_u32(S.w.w1), HID, IN, false);
            tc::mma_commit(&P.mbar);
        }
        // the next tile's features, loaded now and stored at the end of this
        // tile: their DRAM latency hides behind the whole tile, not behind
        // layer 1 alone (6% off the kernel)
        uint4 na, nb;
        load_feat<HOST_ROWS>(feat, n, tile + stride, tp, na, nb);
        bool done = ok && tc::mbar_wait(&P.mbar, phase);
        phase ^= 1u;
        tc::fence_after_sync();
        epilogue();
        tc::fence_async_smem();
        tc::fence_before_sync();
        ok = tc::named_sync_and(bar, kPipeThreads, done);
        tc::fence_after_sync();
        // layer 2: h1 (128 x 128) . W2^T + 1 . b2^T
        if (tp == 0 && ok) {
            tc::mma_tile(tacc, sh, tc::smem_u32(S.w.w2), HID, HID, false);
            tc::mma_tile(tacc, tc::smem_u32(S.w.ones), tc::smem_u32(S.w.w2b), HID, 16, true);
            tc::mma_commit(&P.mbar);
        }
        done = ok && tc::mbar_wait(&P.mbar, phase);
        phase ^= 1u;
        tc::fence_after_sync();
        epilogue();
        tc::fence_async_smem();
        tc::fence_before_sync();
        ok = tc::named_sync_and(bar, kPipeThreads, done);
        tc::fence_after_sync();
        // layer 3: h2 (128 x 128) . W3^T -> columns [0, 16)
        if (tp == 0 && ok) {
            tc::mma_tile(tacc, sh, tc::smem_u32(S.w.w3), OUT, HID, false);
            tc::mma_commit(&P.mbar);
        }
        done = ok && tc::mbar_wait(&P.mbar, phase);
        phase ^= 1u;
        tc::fence_after_sync();
        if (w < 4) {
            float v[16];
            tc::tmem_ld16(tacc + ((uint32_t)(32 * w) << 16), v);
            const int gi = tile * 128 + 32 * w + (tp & 31);
            if (gi < n && done) {
                const float4 y = make_float4(v[0] + S.w.b3[0], v[1] + S.w.b3[1], v[2] + S.w.b3[2], 0.0f);
                if (!HOST_ROWS) {
                    __stcs(out + gi, y);
                } else {
                    float4 *o = out + (size_t)gi * (OUT / 4);
                    o[0] = y;
#pragma unroll
                    for (int q = 1; q < OUT / 4; ++q) o[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            }
        }
        store_feat(P.x, tp, na, nb);  // layer 1 consumed x long ago
        tc::fence_async_smem();
        tc::fence_before_sync();
        ok = tc::named_sync_and(bar, kPipeThreads, done);  // read before layer 1 reuses it
        tc::fence_after_sync();
    }
    if (!ok && tp == 0) {
        if (HOST_ROWS)
            *reinterpret_cast<volatile unsigned *>(err) = 1u;  // page-locked host memory
        else
            atomicAdd(err, 1u);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) tc::tmem_dealloc(S.w.taddr, kTmemCols);
}

// ---------------------------------------------------------------------------
// generic tcgen05 GEMM (sph_learned_gemm_check)
// ---------------------------------------------------------------------------

// C[m][n] (ldc) = sum_k A(m, k) B(n, k), A(m, k) = A[m * sam + k * sak],
// B(n, k) = B[n * sbn + k * sbk] (BF16), FP32 result; M, N, K any sizes
// (zero padded to the 128 x BN x 64 tiles).  One 128-thread CTA per tile.
constexpr int kGemmK = 64;

struct GemmSmem {
    unsigned char a[128 * kGemmK * 2];
    unsigned char b[128 * kGemmK * 2];
    uint64_t mbar;
    uint32_t taddr;
};

__global__ void __launch_bounds__(128, 1)
k_gemm(int M, int N, int K, const __nv_bfloat16 *__restrict__ A, long long sam, long long sak,
       const __nv_bfloat16 *__restrict__ B, long long sbn, long long sbk, float *__restrict__ C,
       long long ldc, int BN, unsigned *__restrict__ err)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    GemmSmem &s = *reinterpret_cast<GemmSmem *>(smem_raw);
    const int t = threadIdx.x, w = t >> 5;
    const int m0 = blockIdx.x * 128, n0 = blockIdx.y * BN;
    if (w == 0) {
        tc::tmem_alloc(&s.taddr, 128);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        tc::mbar_init(&s.mbar, 1);
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = s.taddr;
    uint32_t phase = 0;
    bool ok = true;
    const __nv_bfloat16 zero = __float2bfloat16(0.0f);
    for (int k0 = 0; k0 < K; k0 += kGemmK) {
        for (int e = t; e < 128 * kGemmK; e += 128) {
            const int r = e / kGemmK, k = e % kGemmK;
            const int gm = m0 + r, gk = k0 + k;
            *reinterpret_cast<__nv_bfloat16 *>(s.a + tc::kmajor_offset(r, k, kGemmK)) =
                (gm < M && gk < K) ? A[gm * sam + gk * sak] : zero;
            if (r < BN) {
                const int gn = n0 + r;
                *reinterpret_cast<__nv_bfloat16 *>(s.b + tc::kmajor_offset(r, k, kGemmK)) =
                    (gn < N && gk < K) ? B[gn * sbn + gk * sbk] : zero;
            }
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (t == 0) {
            tc::mma_tile(tm, tc::smem_u32(s.a), tc::smem_u32(s.b), BN, kGemmK, k0 > 0);
            tc::mma_commit(&s.mbar);
        }
        const bool done = tc::mbar_wait(&s.mbar, phase);
        phase ^= 1u;
        tc::fence_before_sync();
        ok = __syncthreads_and(done) != 0;  // uniform: the smem tiles are free again
        tc::fence_after_sync();
        if (!ok) break;
    }
    if (ok) {
        const int row = 32 * (w & 3) + (t & 31);
        const uint32_t lane = (uint32_t)(32 * (w & 3)) << 16;
        for (int c = 0; c < BN; c += 16) {
            float v[16];
            tc::tmem_ld16(tm + lane + (uint32_t)c, v);
            const int gm = m0 + row;
            if (gm < M)
                for (int e = 0; e < 16; ++e) {
                    const int gn = n0 + c + e;
                    if (gn < N) C[gm * ldc + gn] = v[e];
                }
        }
    } else if (t == 0) {
        atomicAdd(err, 1u);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (w == 0) tc::tmem_dealloc(tm, 128);
}

// ---------------------------------------------------------------------------
// training: one batch is three kernels
// ---------------------------------------------------------------------------

// Forward and backward pass of one batch, 128 samples at a time: a CTA
// gathers a tile of samples, runs the three layers, the loss gradient and
// the backward products with everything that passes between them in shared
// memory, tensor memory or registers, and leaves the tiles that the weight
// gradients are made of (k_grad).
//
// Why one kernel: a batch of 4,096 is 2.4e8 multiply-adds, about 1 us of one
// SM's tensor core per tile, but as separate products its operands make
// eight round trips through memory.  What bounds a tile here is the chain of
// its five dependent products and their epilogues.  A whole training step of
// 4,096 samples: 2.66 ms as separate GEMMs and elementwise kernels, 46 us here
// (GB300): 11 for this pass, 31 for k_grad, 4 for k_adam.
//
// The transposed operands of the backward products (W2, W3 by rows; the
// activations, gradients and features as M x K with K over the samples) are
// MN-major views of the very tiles the forward pass staged.  The products are
// those of the inference kernel in the same K order; the biases, which are
// weights of its products, are added in FP32 here, so an activation may differ
// from inference by a BF16 unit.
constexpr int kTrainThreads = 512;
constexpr uint32_t kTrainTmem = 128;
constexpr uint32_t kColAcc = 0;  // tensor memory: the running product
// What k_train leaves of a tile for k_grad: its operand tiles, as they lie in
// shared memory (byte offsets).
constexpr size_t kImgH1 = 0, kImgH2 = 128 * HID * 2, kImgZ1 = 2 * kImgH2, kImgZ2 = 3 * kImgH2,
                 kImgX = 4 * kImgH2, kImgDy = kImgX + 128 * IN * 2, kTileImage = kImgDy + 128 * OUT * 2;

struct alignas(128) TrainSmem {
    unsigned char w1[HID * IN * 2];
    unsigned char w2[HID * HID * 2];
    unsigned char w3[OUT * HID * 2];
    unsigned char x[128 * IN * 2];
    unsigned char h1[128 * HID * 2];   // activations, then dZ1
    unsigned char h2[128 * HID * 2];   // activations, then dZ2
    unsigned char dy[128 * OUT * 2];
    float b1[HID], b2[HID], b3[OUT];   // biases as the forward pass adds them
    double loss[4];
    uint64_t mbar;
    uint32_t taddr;
};

// Makes the CTA's shared-memory writes visible to the tensor core and joins
// the CTA; false once any thread's wait has given up.
__device__ __forceinline__ bool join_for_mma(bool ok)
{
    tc::fence_async_smem();
    tc::fence_before_sync();
    const bool all = __syncthreads_and(ok) != 0;
    tc::fence_after_sync();
    return all;
}

// cmask: outputs in the loss (bit 0, 1 displacement, bit 2 error); trunk =
// false: the output layer's gradients alone.  img: the tiles' images for
// k_grad, ploss: gridDim.x squared-error sums.
__global__ void __launch_bounds__(kTrainThreads, 1)
k_train(int tiles, const int *__restrict__ order, const __nv_bfloat16 *__restrict__ X,
        const float4 *__restrict__ T, const __nv_bfloat16 *__restrict__ wbf,
        const float *__restrict__ wf, int cmask, bool trunk, unsigned char *__restrict__ img,
        double *__restrict__ ploss, unsigned *__restrict__ err)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    TrainSmem &s = *reinterpret_cast<TrainSmem *>(smem_raw);
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    // a thread's share of an accumulator: one row, 32 columns
    const int row = 32 * (w & 3) + lane, c0 = 32 * (w >> 2);
    if (w == 0) {
        tc::tmem_alloc(&s.taddr, kTrainTmem);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        tc::mbar_init(&s.mbar, 1);
        tc::mbar_fence_init();
    }
    // samples do not depend on the previous step; the weights do
    const int first = blockIdx.x;
    const int xr = t >> 2, xk = t & 3;  // the thread's 16-byte piece of a feature row
    uint4 xv = make_uint4(0, 0, 0, 0);
    float4 tv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto load_tile = [&](int tile) {
        xv = __ldg(reinterpret_cast<const uint4 *>(X + (size_t)__ldg(order + tile * 128 + xr) * IN) + xk);
        if (w < 4) tv = __ldg(T + __ldg(order + tile * 128 + row));
    };
    load_tile(first);
    pdl_enter();
    stage_matrix(s.w1, wbf + OFF_W1, HID, IN);
    stage_matrix(s.w2, wbf + OFF_W2, HID, HID);
    stage_matrix(s.w3, wbf + OFF_W3, OUT, HID);
    if (t < HID) {
        s.b1[t] = __bfloat162float(__float2bfloat16(__ldcg(wf + OFF_B1 + t)));
        s.b2[t] = __bfloat162float(__float2bfloat16(__ldcg(wf + OFF_B2 + t)));
    }
    if (t < OUT) s.b3[t] = __ldcg(wf + OFF_B3 + t);

    const float rows_f = (float)(tiles * 128);
    const uint32_t lane_base = (uint32_t)(32 * (w & 3)) << 16;
    uint32_t tm = 0, phase = 0;
    bool ok = true;
    double loss = 0.0;
    auto wait = [&]() {
        const bool done = tc::mbar_wait(&s.mbar, phase);
        phase ^= 1u;
        tc::fence_after_sync();
        return done;
    };
    // z = product + bias; the activations go to tile h and its image, act'(z) to g
    float g1[32], g2[32];
    auto hidden = [&](unsigned char *h, unsigned char *image, const float *b, float (&g)[32]) {
        float v[32];
        tc::tmem_ld32(tm + kColAcc + lane_base + (uint32_t)c0, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c = 8 * q + 2 * e;
                const float z0 = v[c] + b[c0 + c], z1 = v[c + 1] + b[c0 + c + 1];
                o[e] = tc::act_bf16x2(z0, z1);
                g[c] = act_grad(z0);
                g[c + 1] = act_grad(z1);
            }
            const uint32_t at = tc::kmajor_offset(row, c0 + 8 * q, HID);
            const uint4 v4 = make_uint4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<uint4 *>(h + at) = v4;
            *reinterpret_cast<uint4 *>(image + at) = v4;
        }
    };
    // dZ = dH act'(z) into the image, and into tile h (if any)
    auto back = [&](unsigned char *h, unsigned char *image, const float (&g)[32]) {
        float v[32];
        tc::tmem_ld32(tm + kColAcc + lane_base + (uint32_t)c0, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c = 8 * q + 2 * e;
                o[e] = tc::pack_bf16x2(v[c] * g[c], v[c + 1] * g[c + 1]);
            }
            const uint32_t at = tc::kmajor_offset(row, c0 + 8 * q, HID);
            const uint4 v4 = make_uint4(o[0], o[1], o[2], o[3]);
            if (h) *reinterpret_cast<uint4 *>(h + at) = v4;
            *reinterpret_cast<uint4 *>(image + at) = v4;
        }
    };
    const uint32_t aw1 = tc::smem_u32(s.w1), aw2 = tc::smem_u32(s.w2), aw3 = tc::smem_u32(s.w3),
                   ax = tc::smem_u32(s.x), ah1 = tc::smem_u32(s.h1), ah2 = tc::smem_u32(s.h2),
                   ady = tc::smem_u32(s.dy);
    for (int tile = first; tile < tiles; tile += gridDim.x) {
        unsigned char *gi = img + (size_t)tile * kTileImage;
        *reinterpret_cast<uint4 *>(s.x + tc::kmajor_offset(xr, 8 * xk, IN)) = xv;
        *reinterpret_cast<uint4 *>(gi + kImgX + tc::kmajor_offset(xr, 8 * xk, IN)) = xv;
        const float4 target = tv;
        if (!join_for_mma(ok)) { ok = false; break; }
        tm = s.taddr;
        // layer 1
        if (t == 0) {
            tc::mma_operands(tm + kColAcc, tc::k_major(ax, IN), tc::k_major(aw1, IN), HID, IN, false);
            tc::mma_commit(&s.mbar);
        }
        if (tile + (int)gridDim.x < tiles) load_tile(tile + gridDim.x);
        ok = wait();
        hidden(s.h1, gi + kImgH1, s.b1, g1);
        if (!join_for_mma(ok)) { ok = false; break; }
        // layer 2
        if (t == 0) {
            tc::mma_operands(tm + kColAcc, tc::k_major(ah1, HID), tc::k_major(aw2, HID), HID, HID, false);
            tc::mma_commit(&s.mbar);
        }
        ok = wait();
        hidden(s.h2, gi + kImgH2, s.b2, g2);
        if (!join_for_mma(ok)) { ok = false; break; }
        // layer 3
        if (t == 0) {
            tc::mma_operands(tm + kColAcc, tc::k_major(ah2, HID), tc::k_major(aw3, HID), OUT, HID, false);
            tc::mma_commit(&s.mbar);
        }
        ok = wait();
        if (w < 4) {
            // dY = mask * 2 (Y - T) / rows
            float y[16];
            tc::tmem_ld16(tm + kColAcc + lane_base, y);
            const float tt[3] = {target.x, target.y, target.z};
            uint32_t d16[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float g = 0.0f;
                if ((cmask >> c) & 1) {
                    const float d = (y[c] + s.b3[c]) - tt[c];
                    loss += (double)d * d;
                    g = 2.0f * d / rows_f;
                }
                d16[c] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16(g));
            }
            const uint4 d0 = make_uint4(d16[0] | (d16[1] << 16), d16[2], 0u, 0u), d1 = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4 *>(s.dy + tc::kmajor_offset(row, 0, OUT)) = d0;
            *reinterpret_cast<uint4 *>(s.dy + tc::kmajor_offset(row, 8, OUT)) = d1;
            *reinterpret_cast<uint4 *>(gi + kImgDy + tc::kmajor_offset(row, 0, OUT)) = d0;
            *reinterpret_cast<uint4 *>(gi + kImgDy + tc::kmajor_offset(row, 8, OUT)) = d1;
        }
        if (!join_for_mma(ok)) { ok = false; break; }
        if (trunk) {
            // dH2 = dY W3
            if (t == 0) {
                tc::mma_operands(tm + kColAcc, tc::k_major(ady, OUT), tc::mn_major(aw3, HID), HID, OUT, false);
                tc::mma_commit(&s.mbar);
            }
            ok = wait();
            back(s.h2, gi + kImgZ2, g2);
            if (!join_for_mma(ok)) { ok = false; break; }
            // dH1 = dZ2 W2
            if (t == 0) {
                tc::mma_operands(tm + kColAcc, tc::k_major(ah2, HID), tc::mn_major(aw2, HID), HID, HID, false);
                tc::mma_commit(&s.mbar);
            }
            ok = wait();
            back(nullptr, gi + kImgZ1, g1);
        }
        // the tile's buffers are free again once every thread is past its
        // wait: the next tile's join follows its feature store, so the store
        // itself must wait here
        if (!join_for_mma(ok)) { ok = false; break; }
    }
    if (ok) {
        if (w < 4) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
            if (lane == 0) s.loss[w] = loss;
        }
    } else if (t == 0) {
        atomicAdd(err, 1u);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (ok && t == 0) ploss[blockIdx.x] = s.loss[0] + s.loss[1] + s.loss[2] + s.loss[3];
    if (w == 0) tc::tmem_dealloc(s.taddr, kTrainTmem);
}

// The weight gradients of a batch: sums over its samples, taken in the samples'
// order by one accumulator each (the tiles' products one after another in
// tensor memory, the biases' sums one row after another), so that they do not
// depend on how many CTAs ran the batch (added up from the CTAs' partial sums
// they were 1e-7 away, which BF16 copies of the weights and Adam made up to
// 2e-5 of an epoch's loss).  A CTA per 16 columns of a product -- dW2 = dZ2^T H1
// (0..7), dW1 = dZ1^T X (8, 9), dW3^T = H2^T dY (10) -- four for the second
// bias (11..14) and one for the third.  What bounds it is one SM reading a whole operand, 1 MB at
// a batch of 4,096, four tiles in flight, and the biases' chains of additions: 31
// us (one CTA for all of b2: 50).
constexpr int kGradThreads = 256, kGradStages = 4, kGradRoles = 16, kGradSlice = 16;

struct alignas(128) GradSmem {
    unsigned char a[kGradStages][128 * HID * 2];
    unsigned char b[kGradStages][128 * kGradSlice * 2];
    uint64_t mbar[2];
    uint32_t taddr;
};

__device__ __forceinline__ void copy16_async(unsigned char *smem, const unsigned char *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(smem)), "l"(src) : "memory");
}

__global__ void __launch_bounds__(kGradThreads, 1)
k_grad(int tiles, const unsigned char *__restrict__ img, bool trunk, float *__restrict__ grad,
       unsigned *__restrict__ err)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    GradSmem &s = *reinterpret_cast<GradSmem *>(smem_raw);
    const int t = threadIdx.x, w = t >> 5;
    const int role = trunk ? (int)blockIdx.x : 10 + 5 * (int)blockIdx.x;
    const bool product = role <= 10, rows_b2 = role > 10 && role < 15, has_b = !rows_b2;
    const size_t a_at = role == 10 ? kImgH2 : role == 8 || role == 9 ? kImgZ1 : kImgZ2;
    const size_t b_at = role < 8 ? kImgH1 : role < 10 ? kImgX : kImgDy;
    const int b_cols = role < 8 ? HID : role < 10 ? IN : OUT;
    const int c0 = role < 8 ? kGradSlice * role : role < 10 ? kGradSlice * (role - 8) : 0;
    if (w == 0) {
        tc::tmem_alloc(&s.taddr, 32);
        tc::tmem_relinquish();
    }
    if (t == 0) {
        tc::mbar_init(&s.mbar[0], 1);
        tc::mbar_init(&s.mbar[1], 1);
        tc::mbar_fence_init();
    }
    pdl_enter();
    auto load = [&](int k) {
        if (k < tiles) {
            const unsigned char *gi = img + (size_t)k * kTileImage;
            const int st = k % kGradStages;
            if (product)
                for (int e = t; e < 128 * HID * 2 / 16; e += kGradThreads)
                    copy16_async(s.a[st] + 16 * e, gi + a_at + 16 * e);
            if (rows_b2)  // 32 columns, row by row
                for (int e = t; e < 128 * 4; e += kGradThreads)
                    copy16_async(s.a[st] + 16 * e,
                                 gi + a_at + tc::kmajor_offset(e >> 2, 32 * (role - 11) + 8 * (e & 3), HID));
            if (has_b)
                copy16_async(s.b[st] + tc::kmajor_offset(t >> 1, 8 * (t & 1), kGradSlice),
                             gi + b_at + tc::kmajor_offset(t >> 1, c0 + 8 * (t & 1), b_cols));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int k = 0; k < kGradStages - 1; ++k) load(k);
    bool ok = true;
    float sum = 0.0f;
    uint32_t tm = 0;
    for (int k = 0; k < tiles; ++k) {
        const int st = k % kGradStages;
        asm volatile("cp.async.wait_group %0;" ::"n"(kGradStages - 2) : "memory");
        ok = join_for_mma(ok);  // the tile is there for every thread (and for the tensor core)
        tm = s.taddr;
        if (product) {
            if (t == 0 && ok) {
                tc::mma_operands(tm, tc::mn_major(tc::smem_u32(s.a[st]), HID),
                                 tc::mn_major(tc::smem_u32(s.b[st]), kGradSlice), kGradSlice, 128, k > 0);
                tc::mma_commit(&s.mbar[k & 1]);
            }
            // the stage loaded next was the last tile's
            if (ok && k > 0) ok = tc::mbar_wait(&s.mbar[(k - 1) & 1], (uint32_t)((k - 1) >> 1) & 1u);
        } else if (t < (rows_b2 ? 32 : OUT)) {
            const unsigned char *tile = rows_b2 ? s.a[st] : s.b[st];
            // the rows' values requested together, then added one after another
#pragma unroll 1
            for (int r0 = 0; r0 < 128; r0 += 32) {
                float v[32];
#pragma unroll
                for (int r = 0; r < 32; ++r)
                    v[r] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16 *>(
                        tile + (rows_b2 ? (uint32_t)((r0 + r) * 64 + 2 * t) : tc::kmajor_offset(r0 + r, t, OUT))));
#pragma unroll
                for (int r = 0; r < 32; ++r) sum = __fadd_rn(sum, v[r]);
            }
        }
        load(k + kGradStages - 1);
    }
    if (product && ok) ok = tc::mbar_wait(&s.mbar[(tiles - 1) & 1], (uint32_t)((tiles - 1) >> 1) & 1u);
    asm volatile("cp.async.wait_all;" ::: "memory");
    ok = join_for_mma(ok);
    if (!ok) {
        if (t == 0) atomicAdd(err, 1u);
    } else if (!product) {
        if (t < (rows_b2 ? 32 : OUT)) grad[(rows_b2 ? OFF_B2 + 32 * (role - 11) : OFF_B3) + t] = sum;
    } else if (w < 4) {
        float u[16];
        tc::tmem_ld16(tm + ((uint32_t)(32 * w) << 16), u);
        const int row = t;
#pragma unroll
        for (int e = 0; e < 16; ++e)
            grad[role < 8    ? OFF_W2 + row * HID + c0 + e
                 : role < 10 ? OFF_W1 + row * IN + c0 + e
                             : OFF_W3 + e * HID + row] = u[e];
    }
    tc::fence_before_sync();
    __syncthreads();
    if (w == 0) tc::tmem_dealloc(s.taddr, 32);
}

// Adam on the FP32 master weights and their BF16 copies; the batch's squared
// error (of `parts` CTAs) is added
// to *loss.  trunk = false: the output layer's rows of cmask alone.  The
// first layer's bias has no gradient: it acts through the weight of the
// constant feature 31.
__global__ void __launch_bounds__(128)
k_adam(int parts, const float *__restrict__ grad, const double *__restrict__ ploss,
       float *__restrict__ w, float *__restrict__ m, float *__restrict__ v, int cmask, bool trunk,
       float lr, float b1t, float b2t, __nv_bfloat16 *__restrict__ wbf, double *__restrict__ loss)
{
    pdl_enter();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e == 0) {
        double a = 0.0;
        for (int c = 0; c < parts; ++c) a += __ldcg(ploss + c);
        *loss += a;
    }
    if (e >= NPARAM) return;
    bool train = trunk;
    if (!trunk && e >= OFF_W3)
        train = (cmask >> (e >= OFF_B3 ? e - OFF_B3 : (e - OFF_W3) / HID)) & 1;
    if (train) {
        float g = 0.0f;
        if (e < OFF_B1 || e >= OFF_W2) g = __ldcg(grad + e);
        const float mm = 0.9f * m[e] + 0.1f * g;
        const float vv = 0.999f * v[e] + 0.001f * g * g;
        m[e] = mm;
        v[e] = vv;
        w[e] -= lr * (mm / (1.0f - b1t)) / (sqrtf(vv / (1.0f - b2t)) + 1e-8f);
    }
    wbf[e] = __float2bfloat16(w[e]);
}

__global__ void k_f32_to_bf16(int n, const float *__restrict__ in, __nv_bfloat16 *__restrict__ out)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) out[e] = __float2bfloat16(in[e]);
}

// ---------------------------------------------------------------------------
// sample collection and calibration
// ---------------------------------------------------------------------------

// splitmix64 finaliser: the sample selection hash.
__host__ __device__ __forceinline__ unsigned long long mix64(unsigned long long z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// 1 for each slot that is a sample: few enough neighbours and, for frac < 1,
// the particle's hash below frac.
__global__ void __launch_bounds__(kBlock)
k_select(int n, const unsigned short *__restrict__ nbc, const int *__restrict__ ids,
         unsigned long long salt, double frac, unsigned *__restrict__ flag)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bool take = (int)nbc[i] <= MAXNB;
    if (take && frac < 1.0)
        take = (double)(mix64(salt ^ (unsigned long long)ids[i]) >> 11) * (1.0 / 9007199254740992.0) < frac;
    flag[i] = take ? 1u : 0u;
}

// Appends the selected slots in slot order, `room` rows at most: row off[i]
// takes slot i's features and targets (plain displacement / s, error 0).
__global__ void __launch_bounds__(kBlock)
k_append(Ctx c, int room, const unsigned *__restrict__ flag, const int *__restrict__ off,
         const __nv_bfloat16 *__restrict__ feat, const float2 *__restrict__ disp,
         __nv_bfloat16 *__restrict__ X, float4 *__restrict__ T, int *__restrict__ slot)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n || !flag[i]) return;
    const int r = off[i];
    if (r >= room) return;
    const float s = out_scale(c.scenes + scene_of(c, i));
    const uint4 *src = reinterpret_cast<const uint4 *>(feat + (size_t)i * IN);
    uint4 *dst = reinterpret_cast<uint4 *>(X + (size_t)r * IN);
#pragma unroll
    for (int q = 0; q < IN / 8; ++q) dst[q] = src[q];
    const float2 d = disp[i];
    T[r] = make_float4(d.x / s, d.y / s, 0.0f, 1.0f);
    slot[r] = i;
}

// Feature rows (as floats) and neighbour counts (-1: always the plain
// relaxation) of the particles with ids [lo, lo + m), by id: a thread per 8
// features, so that a row's 64 bytes are read and its 128 written in full
// sectors.  (On the host this conversion and scatter took 17 ns a particle;
// 131,071 particles 2.4 -> 0.52 ms with the copies.)
__global__ void __launch_bounds__(kBlock)
k_rows_by_id(int n, int lo, int m, const int *__restrict__ ids,
             const __nv_bfloat16 *__restrict__ feat, const unsigned short *__restrict__ nbc,
             float *__restrict__ rows, int *__restrict__ counts)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = e >> 2;
    const int q = (int)(e & 3);
    if (i >= n) return;
    const int r = ids[i] - lo;
    if (r < 0 || r >= m) return;
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(feat + (size_t)i * IN) + q);
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
    float f[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        f[2 * k] = __uint_as_float(u[k] << 16);
        f[2 * k + 1] = __uint_as_float(u[k] & 0xFFFF0000u);
    }
    float4 *dst = reinterpret_cast<float4 *>(rows + (size_t)r * IN) + 2 * q;
    dst[0] = make_float4(f[0], f[1], f[2], f[3]);
    dst[1] = make_float4(f[4], f[5], f[6], f[7]);
    if (q == 0) counts[r] = nbc[i] == 65535 ? -1 : (int)nbc[i];
}

// Density at displaced positions pos + disp (sorted order) over the stencil
// of the particle's undisplaced cell: the density each particle ends the
// relaxation with under a displacement field.
__global__ void k_density_displaced(Ctx c, const float2 *__restrict__ pos,
                                    const float2 *__restrict__ disp, const int *__restrict__ start,
                                    const unsigned *__restrict__ occ_in, float *__restrict__ rho)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const Scene *S = c.scenes + scene_of(c, i);
    const SG g = load_grid(S);
    const float hh = __ldg(&S->P.smoothing_radius), h2 = hh * hh, h_recip = 1.0f / hh;
    const bool capped = *occ_in > (unsigned)c.max_bucket;
    const float2 p0 = pos[i], dp = disp[i];
    const float px = p0.x + dp.x, py = p0.y + dp.y;
    const unsigned key = cell_key(p0.x, p0.y, g);
    float a = 0.0f;
    if (searchable(key, i, start, g, capped, c.max_bucket)) {
        for_each_candidate(key, start, g, capped, c.max_bucket, c.n, [&](int j) {
            if (j == i) return;
            const float2 q = pos[j], dq = disp[j];
            const float r2 = dist2(px - (q.x + dq.x), py - (q.y + dq.y));
            if (r2 > h2) return;
            const float ratio = (r2 > 0.0f ? r2 * rsqrtf(r2) : 0.0f) * h_recip;
            if (ratio < 1.0f) a += (1.0f - ratio) * (1.0f - ratio);
        });
    }
    rho[i] = a;
}

// Network displacement (sorted order) from its outputs.
__global__ void k_net_disp(Ctx c, const float4 *__restrict__ y, float2 *__restrict__ disp)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const float s = out_scale(c.scenes + scene_of(c, i));
    const float4 v = y[i];
    disp[i] = make_float2(v.x * s, v.y * s);
}

// Error targets of rows [0, rows): |rho_net - rho_plain| in percent of the
// rest density, clipped at 10.
__global__ void k_err_targets(Ctx c, const float *__restrict__ rho_net,
                              const float *__restrict__ rho_plain, const int *__restrict__ slot,
                              int rows, float4 *__restrict__ T)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const int i = slot[r];
    const float rest = __ldg(&c.scenes[scene_of(c, i)].P.rest_density);
    const float e = fabsf(rho_net[i] - rho_plain[i]) / rest * 100.0f;
    float4 t = T[r];
    t.z = fminf(e, 10.0f);
    T[r] = t;
}

// Self-test of the bounded tensor-core wait: waits on an mbarrier that no
// operation arrives at; the wait gives up after its poll limit and the
// kernel records that (*gave_up = 1) instead of hanging.
__global__ void k_wait_selftest(unsigned *__restrict__ gave_up)
{
    __shared__ uint64_t mbar;
    if (threadIdx.x == 0) {
        tc::mbar_init(&mbar, 1);
        tc::mbar_fence_init();
    }
    __syncthreads();
    const bool done = tc::mbar_wait(&mbar, 0);
    if (threadIdx.x == 0) *gave_up = done ? 0u : 1u;
}

}  // namespace ml

// The learned-relaxation model.
struct LearnedModel {
    float *w = nullptr;         // FP32 master weights (device)
    float *m = nullptr, *v = nullptr;
    __nv_bfloat16 *wbf = nullptr;
    int adam_t = 0;
    // samples
    __nv_bfloat16 *X = nullptr;
    float4 *T = nullptr;
    int *slot = nullptr;  // sorted slot of each sample of the last collection (calibration)
    int nsamples = 0, cap = 0;
    unsigned calls = 0;
    unsigned *d_err = nullptr;
    // training workspace, kept between calls: partial gradients and squared
    // errors of a step's CTAs, the epoch's running sum (the last of `loss`),
    // the epoch's sample order
    float *grad = nullptr;
    unsigned char *img = nullptr;
    double *loss = nullptr;
    int *order = nullptr;
    int parts_cap = 0, order_cap = 0, img_cap = 0;
    // sph_learned_forward's workspace, kept between calls: two buffers of
    // at most kForwardRows float rows and their outputs, the second stream,
    // and a page-locked word that a wait that gave up sets
    float *fwd_in[2] = {nullptr, nullptr};
    float4 *fwd_out[2] = {nullptr, nullptr};
    int fwd_cap[2] = {0, 0};
    cudaStream_t stream2 = nullptr;
    unsigned *h_err = nullptr;
    cudaStream_t stream = nullptr;
    unsigned long long seed = 0;
    // Host threads may share a model.  busy: held by a call while it has work
    // on the model's streams (a call of sph_learned_forward, an epoch), so
    // that the forward workspace is one call's at a time and a call's pieces
    // all see the same weights; train_busy: held by a whole training call,
    // whose workspace outlives its epochs.  train_busy is taken first.
    std::mutex busy, train_busy;
};

}  // namespace sph

struct sph_learned : sph::LearnedModel {};

namespace sph {
namespace {

#define LTRY(expr)                          \
    do {                                    \
        const int _rc = (expr);             \
        if (_rc != SPH_OK) return _rc;      \
    } while (0)
#define LCUDA(call) LTRY(cuda_fail((call), #call))

inline int nblk(long long n, int bs = 256) { return (int)((n + bs - 1) / bs); }

size_t mlp_smem() { return sizeof(ml::MlpSmem) + 1024; }
size_t train_smem() { return sizeof(ml::TrainSmem) + 1024; }
size_t grad_smem() { return sizeof(ml::GradSmem) + 1024; }
// At least 60 KB, so that at most three GEMM CTAs (3 x 128 TMEM columns)
// share an SM.
size_t gemm_smem() { return std::max(sizeof(ml::GemmSmem) + 1024, (size_t)60 * 1024); }

int configure_kernels()
{
    static bool done = false;
    if (done) return SPH_OK;
    LCUDA(cudaFuncSetAttribute(ml::k_mlp<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_smem()));
    LCUDA(cudaFuncSetAttribute(ml::k_mlp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_smem()));
    LCUDA(cudaFuncSetAttribute(ml::k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem()));
    LCUDA(cudaFuncSetAttribute(ml::k_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grad_smem()));
    LCUDA(cudaFuncSetAttribute(ml::k_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem()));
    done = true;
    return SPH_OK;
}

// Generic GEMM launch: C = A . B^T with strided operands.
int gemm(cudaStream_t st, int M, int N, int K, const __nv_bfloat16 *A, long long sam, long long sak,
         const __nv_bfloat16 *B, long long sbn, long long sbk, float *C, long long ldc, unsigned *err)
{
    const int BN = N >= 128 ? 128 : (N <= 16 ? 16 : (N <= 32 ? 32 : (N <= 64 ? 64 : 128)));
    dim3 grid((M + 127) / 128, (N + BN - 1) / BN);
    ml::k_gemm<<<grid, 128, gemm_smem(), st>>>(M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, BN, err);
    return cuda_fail(cudaGetLastError(), "gemm launch");
}

int check_err(LearnedModel *l)
{
    unsigned e = 0;
    LCUDA(cudaMemcpyAsync(&e, l->d_err, sizeof(e), cudaMemcpyDeviceToHost, l->stream));
    LCUDA(cudaStreamSynchronize(l->stream));
    if (e) {
        set_error("tensor-core wait gave up %u times (mbarrier not completed)", e);
        return SPH_ERR_CUDA;
    }
    return SPH_OK;
}

int num_sms()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// Particles of one piece of sph_learned_features.
constexpr int kFeaturePiece = 262144;

// Rows of one piece of sph_learned_forward.
constexpr int kForwardRows = 131072;

// Buffer b of the forward workspace for `rows` rows.
int ensure_forward(LearnedModel *l, int b, int rows)
{
    if (!l->h_err) {
        LCUDA(cudaHostAlloc((void **)&l->h_err, sizeof(unsigned), cudaHostAllocMapped));
        *l->h_err = 0u;
    }
    if (b == 1 && !l->stream2)
        LCUDA(cudaStreamCreateWithFlags(&l->stream2, cudaStreamNonBlocking));
    if (rows <= l->fwd_cap[b]) return SPH_OK;
    cudaFree(l->fwd_in[b]);
    cudaFree(l->fwd_out[b]);
    l->fwd_in[b] = nullptr;
    l->fwd_out[b] = nullptr;
    l->fwd_cap[b] = 0;
    LCUDA(cudaMalloc(&l->fwd_in[b], (size_t)rows * ml::IN * sizeof(float)));
    LCUDA(cudaMalloc(&l->fwd_out[b], (size_t)rows * ml::OUT * sizeof(float)));
    l->fwd_cap[b] = rows;
    return SPH_OK;
}

// Tile images that a model keeps between training calls: 64 MB, a batch of
// 59,904.
constexpr int kKeptTiles = 468;

// The training workspace for steps of `parts` CTAs and `rows` samples an epoch.
int ensure_training(LearnedModel *l, int parts, int tiles, int rows)
{
    if (!l->grad) LCUDA(cudaMalloc(&l->grad, ml::NPARAM * sizeof(float)));
    if (tiles > l->img_cap) {
        cudaFree(l->img);
        l->img = nullptr;
        l->img_cap = 0;
        LCUDA(cudaMalloc(&l->img, (size_t)tiles * ml::kTileImage));
        l->img_cap = tiles;
    }
    if (parts > l->parts_cap) {
        cudaFree(l->loss);
        l->loss = nullptr;
        l->parts_cap = 0;
        LCUDA(cudaMalloc(&l->loss, ((size_t)parts + 1) * sizeof(double)));
        l->parts_cap = parts;
    }
    if (rows > l->order_cap) {
        cudaFree(l->order);
        l->order = nullptr;
        l->order_cap = 0;
        LCUDA(cudaMalloc(&l->order, (size_t)rows * sizeof(int)));
        l->order_cap = rows;
    }
    return SPH_OK;
}

// One forward + backward + Adam step on the samples order[0..batch) (batch a
// multiple of 128).  cmask: outputs in the loss; trunk = false trains the
// output layer only.
int train_batch(LearnedModel *l, const int *order, int batch, int parts, int cmask, bool trunk,
                float lr)
{
    using namespace ml;
    launch_step(k_train, parts, kTrainThreads, train_smem(), l->stream, batch / 128, order,
               (const __nv_bfloat16 *)l->X, (const float4 *)l->T, (const __nv_bfloat16 *)l->wbf,
               (const float *)l->w, cmask, trunk, l->img, l->loss, l->d_err);
    launch_step(k_grad, trunk ? kGradRoles : 2, kGradThreads, grad_smem(), l->stream, batch / 128,
               (const unsigned char *)l->img, trunk, l->grad, l->d_err);
    ++l->adam_t;
    const float b1t = powf(0.9f, (float)l->adam_t), b2t = powf(0.999f, (float)l->adam_t);
    launch_step(k_adam, nblk(NPARAM, 128), 128, 0, l->stream, parts, (const float *)l->grad,
               (const double *)l->loss, l->w, l->m, l->v, cmask, trunk, lr, b1t, b2t, l->wbf,
               l->loss + l->parts_cap);
    return cuda_fail(cudaGetLastError(), "training step");
}

// Trains on samples [first, first + nsamples) for `epochs` shuffled passes.
int train_loop(LearnedModel *l, int first, int nsamples, int epochs, int batch, float lr,
               int cmask, bool trunk, float *loss)
{
    using namespace ml;
    if (nsamples < 128) {
        set_error("%d training samples: at least 128 are needed", nsamples);
        return SPH_ERR_STATE;
    }
    LTRY(configure_kernels());
    std::lock_guard<std::mutex> one_training(l->train_busy);
    batch = std::max(128, std::min(batch, nsamples) / 128 * 128);
    const int per_epoch = nsamples / batch;
    // a CTA per tile of 128 samples, at most one per SM
    const int parts = std::min(batch / 128, num_sms());
    // tile images of large batches (143 KB for every 128 samples) are given
    // back when the call ends, on every way out
    struct Trim {
        LearnedModel *l;
        ~Trim()
        {
            if (l->img_cap <= kKeptTiles) return;
            cudaFree(l->img);
            l->img = nullptr;
            l->img_cap = 0;
        }
    } trim{l};
    LTRY(ensure_training(l, parts, batch / 128, per_epoch * batch));
    double *d_loss = l->loss + l->parts_cap;
    std::vector<int> order(nsamples);
    for (int i = 0; i < nsamples; ++i) order[i] = first + i;
    unsigned long long rng = l->seed * 0x9E3779B97F4A7C15ull + 17ull + (unsigned long long)l->adam_t;
    auto next = [&]() {
        rng += 0x9E3779B97F4A7C15ull;
        unsigned long long z = rng;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    double last = 0.0;
    for (int ep = 0; ep < epochs; ++ep) {
        for (int i = nsamples - 1; i > 0; --i) std::swap(order[i], order[(int)(next() % (i + 1))]);
        std::lock_guard<std::mutex> one_epoch(l->busy);
        LCUDA(cudaMemcpyAsync(l->order, order.data(), (size_t)per_epoch * batch * sizeof(int),
                              cudaMemcpyHostToDevice, l->stream));
        LCUDA(cudaMemsetAsync(d_loss, 0, sizeof(double), l->stream));
        for (int it = 0; it < per_epoch; ++it)
            LTRY(train_batch(l, l->order + (size_t)it * batch, batch, parts, cmask, trunk, lr));
        double acc = 0.0;
        LCUDA(cudaMemcpyAsync(&acc, d_loss, sizeof(double), cudaMemcpyDeviceToHost, l->stream));
        LCUDA(cudaStreamSynchronize(l->stream));
        last = acc / ((double)per_epoch * batch);
    }
    LTRY(check_err(l));
    if (loss) *loss = (float)last;
    return SPH_OK;
}

// Message pass on the handle's C order into (feat, nbc), from the density
// records and hit masks the density pass has just left in the handle's
// C-order arrays; no row of features for a particle of more than max_nb
// neighbours.
int launch_messages(sph_cuda *h, __nv_bfloat16 *feat, unsigned short *nbc, int max_nb)
{
    if (h->n == 0) return SPH_OK;
    launch_step(h->long_masks ? ml::k_messages<true> : ml::k_messages<false>, nblk(h->n), kBlock, 0,
               h->stream, make_ctx(h), (const float4 *)h->xr_c, (const ulonglong2 *)h->mask01_c,
               (const unsigned long long *)h->mask2_c, (const int4 *)h->rows_c,
               (const float2 *)h->prev_c, (const int *)h->start_c,
               (const unsigned *)&h->d_state->build_max_occ[SLOT_PREDICTED], feat, nbc,
               &h->d_state->fb_count, max_nb);
    return cuda_fail(cudaGetLastError(), "messages");
}

int run_mlp(cudaStream_t st, LearnedModel *l, int n, const __nv_bfloat16 *feat, float4 *out,
            int sms)
{
    if (n == 0) return SPH_OK;
    LTRY(configure_kernels());
    const int grid = std::min((n + 127) / 128, sms > 0 ? sms : num_sms());
    launch_step(ml::k_mlp<false>, grid, ml::kMlpThreads, mlp_smem(), st, n, (const void *)feat,
               (const __nv_bfloat16 *)l->wbf, (const float *)l->w, out, l->d_err);
    return cuda_fail(cudaGetLastError(), "mlp launch");
}

// The per-particle buffers of a learned step (allocated once per handle).
int ensure_learned_buffers(sph_cuda *h)
{
    if (h->feat_c) return SPH_OK;
    const size_t N = (size_t)h->capacity + 1;
    LCUDA(cudaMalloc(&h->feat_c, N * ml::IN * sizeof(__nv_bfloat16)));
    LCUDA(cudaMalloc(&h->nbc_c, N * sizeof(unsigned short)));
    LCUDA(cudaMalloc(&h->net_c, N * sizeof(float4)));
    LCUDA(cudaMalloc(&h->fb_list, N * sizeof(int)));
    return SPH_OK;
}

// The predicted state of h's next step with its features and, with `l`,
// the network's outputs in h->net_c.  Leaves the A state as it is.
int predicted_features(sph_cuda *h, LearnedModel *l)
{
    LTRY(ensure_learned_buffers(h));
    LTRY(enqueue_predicted_state(h));  // ends with the density pass
    LTRY(launch_messages(h, (__nv_bfloat16 *)h->feat_c, h->nbc_c, INT_MAX));
    if (l) {
        LCUDA(cudaStreamSynchronize(l->stream));  // weights written on the model's stream
        LTRY(run_mlp(h->stream, l, h->n, (const __nv_bfloat16 *)h->feat_c, h->net_c, h->num_sms));
    }
    return SPH_OK;
}

}  // namespace

// Learned passes of a step (called by enqueue_step when a model is
// attached): the features (the plain density pass, then the message pass)
// on the C order, then the network.  With `events`, events[0] is recorded
// after the features and events[1] after the network.
int launch_learned_passes(sph_cuda *h, cudaEvent_t *events)
{
    LearnedModel *l = h->learned;
    LTRY(launch_density_pass(h));
    LTRY(launch_messages(h, (__nv_bfloat16 *)h->feat_c, h->nbc_c, ml::MAXNB));
    if (events) cudaEventRecord(events[0], h->stream);
    LTRY(run_mlp(h->stream, l, h->n, (const __nv_bfloat16 *)h->feat_c, h->net_c, h->num_sms));
    if (events) cudaEventRecord(events[1], h->stream);
    return SPH_OK;
}

unsigned bounds_flags_learned() { return read_bounds_flag(); }

void free_learned_buffers(sph_cuda *h)
{
    if (h->feat_c) cudaFree(h->feat_c);
    if (h->nbc_c) cudaFree(h->nbc_c);
    if (h->net_c) cudaFree(h->net_c);
    if (h->fb_list) cudaFree(h->fb_list);
    h->fb_list = nullptr;
    h->feat_c = nullptr;
    h->nbc_c = nullptr;
    h->net_c = nullptr;
    h->learned = nullptr;
}

}  // namespace sph

using namespace sph;

extern "C" {

int sph_learned_num_params(void) { return ml::NPARAM; }

int sph_learned_wait_selftest(int *gave_up)
{
    if (!gave_up) {
        set_error("null argument");
        return SPH_ERR_INVALID;
    }
    unsigned *d = nullptr;
    LCUDA(cudaMalloc(&d, sizeof(unsigned)));
    int rc = cuda_fail(cudaMemset(d, 0xFF, sizeof(unsigned)), "memset");
    if (!rc) {
        ml::k_wait_selftest<<<1, 32>>>(d);
        rc = cuda_fail(cudaGetLastError(), "selftest launch");
    }
    unsigned h = 0xFFFFFFFFu;
    if (!rc) rc = cuda_fail(cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost), "selftest");
    cudaFree(d);
    if (!rc) *gave_up = (int)h;
    return rc;
}

int sph_learned_create(sph_learned_t **out, int max_samples, unsigned long long seed)
{
    if (!out || max_samples < 0) {
        set_error("sph_learned_create: bad arguments");
        return SPH_ERR_INVALID;
    }
    *out = nullptr;
    sph_learned *l = new (std::nothrow) sph_learned();
    if (!l) return SPH_ERR_ALLOC;
    l->seed = seed;
    l->cap = max_samples;
    auto fail = [&](int rc) {
        sph_learned_destroy(l);
        return rc;
    };
    int rc = configure_kernels();
    if (rc) return fail(rc);
    if ((rc = cuda_fail(cudaStreamCreateWithFlags(&l->stream, cudaStreamNonBlocking), "stream")) ||
        (rc = cuda_fail(cudaMalloc(&l->w, ml::NPARAM * sizeof(float)), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&l->m, ml::NPARAM * sizeof(float)), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&l->v, ml::NPARAM * sizeof(float)), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&l->wbf, ml::NPARAM * sizeof(__nv_bfloat16)), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&l->d_err, sizeof(unsigned)), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&l->X, ((size_t)max_samples + 1) * ml::IN * sizeof(__nv_bfloat16)),
                        "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&l->T, ((size_t)max_samples + 1) * sizeof(float4)), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&l->slot, ((size_t)max_samples + 1) * sizeof(int)), "cudaMalloc")))
        return fail(rc);
    // Glorot-uniform weights from a seeded splitmix64 stream, zero biases
    std::vector<float> w(ml::NPARAM, 0.0f);
    unsigned long long z0 = seed;
    auto uni = [&]() {
        z0 += 0x9E3779B97F4A7C15ull;
        unsigned long long z = z0;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int rows, int cols) {
        const double lim = std::sqrt(6.0 / (rows + cols));
        for (int e = 0; e < rows * cols; ++e) w[off + e] = (float)((uni() * 2.0 - 1.0) * lim);
    };
    fill(ml::OFF_W1, ml::HID, ml::IN);
    fill(ml::OFF_W2, ml::HID, ml::HID);
    fill(ml::OFF_W3, ml::OUT, ml::HID);
    rc = sph_learned_set_params(l, w.data());
    if (rc) return fail(rc);
    *out = l;
    return SPH_OK;
}

int sph_learned_destroy(sph_learned_t *l)
{
    if (!l) return SPH_OK;
    if (l->stream) cudaStreamSynchronize(l->stream);
    if (l->stream2) cudaStreamSynchronize(l->stream2);
    void *ptrs[] = {l->w, l->m, l->v, l->wbf, l->d_err, l->X, l->T, l->slot, l->grad, l->img,
                    l->loss, l->order, l->fwd_in[0], l->fwd_in[1], l->fwd_out[0], l->fwd_out[1]};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (l->h_err) cudaFreeHost(l->h_err);
    if (l->stream2) cudaStreamDestroy(l->stream2);
    if (l->stream) cudaStreamDestroy(l->stream);
    delete l;
    return SPH_OK;
}

int sph_learned_get_params(sph_learned_t *l, float *out)
{
    if (!l || !out) {
        set_error("null argument");
        return SPH_ERR_INVALID;
    }
    LCUDA(cudaMemcpy(out, l->w, ml::NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    return SPH_OK;
}

int sph_learned_set_params(sph_learned_t *l, const float *in)
{
    if (!l || !in) {
        set_error("null argument");
        return SPH_ERR_INVALID;
    }
    std::lock_guard<std::mutex> one_call(l->busy);
    LCUDA(cudaMemcpyAsync(l->w, in, ml::NPARAM * sizeof(float), cudaMemcpyHostToDevice, l->stream));
    LCUDA(cudaMemsetAsync(l->m, 0, ml::NPARAM * sizeof(float), l->stream));
    LCUDA(cudaMemsetAsync(l->v, 0, ml::NPARAM * sizeof(float), l->stream));
    LCUDA(cudaMemsetAsync(l->d_err, 0, sizeof(unsigned), l->stream));
    ml::k_f32_to_bf16<<<nblk(ml::NPARAM), 256, 0, l->stream>>>(ml::NPARAM, l->w, l->wbf);
    LCUDA(cudaStreamSynchronize(l->stream));
    l->adam_t = 0;
    return SPH_OK;
}

int sph_learned_gemm_check(const float *A, const float *B, float *C, int M, int N, int K)
{
    if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) {
        set_error("gemm_check: bad arguments");
        return SPH_ERR_INVALID;
    }
    LTRY(configure_kernels());
    cudaStream_t st = nullptr;
    LCUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    std::vector<__nv_bfloat16> a((size_t)M * K), b((size_t)N * K);
    for (size_t e = 0; e < a.size(); ++e) a[e] = __float2bfloat16(A[e]);
    for (size_t e = 0; e < b.size(); ++e) b[e] = __float2bfloat16(B[e]);
    __nv_bfloat16 *da = nullptr, *db = nullptr;
    float *dc = nullptr;
    unsigned *derr = nullptr;
    int rc = SPH_OK;
    if ((rc = cuda_fail(cudaMalloc(&da, a.size() * 2), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&db, b.size() * 2), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&dc, (size_t)M * N * 4), "cudaMalloc")) ||
        (rc = cuda_fail(cudaMalloc(&derr, 4), "cudaMalloc"))) {
    } else {
        cudaMemcpyAsync(da, a.data(), a.size() * 2, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(db, b.data(), b.size() * 2, cudaMemcpyHostToDevice, st);
        cudaMemsetAsync(derr, 0, 4, st);
        rc = gemm(st, M, N, K, da, K, 1, db, K, 1, dc, N, derr);
        unsigned e = 0;
        if (rc == SPH_OK) {
            cudaMemcpyAsync(C, dc, (size_t)M * N * 4, cudaMemcpyDeviceToHost, st);
            cudaMemcpyAsync(&e, derr, 4, cudaMemcpyDeviceToHost, st);
            rc = cuda_fail(cudaStreamSynchronize(st), "gemm sync");
        }
        if (rc == SPH_OK && e) {
            set_error("tensor-core wait gave up");
            rc = SPH_ERR_CUDA;
        }
    }
    cudaFree(da);
    cudaFree(db);
    cudaFree(dc);
    cudaFree(derr);
    cudaStreamDestroy(st);
    return rc;
}

int sph_learned_forward(sph_learned_t *l, const float *features, int n, float *out)
{
    if (!l || (n > 0 && (!features || !out)) || n < 0) {
        set_error("forward: bad arguments");
        return SPH_ERR_INVALID;
    }
    if (n == 0) return SPH_OK;
    LTRY(configure_kernels());
    std::lock_guard<std::mutex> one_call(l->busy);
    // the caller's rows go to the device as they are, kForwardRows at a time
    // on two streams, so that the copies of one piece can overlap the
    // kernel and the copies of another
    const int nbuf = n > kForwardRows ? 2 : 1;
    // outputs that overlap the features: nothing may be written to them
    // before every row is read
    const bool overlap = (uintptr_t)out < (uintptr_t)(features + (size_t)n * ml::IN) &&
                         (uintptr_t)features < (uintptr_t)(out + (size_t)n * ml::OUT);
    std::vector<float> copy;
    if (overlap && nbuf > 1) {
        copy.assign(features, features + (size_t)n * ml::IN);
        features = copy.data();
    }
    for (int b = 0; b < nbuf; ++b) LTRY(ensure_forward(l, b, std::min(n, kForwardRows)));
    // a few rows: read and written in the caller's memory (kInPlaceRows)
    const size_t in_bytes = (size_t)n * ml::IN * sizeof(float), out_bytes = (size_t)n * ml::OUT * sizeof(float);
    const float *own_in = nullptr;
    float4 *own_out = nullptr;
    if (!overlap && in_bytes <= kInPlaceRows) {
        own_in = static_cast<const float *>(host_in_place(features, in_bytes, 16, false));
        own_out = static_cast<float4 *>(host_in_place(out, out_bytes, 16, true));
    }
    PageToucher pages(out, overlap || own_out ? 0 : out_bytes);
    int rc = SPH_OK, k = 0;
    for (int i0 = 0; i0 < n && rc == SPH_OK; i0 += kForwardRows, k ^= 1) {
        const int rows = std::min(n - i0, kForwardRows);
        cudaStream_t st = k ? l->stream2 : l->stream;
        if (!own_in)
            rc = cuda_fail(cudaMemcpyAsync(l->fwd_in[k], features + (size_t)i0 * ml::IN,
                                           (size_t)rows * ml::IN * sizeof(float),
                                           cudaMemcpyHostToDevice, st),
                           "feature rows");
        if (rc != SPH_OK) break;
        ml::k_mlp<true><<<std::min((rows + 127) / 128, num_sms()), ml::kMlpThreads, mlp_smem(), st>>>(
            rows, own_in ? own_in : l->fwd_in[k], l->wbf, l->w, own_out ? own_out : l->fwd_out[k], l->h_err);
        rc = cuda_fail(cudaGetLastError(), "mlp launch");
        pages.done();
        if (rc == SPH_OK && !own_out)
            rc = cuda_fail(cudaMemcpyAsync(out + (size_t)i0 * ml::OUT, l->fwd_out[k],
                                           (size_t)rows * ml::OUT * sizeof(float),
                                           cudaMemcpyDeviceToHost, st),
                           "network outputs");
    }
    const int rs = cuda_fail(cudaStreamSynchronize(l->stream), "forward");
    const int rs2 = nbuf > 1 ? cuda_fail(cudaStreamSynchronize(l->stream2), "forward") : SPH_OK;
    if (rc != SPH_OK || rs != SPH_OK || rs2 != SPH_OK) return rc != SPH_OK ? rc : rs != SPH_OK ? rs : rs2;
    if (*l->h_err) {
        *l->h_err = 0u;
        set_error("tensor-core wait gave up (mbarrier not completed)");
        return SPH_ERR_CUDA;
    }
    return SPH_OK;
}

int sph_learned_features(sph_cuda_t *h, float *features, int *counts)
{
    if (!h || !features) {
        set_error("features: null argument");
        return SPH_ERR_INVALID;
    }
    const int n = h->n;
    if (n == 0) return SPH_OK;
    LTRY(predicted_features(h, nullptr));
    PageToucher row_pages(features, (size_t)n * ml::IN * sizeof(float));
    PageToucher count_pages(counts, counts ? (size_t)n * sizeof(int) : 0);
    // by id, kFeaturePiece particles at a time (a bounded scratch)
    const int piece = std::min(n, kFeaturePiece);
    LTRY(ensure_scratch(h, (size_t)piece * (ml::IN * sizeof(float) + sizeof(int)) + 256));
    float *rows = (float *)h->d_scratch;
    int *cnt = (int *)(rows + (size_t)piece * ml::IN);
    for (int lo = 0; lo < n; lo += piece) {
        const int m = std::min(piece, n - lo);
        ml::k_rows_by_id<<<nblk(4ll * n), kBlock, 0, h->stream>>>(
            n, lo, m, h->id_c, (const __nv_bfloat16 *)h->feat_c, h->nbc_c, rows, cnt);
        LCUDA(cudaGetLastError());
        row_pages.done();
        LCUDA(cudaMemcpyAsync(features + (size_t)lo * ml::IN, rows, (size_t)m * ml::IN * sizeof(float),
                              cudaMemcpyDeviceToHost, h->stream));
        if (counts) {
            count_pages.done();
            LCUDA(cudaMemcpyAsync(counts + lo, cnt, (size_t)m * sizeof(int), cudaMemcpyDeviceToHost,
                                  h->stream));
        }
    }
    LCUDA(cudaStreamSynchronize(h->stream));
    return SPH_OK;
}

namespace {

// Samples of h's predicted state: features and plain displacements of the
// selected particles appended at l->nsamples.  fraction >= 1 takes every
// eligible particle.  Returns the number appended in *added.
int collect_samples(LearnedModel *l, sph_cuda *h, float fraction, int *added)
{
    *added = 0;
    const int n = h->n;
    if (n == 0) return SPH_OK;
    LTRY(predicted_features(h, nullptr));
    // scratch: displacements, selection flags and their prefix sums (16-byte
    // aligned, as the scan needs them)
    const size_t db = (((size_t)n * 8) + 255) & ~(size_t)255;
    const size_t fb = (((size_t)n + 1) * 4 + 255) & ~(size_t)255;
    LTRY(ensure_scratch(h, db + 2 * fb));
    float2 *disp = (float2 *)h->d_scratch;
    unsigned *flag = (unsigned *)((char *)h->d_scratch + db);
    int *off = (int *)((char *)h->d_scratch + db + fb);
    // plain displacement (C order) through the learned relaxation with every
    // particle forced to fall back
    const float thr = h->learned_thr;
    sph::LearnedModel *keep = h->learned;
    h->learned_thr = -1.0f;
    int rc = launch_learned_relax(h, disp);
    h->learned_thr = thr;
    h->learned = keep;
    LTRY(rc);
    const unsigned long long salt = ml::mix64(l->seed ^ (0xA5A5A5A5ull + l->calls));
    const double frac = std::min(1.0, std::max(0.0, (double)fraction));
    const int room = std::max(0, l->cap - l->nsamples);
    ml::k_select<<<nblk(n), kBlock, 0, h->stream>>>(n, h->nbc_c, h->id_c, salt, frac, flag);
    LTRY(launch_prefix(h, flag, n, off));
    ml::k_append<<<nblk(n), kBlock, 0, h->stream>>>(
        make_ctx(h), room, flag, off, (const __nv_bfloat16 *)h->feat_c, disp,
        l->X + (size_t)l->nsamples * ml::IN, l->T + l->nsamples, l->slot + l->nsamples);
    LCUDA(cudaGetLastError());
    int total = 0;
    LCUDA(cudaMemcpyAsync(&total, off + n, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    LCUDA(cudaStreamSynchronize(h->stream));
    const int rows = std::min(total, room);
    l->nsamples += rows;
    ++l->calls;
    *added = rows;
    return SPH_OK;
}

}  // namespace

int sph_learned_collect(sph_learned_t *l, sph_cuda_t *h, float fraction, int *added)
{
    if (!l || !h) {
        set_error("collect: null argument");
        return SPH_ERR_INVALID;
    }
    int got = 0;
    LTRY(collect_samples(l, h, fraction, &got));
    if (added) *added = got;
    return SPH_OK;
}

int sph_learned_num_samples(sph_learned_t *l)
{
    return l ? l->nsamples : 0;
}

int sph_learned_clear_samples(sph_learned_t *l)
{
    if (!l) {
        set_error("null model");
        return SPH_ERR_INVALID;
    }
    l->nsamples = 0;
    return SPH_OK;
}

int sph_learned_train(sph_learned_t *l, int epochs, int batch, float lr, float *loss)
{
    if (!l || epochs <= 0 || batch <= 0 || !(lr > 0.0f)) {
        set_error("train: bad arguments");
        return SPH_ERR_INVALID;
    }
    return train_loop(l, 0, l->nsamples, epochs, batch, lr, 0x3, true, loss);
}

int sph_learned_calibrate(sph_learned_t *l, sph_cuda_t *h, int epochs, float lr, float *loss)
{
    if (!l || !h || epochs <= 0 || !(lr > 0.0f)) {
        set_error("calibrate: bad arguments");
        return SPH_ERR_INVALID;
    }
    const int n = h->n;
    if (n == 0) return SPH_OK;
    // every eligible particle of the predicted state, appended after the
    // training samples (dropped again afterwards)
    const int base = l->nsamples;
    int rows = 0;
    LTRY(collect_samples(l, h, 1.0f, &rows));
    int rc = SPH_OK;
    float2 *dnet = nullptr, *dplain = nullptr;
    float *rn = nullptr, *rp = nullptr;
    do {
        if ((rc = cuda_fail(cudaMalloc(&dnet, (size_t)n * 8), "cudaMalloc")) ||
            (rc = cuda_fail(cudaMalloc(&dplain, (size_t)n * 8), "cudaMalloc")) ||
            (rc = cuda_fail(cudaMalloc(&rn, (size_t)n * 4), "cudaMalloc")) ||
            (rc = cuda_fail(cudaMalloc(&rp, (size_t)n * 4), "cudaMalloc")))
            break;
        // plain displacement: everyone falls back
        const float thr = h->learned_thr;
        h->learned_thr = -1.0f;
        rc = launch_learned_relax(h, dplain);
        h->learned_thr = thr;
        if (rc) break;
        // network displacement of the same state
        if ((rc = cuda_fail(cudaMemsetAsync(l->d_err, 0, 4, h->stream), "memset")) ||
            (rc = cuda_fail(cudaStreamSynchronize(l->stream), "sync")))
            break;
        if ((rc = run_mlp(h->stream, l, n, (const __nv_bfloat16 *)h->feat_c, h->net_c, h->num_sms)))
            break;
        const Ctx c = make_ctx(h);
        const unsigned *occ = &h->d_state->build_max_occ[SLOT_PREDICTED];
        ml::k_net_disp<<<nblk(n), kBlock, 0, h->stream>>>(c, h->net_c, dnet);
        ml::k_density_displaced<<<nblk(n), kBlock, 0, h->stream>>>(c, h->pos_c, dnet, h->start_c,
                                                                   occ, rn);
        ml::k_density_displaced<<<nblk(n), kBlock, 0, h->stream>>>(c, h->pos_c, dplain,
                                                                   h->start_c, occ, rp);
        if (rows > 0)
            ml::k_err_targets<<<nblk(rows), kBlock, 0, h->stream>>>(c, rn, rp, l->slot + base, rows,
                                                                    l->T + base);
        rc = cuda_fail(cudaStreamSynchronize(h->stream), "calibrate");
        if (rc == SPH_OK) rc = check_err(l);
    } while (false);
    cudaFree(dnet);
    cudaFree(dplain);
    cudaFree(rn);
    cudaFree(rp);
    if (rc == SPH_OK) rc = train_loop(l, base, rows, epochs, 4096, lr, 0x4, false, loss);
    l->nsamples = base;
    return rc;
}

int sph_cuda_set_learned(sph_cuda_t *h, sph_learned_t *l, float threshold)
{
    if (!h) {
        set_error("null handle");
        return SPH_ERR_INVALID;
    }
    LCUDA(cudaStreamSynchronize(h->stream));
    if (l) {
        LTRY(configure_kernels());
        LTRY(ensure_learned_buffers(h));
        // the weights are written on the model's stream and read on the handle's
        LCUDA(cudaStreamSynchronize(l->stream));
    }
    h->learned = l;
    h->learned_thr = threshold;
    const unsigned long long zero[2] = {0ull, 0ull};
    LCUDA(cudaMemcpy(&h->d_state->learned_steps, zero, sizeof(zero), cudaMemcpyHostToDevice));
    destroy_graph(h);  // the step changes
    return SPH_OK;
}

int sph_cuda_learned_counts(sph_cuda_t *h, unsigned long long *learned, unsigned long long *fallback)
{
    if (!h || !learned || !fallback) {
        set_error("null argument");
        return SPH_ERR_INVALID;
    }
    unsigned long long v[2];
    LCUDA(cudaMemcpyAsync(v, &h->d_state->learned_steps, sizeof(v), cudaMemcpyDeviceToHost,
                          h->stream));
    LCUDA(cudaStreamSynchronize(h->stream));
    if (h->learned) {
        // a tensor-core wait that gave up inside a step leaves its tiles'
        // outputs unwritten: report it here rather than hide it
        unsigned e = 0;
        LCUDA(cudaMemcpy(&e, h->learned->d_err, sizeof(e), cudaMemcpyDeviceToHost));
        if (e) {
            set_error("the network kernel's tensor-core wait gave up %u times: results of "
                      "the learned steps are not valid", e);
            return SPH_ERR_CUDA;
        }
    }
    const unsigned long long total = v[0] * (unsigned long long)h->n;
    *fallback = v[1];
    *learned = total >= v[1] ? total - v[1] : 0ull;
    return SPH_OK;
}

}  // extern "C"
