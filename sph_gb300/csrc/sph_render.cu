// sph_render.cu -- the render rank's liquid-surface image as compute
// kernels into device buffers (no graphics API): the four passes of
// draw_liquid (liquid_gl.c:305-447) at the reduced texture resolution
// (screen / 2, liquid_gl.c:43-48) and the composite at screen resolution.
//
//   1 k_splat      metaball point sprites (shaders/liquid_particle.frag:10-20):
//                  intensity 1 - 3 r^2 for r^2 <= 0.34 (r in units of the
//                  sprite radius), additive blending into an 8-bit alpha
//                  texture (liquid_gl.c:318-343, 106): every fragment adds
//                  round(255 i), the sum saturates at 255.  Integer atomics
//                  make the result independent of the drawing order.
//   2 k_blur<V>    15-tap Gaussian along y, then along x
//                  (shaders/vert_blur.vert:12-26, horz_blur.vert,
//                  blur.frag:12-29): taps at +-0.004 k texture units,
//                  bilinear filtering with clamp to edge (liquid_gl.c:107-110),
//                  each pass stored back to 8 bits.
//   3 k_composite  shaders/render_liquid_texture.frag:11-17 at screen size:
//                  alpha a (bilinear), discard below 0.1, colour
//                  (w, w, 1) with w = smoothstep(-0.15, -0.1, -a) blended
//                  with alpha 0.75 smoothstep(0.1, 0.11, a) over a black
//                  background (liquid_gl.c:436-444).
// The blur passes' texture-coordinate flips (liquid_gl.c:146-160 and
// render_liquid_texture.vert) cancel in pairs and the kernel is symmetric,
// so images are kept bottom row first until the final file order.
#include <algorithm>
#include <cmath>

#include "sph_device.cuh"

namespace sph {
namespace render {

// Gaussian taps of blur.frag (centre, then +-1 .. +-7 in steps of 0.004).
__constant__ float kTap[8] = {0.159576912161f, 0.147308056121f, 0.115876621105f,
                              0.0776744219933f, 0.0443683338718f, 0.0215963866053f,
                              0.00895781211794f, 0.0044299121055113265f};

// Sprite geometry: points are the packed shorts / SHRT_MAX in [-1, 1]
// (renderer.c:333-337); the sprite diameter is 0.020 of the screen width
// (renderer.c:224), divided by the texture reduction (liquid_gl.c:77).
struct Sprite {
    float cx, cy;
    int x0, x1, y0, y1;
};

__device__ __forceinline__ Sprite sprite_of(short2 c, int w, int h, float radius)
{
    Sprite s;
    const float px = (float)c.x / 32767.0f, py = (float)c.y / 32767.0f;
    s.cx = (px + 1.0f) * 0.5f * (float)w;
    s.cy = (py + 1.0f) * 0.5f * (float)h;
    const float reach = 0.5831f * radius + 1.0f;  // sqrt(0.34) = 0.5831
    s.x0 = max(0, (int)floorf(s.cx - reach));
    s.x1 = min(w - 1, (int)ceilf(s.cx + reach));
    s.y0 = max(0, (int)floorf(s.cy - reach));
    s.y1 = min(h - 1, (int)ceilf(s.cy + reach));
    return s;
}

// The sums saturate at 255, and in a fluid of many particles per texel nearly
// every fragment falls on a texel that is full already: a texel read as full
// takes no more atomics, which leaves the saturated image as it is whatever
// the order (a stale read only costs an atomic more).
// `pitch`: texels from row to row, a multiple of 4, so that four texels are
// read at once.
__device__ __forceinline__ void splat_row(const Sprite &s, int y, int pitch, float radius,
                                          unsigned *__restrict__ acc)
{
    const float inv = 1.0f / radius;
    const float dy = ((float)y + 0.5f - s.cy) * inv;
    if (dy * dy > 0.34f) return;  // beside the disc: most rows of a sprite of a few texels
    // the row's span, a texel wider than the disc on either side
    const float half = sqrtf(0.34f - dy * dy) * radius + 1.0f;
    const int xa = max(s.x0, (int)floorf(s.cx - 0.5f - half));
    const int xb = min(s.x1, (int)ceilf(s.cx - 0.5f + half));
    unsigned *row = acc + (size_t)y * pitch;
    // kGroup x 4 texels requested together (1,048,576 particles' image: with
    // one 4 us more, with five, a whole row, 3 us more: the later texels have
    // filled up by the time the first ones are done)
    constexpr int kGroup = 2;
    for (int g4 = xa & ~3; g4 <= xb; g4 += 4 * kGroup) {
        uint4 t[kGroup];
#pragma unroll
        for (int q = 0; q < kGroup; ++q)
            t[q] = g4 + 4 * q <= xb ? __ldcg(reinterpret_cast<const uint4 *>(row + g4 + 4 * q))
                                    : make_uint4(255u, 255u, 255u, 255u);
#pragma unroll
        for (int q = 0; q < kGroup; ++q) {
            if (min(min(t[q].x, t[q].y), min(t[q].z, t[q].w)) >= 255u) continue;
            const unsigned have[4] = {t[q].x, t[q].y, t[q].z, t[q].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = g4 + 4 * q + k;
                const float dx = ((float)x + 0.5f - s.cx) * inv;
                const float r2 = dx * dx + dy * dy;
                if (r2 > 0.34f || x < xa || x > xb || have[k] >= 255u) continue;
                const int v = __float2int_rn((1.0f - 3.0f * r2) * 255.0f);
                if (v > 0) atomicAdd(row + x, (unsigned)v);
            }
        }
    }
}

// Particles 0, step, 2 step, ..., LANES threads each (a sprite is a chain of
// some fifty dependent reads and atomics for one thread); or with `full` (a
// bit per kBlk x kBlk texels, words_x words a row of blocks: every texel of
// the block is full) the others, whose rows of full blocks are left out.  In
// two passes -- a sample of the particles, then the rest against the sample's
// full blocks -- the interior of a fluid costs a few bit tests a particle.
// 1,048,576 particles on 960 x 540 texels: 322 us in one pass with an atomic
// per fragment, 54 us so.  In a large second pass more lanes only send more
// atomics to texels that are about to be full.
constexpr int kBlk = 4;

template <int LANES>
__global__ void __launch_bounds__(256)
k_splat(int n, int step, const short2 *__restrict__ coords, int w, int h, float radius, int pitch,
        unsigned *__restrict__ acc, const unsigned *__restrict__ full, int words_x)
{
    pdl_enter();
    const long long th = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned t = (unsigned)(th / LANES);  // below 2^31, as n is
    const long long i = full ? (long long)t + t / (unsigned)(step - 1) + 1 : (long long)t * step;
    if (i >= n) return;
    const Sprite s = sprite_of(coords[i], w, h, radius);
    if (s.x0 > s.x1) return;
    if (!full) {
        for (int y = s.y0 + (int)(th % LANES); y <= s.y1; y += LANES) splat_row(s, y, pitch, radius, acc);
        return;
    }
    const int bx0 = s.x0 / kBlk, bx1 = s.x1 / kBlk;
    for (int by = s.y0 / kBlk + (int)(th % LANES); by <= s.y1 / kBlk; by += LANES) {
        bool all = true;
        const unsigned *row = full + (size_t)by * words_x;
        for (int q = bx0 >> 5; q <= bx1 >> 5; ++q) {
            const int lo = max(bx0 - 32 * q, 0), hi = min(bx1 - 32 * q, 31);
            const unsigned want = (0xFFFFFFFFu << lo) & (0xFFFFFFFFu >> (31 - hi));
            all = all && (__ldg(row + q) & want) == want;
        }
        if (all) continue;
        const int y1 = min(s.y1, by * kBlk + kBlk - 1);
        for (int y = max(s.y0, by * kBlk); y <= y1; ++y) splat_row(s, y, pitch, radius, acc);
    }
}

// The full blocks of the accumulated texture, a warp per word.
__global__ void __launch_bounds__(256)
k_full_blocks(int w, int h, int pitch, const unsigned *__restrict__ acc, unsigned *__restrict__ full,
              int words_x)
{
    pdl_enter();
    const int bx = blockIdx.x * blockDim.x + threadIdx.x, by = blockIdx.y;
    bool all = bx * kBlk < w;
    for (int y = by * kBlk; y < min(h, (by + 1) * kBlk) && all; ++y)
        for (int x = bx * kBlk; x < min(w, (bx + 1) * kBlk); ++x)
            all = all && acc[(size_t)y * pitch + x] >= 255u;
    const unsigned bits = __ballot_sync(0xffffffffu, all);
    if ((threadIdx.x & 31) == 0 && (bx >> 5) < words_x) full[(size_t)by * words_x + (bx >> 5)] = bits;
}

// Texel values: the accumulated sums, saturated, or 8-bit texels.
__device__ __forceinline__ float texel(const unsigned *__restrict__ t, size_t i)
{
    return (float)min(t[i], 255u);
}
__device__ __forceinline__ float texel(const unsigned char *__restrict__ t, size_t i)
{
    return (float)t[i];
}

// Bilinear sample of an 8-bit texture along one axis at texel coordinate t
// (texel centres at integers), clamped to the edge.
template <class T>
__device__ __forceinline__ float lerp_axis(const T *__restrict__ row, int stride, int len, float t)
{
    const float f = floorf(t);
    const int i0 = (int)f;
    const float a = t - f;
    const int j0 = min(max(i0, 0), len - 1), j1 = min(max(i0 + 1, 0), len - 1);
    return (1.0f - a) * texel(row, (size_t)j0 * stride) + a * texel(row, (size_t)j1 * stride);
}

// One blur pass: VERTICAL along y (offsets in units of the texture height),
// else along x.  Output stored to 8 bits.  The first pass reads the splat's
// sums (saturated as it reads them).
template <bool VERTICAL, class T>
__global__ void k_blur(int w, int h, int pitch, const T *__restrict__ in,
                       unsigned char *__restrict__ out)
{
    pdl_enter();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= w || y >= h) return;
    const int len = VERTICAL ? h : w;
    const int pos = VERTICAL ? y : x;
    const T *line = VERTICAL ? in + x : in + (size_t)y * pitch;
    const int stride = VERTICAL ? pitch : 1;
    float s = kTap[0] * texel(line, (size_t)pos * stride);
#pragma unroll
    for (int k = 1; k <= 7; ++k) {
        const float o = 0.004f * (float)k * (float)len;
        s += kTap[k] * (lerp_axis(line, stride, len, (float)pos - o) +
                        lerp_axis(line, stride, len, (float)pos + o));
    }
    out[(size_t)y * w + x] = (unsigned char)min(255, max(0, __float2int_rn(s)));
}

__device__ __forceinline__ float smoothstep(float e0, float e1, float x)
{
    const float t = fminf(fmaxf((x - e0) / (e1 - e0), 0.0f), 1.0f);
    return t * t * (3.0f - 2.0f * t);
}

// Screen pixel (X, Y) (Y = 0 at the bottom): its RGB8 in the low 24 bits.
__device__ __forceinline__ unsigned composite_pixel(int X, int Y, int W, int H, int w, int h,
                                                    const unsigned char *__restrict__ a)
{
    const float u = ((float)X + 0.5f) / (float)W * (float)w - 0.5f;
    const float v = ((float)Y + 0.5f) / (float)H * (float)h - 0.5f;
    const float fu = floorf(u), fv = floorf(v);
    const int i0 = (int)fu, j0 = (int)fv;
    const float au = u - fu, av = v - fv;
    const int ia = min(max(i0, 0), w - 1), ib = min(max(i0 + 1, 0), w - 1);
    const int ja = min(max(j0, 0), h - 1), jb = min(max(j0 + 1, 0), h - 1);
    const float s00 = a[(size_t)ja * w + ia], s01 = a[(size_t)ja * w + ib];
    const float s10 = a[(size_t)jb * w + ia], s11 = a[(size_t)jb * w + ib];
    const float alpha = ((1.0f - av) * ((1.0f - au) * s00 + au * s01) +
                         av * ((1.0f - au) * s10 + au * s11)) / 255.0f;
    float r = 0.0f, g = 0.0f, b = 0.0f;
    if (alpha >= 0.1f) {
        const float o = 0.75f * smoothstep(0.1f, 0.11f, alpha);
        const float white = smoothstep(-0.15f, -0.1f, -alpha);
        r = white * o;
        g = white * o;
        b = o;
    }
    return (unsigned)(unsigned char)__float2int_rn(r * 255.0f) |
           (unsigned)(unsigned char)__float2int_rn(g * 255.0f) << 8 |
           (unsigned)(unsigned char)__float2int_rn(b * 255.0f) << 16;
}

// The image, top row first.  A thread makes four pixels of a row where the
// width keeps every row's start on a word (WORDS), else one, with byte stores.
// The image may be the caller's own memory (kInPlaceImage).
template <bool WORDS>
__global__ void __launch_bounds__(256)
k_composite(int W, int H, int w, int h, const unsigned char *__restrict__ a,
            unsigned char *__restrict__ rgb)
{
    pdl_enter();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int Y = blockIdx.y;
    if (WORDS) {
        // four pixels a thread, the CTA's bytes by way of shared memory, so
        // that they leave in whole 16-byte pieces
        __shared__ uint4 stage[192];
        if (4 * q < W) {
            unsigned c[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) c[k] = composite_pixel(4 * q + k, Y, W, H, w, h, a);
            unsigned *p = reinterpret_cast<unsigned *>(stage) + 3 * threadIdx.x;
            p[0] = c[0] | c[1] << 24;
            p[1] = c[1] >> 8 | c[2] << 16;
            p[2] = c[2] >> 16 | c[3] << 8;
        }
        __syncthreads();
        constexpr int kBytes = 4 * 3 * 256;  // a CTA's share of the row
        const int at = blockIdx.x * kBytes, bytes = min(kBytes, W * 3 - at);
        unsigned char *row = rgb + (size_t)(H - 1 - Y) * W * 3 + at;
        if (W % 16 == 0) {
            if (16 * (int)threadIdx.x < bytes) reinterpret_cast<uint4 *>(row)[threadIdx.x] = stage[threadIdx.x];
        } else {
            for (int e = threadIdx.x; 4 * e < bytes; e += blockDim.x)
                reinterpret_cast<unsigned *>(row)[e] = reinterpret_cast<unsigned *>(stage)[e];
        }
    } else {
        if (q >= W) return;
        const unsigned c = composite_pixel(q, Y, W, H, w, h, a);
        unsigned char *p = rgb + ((size_t)(H - 1 - Y) * W + q) * 3;
        p[0] = (unsigned char)c;
        p[1] = (unsigned char)(c >> 8);
        p[2] = (unsigned char)(c >> 16);
    }
}

}  // namespace render

int launch_pack(sph_cuda *h, short2 *out);

// Particles from which the splat runs in two passes.  Microseconds an image
// of a dam break (1,280 x 720 / 1,920 x 1,080 / 3,840 x 2,160) in one pass and
// in two: 32,000 particles 68 and 65 / 92 and 95 / 240 and 260, 65,536 88 and
// 62 / 120 and 95 / 265 and 262, 300,000 219 and 73 / 265 and 106 / 424 and
// 272.  Spread evenly over the image, which leaves few blocks full, one pass is
// up to a fifth faster below 1,000,000.
constexpr int kSplatTwoPass = 65536;
// Every how manieth particle the first pass takes: a sixteenth of them, down to
// a sixty-fourth, about 16,384 in between, which fill what the fluid covers
// (300,000 particles, 1,280 x 720: 73 us, a thirty-second 130).
constexpr int kSampleMin = 16, kSampleMax = 64, kSampleSize = 16384;
// Particles up to which the second pass takes them with four lanes, to have the
// GPU filled (200,000, 1,920 x 1,080: 112 us with one, 101 with four; 500,000
// 112 and 119).
constexpr int kSplatFew = 400000;

// The whole image from device coordinates; scratch (render_scratch bytes,
// 256-byte aligned) holds the reduced textures.  *alpha is set to the blurred
// reduced alpha in it.
struct RenderScratch {
    size_t acc, full, t0, t1, total;
    int words_x, blocks_y, pitch;  // pitch of the sums, in texels
};

static RenderScratch render_layout(int W, int H)
{
    const size_t m = (size_t)(W / 2) * (H / 2);
    RenderScratch r;
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const int bx = (W / 2 + render::kBlk - 1) / render::kBlk;
    r.words_x = (bx + 31) / 32;
    r.blocks_y = (H / 2 + render::kBlk - 1) / render::kBlk;
    r.pitch = (W / 2 + 3) & ~3;
    r.acc = 0;
    r.full = r.acc + up((size_t)r.pitch * (H / 2) * 4);
    r.t0 = r.full + up((size_t)r.words_x * r.blocks_y * 4);
    r.t1 = r.t0 + up(m);
    r.total = r.t1 + up(m);
    return r;
}

static size_t render_scratch(int W, int H) { return render_layout(W, H).total; }

static int render_clear(cudaStream_t st, int W, int H, unsigned char *scratch)
{
    const RenderScratch lay = render_layout(W, H);
    return cuda_fail(cudaMemsetAsync(scratch + lay.acc, 0, (size_t)lay.pitch * (H / 2) * 4, st), "clear");
}

// After render_clear: the blurred reduced alpha from device coordinates.
static int render_alpha(cudaStream_t st, const short2 *coords, int n, int W, int H,
                        unsigned char *scratch, unsigned char **alpha)
{
    using namespace render;
    const int w = W / 2, h = H / 2;
    const RenderScratch lay = render_layout(W, H);
    unsigned *acc = reinterpret_cast<unsigned *>(scratch + lay.acc);
    unsigned *full = reinterpret_cast<unsigned *>(scratch + lay.full);
    unsigned char *t0 = scratch + lay.t0, *t1 = scratch + lay.t1;
    const float radius = 0.5f * ((float)W * 0.020f / 2.0f);
    auto blocks = [](long long k) { return (int)((k + 255) / 256); };
    // two passes where the particles are many enough for full blocks to be
    // likely and to pay for the two launches more
    if (n >= kSplatTwoPass) {
        const int step = std::max(kSampleMin, std::min(kSampleMax, n / kSampleSize));
        const int first = (n + step - 1) / step, lanes = n <= kSplatFew ? 4 : 1;
        launch_step(k_splat<8>, blocks((long long)first * 8), 256, 0, st, n, step, coords, w, h, radius,
                    lay.pitch, acc, (const unsigned *)nullptr, 0);
        launch_step(k_full_blocks, dim3((lay.words_x * 32 + 255) / 256, lay.blocks_y), 256, 0, st, w, h,
                    lay.pitch, (const unsigned *)acc, full, lay.words_x);
        launch_step(lanes > 1 ? k_splat<4> : k_splat<1>, blocks((long long)(n - first) * lanes), 256, 0, st, n,
                    step, coords, w, h, radius, lay.pitch, acc, (const unsigned *)full, lay.words_x);
    } else if (n > 0) {
        launch_step(k_splat<8>, blocks((long long)n * 8), 256, 0, st, n, 1, coords, w, h, radius, lay.pitch, acc,
                    (const unsigned *)nullptr, 0);
    }
    const dim3 rows((w + 255) / 256, h);
    launch_step(k_blur<true, unsigned>, rows, 256, 0, st, w, h, lay.pitch, (const unsigned *)acc, t1);
    launch_step(k_blur<false, unsigned char>, rows, 256, 0, st, w, h, w, (const unsigned char *)t1, t0);
    *alpha = t0;
    return cuda_fail(cudaGetLastError(), "render");
}

static int render_composite(cudaStream_t st, const unsigned char *alpha, int W, int H,
                            unsigned char *rgb)
{
    using namespace render;
    const int w = W / 2, h = H / 2;
    if (W % 4 == 0)
        launch_step(k_composite<true>, dim3((W / 4 + 255) / 256, H), 256, 0, st, W, H, w, h,
                    alpha, rgb);
    else
        launch_step(k_composite<false>, dim3((W + 255) / 256, H), 256, 0, st, W, H, w, h,
                    alpha, rgb);
    return cuda_fail(cudaGetLastError(), "composite");
}

static int check_size(int W, int H)
{
    if (W < 2 || H < 2 || W > 16384 || H > 16384) {
        set_error("image size %d x %d outside [2, 16384]", W, H);
        return SPH_ERR_INVALID;
    }
    return SPH_OK;
}

}  // namespace sph

using namespace sph;

extern "C" {

int sph_render_liquid(const short *coords, int n, int width, int height, unsigned char *rgb,
                      unsigned char *alpha)
{
    if ((!coords && n > 0) || n < 0 || !rgb) {
        set_error("sph_render_liquid: bad arguments");
        return SPH_ERR_INVALID;
    }
    int rc = check_size(width, height);
    if (rc) return rc;
    const size_t img = (size_t)width * height * 3, m = (size_t)(width / 2) * (height / 2);
    const size_t cb = (((size_t)n * 4) + 255) & ~(size_t)255;
    unsigned char *buf = nullptr;
    cudaStream_t st = nullptr;
    rc = cuda_fail(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "stream");
    if (rc) return rc;
    const size_t total = cb + ((img + 255) & ~(size_t)255) + render_scratch(width, height);
    rc = cuda_fail(cudaMalloc(&buf, total), "cudaMalloc");
    if (!rc) {
        short2 *d_coords = reinterpret_cast<short2 *>(buf);
        unsigned char *d_rgb = buf + cb;
        unsigned char *scratch = d_rgb + ((img + 255) & ~(size_t)255), *d_alpha = nullptr;
        if (n > 0)
            rc = cuda_fail(cudaMemcpyAsync(d_coords, coords, (size_t)n * 4, cudaMemcpyHostToDevice, st),
                           "coords");
        if (!rc) rc = render_clear(st, width, height, scratch);
        if (!rc) rc = render_alpha(st, d_coords, n, width, height, scratch, &d_alpha);
        if (!rc) rc = render_composite(st, d_alpha, width, height, d_rgb);
        if (!rc) rc = cuda_fail(cudaMemcpyAsync(rgb, d_rgb, img, cudaMemcpyDeviceToHost, st), "image");
        if (!rc && alpha)
            rc = cuda_fail(cudaMemcpyAsync(alpha, d_alpha, m, cudaMemcpyDeviceToHost, st), "alpha");
        if (!rc) rc = cuda_fail(cudaStreamSynchronize(st), "sync");
    }
    cudaStreamSynchronize(st);
    if (buf) cudaFree(buf);
    cudaStreamDestroy(st);
    return rc;
}

int sph_cuda_render_liquid(sph_cuda_t *h, int width, int height, unsigned char *rgb,
                           unsigned char *alpha)
{
    if (!h || !rgb) {
        set_error("sph_cuda_render_liquid: null argument");
        return SPH_ERR_INVALID;
    }
    int rc = check_size(width, height);
    if (rc) return rc;
    const int n = h->n;
    const size_t img = (size_t)width * height * 3, m = (size_t)(width / 2) * (height / 2);
    const size_t cb = (((size_t)n * 4) + 255) & ~(size_t)255;
    const size_t ib = (img + 255) & ~(size_t)255;
    rc = ensure_scratch(h, cb + ib + render_scratch(width, height) + 256);
    if (rc) return rc;
    unsigned char *base = (unsigned char *)h->d_scratch;
    short2 *d_coords = reinterpret_cast<short2 *>(base);
    unsigned char *d_rgb = base + cb, *scratch = d_rgb + ib, *d_alpha = nullptr;
    rc = render_clear(h->stream, width, height, scratch);
    if (rc) return rc;
    if (n > 0) {
        rc = launch_pack(h, d_coords);
        if (rc) return rc;
    }
    rc = render_alpha(h->stream, d_coords, n, width, height, scratch, &d_alpha);
    if (rc) return rc;
    // composed in the caller's memory where the stores are whole 16-byte pieces
    unsigned char *own = nullptr;
    if (width % 16 == 0 && img <= kInPlaceImage)
        own = static_cast<unsigned char *>(host_in_place(rgb, img, 16, true));
    rc = render_composite(h->stream, d_alpha, width, height, own ? own : d_rgb);
    if (!own) {
        PageToucher pages(rgb, img);  // while the kernels run
        pages.done();
        if (!rc)
            rc = cuda_fail(cudaMemcpyAsync(rgb, d_rgb, img, cudaMemcpyDeviceToHost, h->stream), "image");
    }
    if (!rc && alpha)
        rc = cuda_fail(cudaMemcpyAsync(alpha, d_alpha, m, cudaMemcpyDeviceToHost, h->stream), "alpha");
    if (!rc) rc = cuda_fail(cudaStreamSynchronize(h->stream), "sync");
    return rc;
}

}  // extern "C"
