// sph_noalloc.cu -- a density pass that allocates no memory.
//
// Some callers of this library cannot call cudaMalloc: a step loop that owns
// a fixed device-memory budget handed out by another framework's allocator,
// or a real-time loop (the render-driven compute rank) that must not take the
// device-wide synchronisation a cudaMalloc/cudaFree can imply.  For them,
// sph_cuda_density_static() computes the reference's density and near
// density (hash_fluid(.., true) + calculate_density, hash.c:127-242 /
// fluid.c:527-539) of caller-owned device arrays, keeping every intermediate
// (cell keys, histogram, cell starts, sorted copies) in the file-scope array
// below, whose size is fixed at compile time.  Every GPU that loads the
// library holds that array (about 4 MB) until the process exits.
#include <mutex>

#include "sph_internal.h"

namespace sph {

namespace {

constexpr size_t kAlign = 256;
constexpr size_t up(size_t b) { return (b + kAlign - 1) / kAlign * kAlign; }

constexpr size_t kN = SPH_STATIC_MAX_PARTICLES;
constexpr size_t kC = SPH_STATIC_MAX_CELLS;
constexpr size_t kTiles = (kC + 1 + kBuildTile - 1) / kBuildTile;

// Layout of the scratch array (byte offsets, each 256-byte aligned).
constexpr size_t kNocellWords = (kC + 1 + 31) / 32 + 1;
constexpr size_t kOffScene = 0;
constexpr size_t kOffPoff = kOffScene + up(sizeof(Scene));
constexpr size_t kOffNocell = kOffPoff + up(2 * sizeof(int));
constexpr size_t kOffState = kOffNocell + up(kNocellWords * sizeof(unsigned));
constexpr size_t kOffCnt = kOffState + up(sizeof(DevState));
constexpr size_t kOffStart = kOffCnt + up((kC + 1) * sizeof(unsigned));
constexpr size_t kOffTiles = kOffStart + up((kC + 2) * sizeof(int));
constexpr size_t kOffPosIn = kOffTiles + up(kTiles * sizeof(int));
constexpr size_t kOffKr = kOffPosIn + up(kN * sizeof(float2));
constexpr size_t kOffTmp = kOffKr + up(kN * sizeof(uint2));
constexpr size_t kOffPosS = kOffTmp + up(kN * sizeof(int));
constexpr size_t kOffIdS = kOffPosS + up(kN * sizeof(float2));
constexpr size_t kScratchBytes = kOffIdS + up(kN * sizeof(int));
// the sorted positions are read up to kRowPad past their end
static_assert(kScratchBytes - kOffIdS >= kRowPad * sizeof(float2), "padding after the sorted positions");

}  // namespace

// The scratch of sph_cuda_density_static: shared by every call on a device.
static __device__ __align__(256) unsigned char g_static_scratch[kScratchBytes];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
void *g_scratch_addr[kMaxDevices] = {};

// Device address of g_static_scratch on the current device (the host-side
// name of the array is only a stand-in).  Looked up again on every call that
// is not being captured into a graph, so that a context torn down and
// recreated (cudaDeviceReset) is seen; a call under stream capture uses the
// address of the last call on this device outside capture, which must
// exist.
int scratch_address(cudaStream_t stream, void **out)
{
    int dev = 0;
    int rc = cuda_fail(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc != SPH_OK) return rc;
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("device ordinal %d above %d", dev, kMaxDevices - 1);
        return SPH_ERR_UNSUPPORTED;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    rc = cuda_fail(cudaStreamIsCapturing(stream, &cap), "cudaStreamIsCapturing");
    if (rc != SPH_OK) return rc;
    std::lock_guard<std::mutex> lock(g_setup_mu);
    if (cap == cudaStreamCaptureStatusNone) {
        void *p = nullptr;
        rc = cuda_fail(cudaGetSymbolAddress(&p, g_static_scratch), "cudaGetSymbolAddress");
        if (rc != SPH_OK) return rc;
        g_scratch_addr[dev] = p;
    } else if (!g_scratch_addr[dev]) {
        set_error("sph_cuda_density_static: the first call on a device must come before any "
                  "stream capture");
        return SPH_ERR_STATE;
    }
    *out = g_scratch_addr[dev];
    return SPH_OK;
}

// The counters of the last call's cell build, into caller device memory.
__global__ void k_static_counters(sph_cuda_counters *out)
{
    const DevState *st = reinterpret_cast<const DevState *>(g_static_scratch + kOffState);
    sph_cuda_counters c;
    c.steps = 0ull;
    c.out_of_grid = st->out_of_grid;
    c.bucket_overflow = st->bucket_overflow;
    c.max_cell_occupancy = st->max_occ;
    c.list_cap_risk = st->list_cap_risk;
    *out = c;
}

}  // namespace
}  // namespace sph

using namespace sph;

extern "C" int sph_cuda_density_static_counters(sph_cuda_counters *d_out, void *stream)
{
    if (!d_out) {
        set_error("sph_cuda_density_static_counters: null device output");
        return SPH_ERR_INVALID;
    }
    // the kernel names the array itself: no device address is needed here
    k_static_counters<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(d_out);
    return cuda_fail(cudaGetLastError(), "sph_cuda_density_static_counters launch");
}

extern "C" int sph_cuda_density_static(const float *x, const float *y, int n,
                                       const neighbor_grid_t *grid, const tunable_parameters *tp,
                                       float *density, float *density_near, void *stream)
{
    if (!grid || !tp) {
        set_error("sph_cuda_density_static: null grid or tunables");
        return SPH_ERR_INVALID;
    }
    if (n < 0 || n > SPH_STATIC_MAX_PARTICLES) {
        set_error("sph_cuda_density_static: %d particles, the static scratch holds at most %d", n,
                  SPH_STATIC_MAX_PARTICLES);
        return n < 0 ? SPH_ERR_INVALID : SPH_ERR_CAPACITY;
    }
    const unsigned long long cells = (unsigned long long)grid->size_x * grid->size_y;
    if (!(grid->spacing > 0.0f) || cells == 0 || grid->max_bucket_size == 0 ||
        grid->max_neighbors == 0) {
        set_error("sph_cuda_density_static: invalid neighbour grid");
        return SPH_ERR_INVALID;
    }
    if (cells > SPH_STATIC_MAX_CELLS) {
        set_error("sph_cuda_density_static: %llu grid cells, the static scratch holds at most %d",
                  cells, SPH_STATIC_MAX_CELLS);
        return SPH_ERR_CAPACITY;
    }
    if (!(tp->smoothing_radius > 0.0f)) {
        set_error("sph_cuda_density_static: smoothing_radius must be positive");
        return SPH_ERR_INVALID;
    }
    if (n > 0 && (!x || !y || !density || !density_near)) {
        set_error("sph_cuda_density_static: null device array");
        return SPH_ERR_INVALID;
    }
    void *base_v = nullptr;
    int rc = scratch_address(static_cast<cudaStream_t>(stream), &base_v);
    if (rc != SPH_OK) return rc;
    if (n == 0) return SPH_OK;

    char *base = static_cast<char *>(base_v);
    StaticArrays a;
    a.scene = reinterpret_cast<Scene *>(base + kOffScene);
    a.p_off = reinterpret_cast<int *>(base + kOffPoff);
    a.nocell = reinterpret_cast<unsigned *>(base + kOffNocell);
    a.state = reinterpret_cast<DevState *>(base + kOffState);
    a.cnt = reinterpret_cast<unsigned *>(base + kOffCnt);
    a.start = reinterpret_cast<int *>(base + kOffStart);
    a.tile_cnt = reinterpret_cast<unsigned *>(base + kOffTiles);
    a.pos_in = reinterpret_cast<float2 *>(base + kOffPosIn);
    a.kr = reinterpret_cast<uint2 *>(base + kOffKr);
    a.tmp = reinterpret_cast<int *>(base + kOffTmp);
    a.pos_s = reinterpret_cast<float2 *>(base + kOffPosS);
    a.id_s = reinterpret_cast<int *>(base + kOffIdS);

    Scene sc{};
    sc.P = *tp;
    sc.spacing = grid->spacing;
    sc.size_x = (int)grid->size_x;
    sc.size_y = (int)grid->size_y;
    sc.ncells = (int)cells;
    sc.c_off = 0;
    sc.p_off = 0;
    sc.n = n;
    sc.max_bucket = (int)grid->max_bucket_size;
    sc.max_neighbors = (int)grid->max_neighbors;
    return launch_static_density(sc, a, x, y, density, density_near,
                                 static_cast<cudaStream_t>(stream));
}
