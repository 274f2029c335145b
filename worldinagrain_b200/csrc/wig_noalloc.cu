// wig_noalloc.cu — an entry point that allocates no device memory: the
// FP64 squared norm of the pressure solve's residual, for callers that own
// every byte of device memory themselves.
//
// Why it exists: wig_fluid_create allocates the handle's scratch (the FP64
// per-block partial sums among it) with cudaMalloc.  Some hosts cannot let a
// library do that: a host that records its work into a CUDA graph while it
// runs (cudaMalloc is not allowed during stream capture), a host whose device
// memory is one pre-reserved pool carved up by its own allocator (a game or
// simulation engine, or a WebGPU bridge that imports buffers it does not
// own), and a host on a real-time path that cannot take the device-wide
// synchronisation cudaMalloc may imply.  Such a host drives the liquid's
// buffers itself and still wants to know how far the solve got.
//
// The scratch this needs, one FP64 partial per 8x8 block, lives in a
// file-scope static __device__ array of WIG_NOALLOC_MAX_BLOCKS entries
// (128 KiB): every GPU that loads this library holds it until the process
// exits.  The array's name in host code is only a host-side stand-in, so the
// host takes the array's device address once per device with
// cudaGetSymbolAddress (the first call on a device does that set-up) and
// passes it to the kernels.  That address is kept until
// wig_fluid_noalloc_forget_device, which a host that resets a device calls.  Every call shares the one array: calls whose
// work overlaps on the GPU (two streams, or two host threads) race on it, and
// their results are worth nothing.  The calls after them are sound: each
// call's count of finished CTAs is a word of its own.

#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>

#include "wig_device.cuh"
#include "wig_sums.cuh"

namespace {

constexpr uint32_t MAX_DEVICES = 64;

// One FP64 partial sum per block; a call writes the entries of all its
// world's blocks before it reads any, so nothing in it has to start at zero.
static __device__ __align__(256) double g_block_partials[WIG_NOALLOC_MAX_BLOCKS];
// The CTAs of a call that have written theirs: a word a call, 0 before it and
// put back to 0 by its last CTA, so that a call's count is its own whatever
// overlaps it.  (One word for all of them, with overlapping calls of other
// grids counted into it, could be left at any value, and every call after it
// summed too early or not at all.)  The calls take the first COUNTERS words in
// turn; a captured call, whose word its graph's replays use for as long as
// they please, takes one of the others and sets it to 0 itself ahead of the
// launch (a node of the graph; ahead of every call it would cost about as
// much as a sixth of it).
constexpr uint32_t COUNTERS = 1024;
static __device__ uint32_t g_done[2u * COUNTERS];

std::mutex g_mutex;
std::atomic<uint32_t> g_calls{0};
struct Scratch {
    double* partials;
    uint32_t* done;
};
Scratch g_scratch_of[MAX_DEVICES] = {};

int set_error(int code, const std::string& msg) {
    wig::set_last_error(msg);
    return code;
}

// The squared residual of the liquid cells of each block worked on (cg's y,
// the CG residual r, where field's z > 0), a warp a block: lane l its cells
// l and l + 32, the block's tree of 64 as the step's tolerance form sums it;
// +0 for a block not worked on (its state word's ACTIVE not set).  The last
// CTA to write its blocks' sums adds them in the step's order (sumColumns).
// One launch: as a launch of 64-thread blocks and one of a single CTA that
// read each block's state and partial in turn, the call took 16.4 us on a
// 1024 x 1024 world.
constexpr int NORM_THREADS = 512, NORM_WARPS = NORM_THREADS / 32;
__global__ void __launch_bounds__(NORM_THREADS, 2) k_r2(uint32_t W, uint32_t H, uint32_t B, uint32_t BW, const uint32_t* blocks,
                                                        const float4* field, const float4* cg, double* partials, uint32_t* done,
                                                        double* out) {
    __shared__ double s[256];
    __shared__ int last;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t n = blockIdx.x * NORM_WARPS + (threadIdx.x >> 5); n < B; n += gridDim.x * NORM_WARPS) {
        double v[2] = {0.0, 0.0};
        if ((blocks[B + n] & 1u) != 0u) {
            const uint32_t bx = n % BW, by = n / BW;
            const uint32_t x = bx * 8u + (lane & 7u);
#pragma unroll
            for (uint32_t h = 0; h < 2u; h++) {
                const uint32_t y = by * 8u + (lane >> 3) + 4u * h;
                if (x >= W || y >= H) continue;
                const uint32_t i = y * W + x;
                const float z = field[2u * i].z;
                const double r = (double)cg[i].y;
                if (z > 0.0f) v[h] = r * r;
            }
        }
        const double t = wig::warpTree(v[0], v[1]);
        if (lane == 0u) partials[n] = t;
    }
    if (lane == 0u) __threadfence();
    __syncthreads();
    if (threadIdx.x == 0u) {
        last = atomicAdd(done, 1u) + 1u == gridDim.x ? 1 : 0;
        if (last) {
            *done = 0u;
            __threadfence();
        }
    }
    __syncthreads();
    if (!last) return;
    wig::sumColumns<double, 1, NORM_THREADS>(B, partials, s);
    wig::treeColumns<double, 1>(s);
    if (threadIdx.x == 0u) *out = s[0];
}

// The device addresses of g_block_partials and g_done on the current device,
// looked up once per device and kept for the process's life: a host that
// destroys and recreates a device's primary context (cudaDeviceReset) loads
// the module anew, so it must call wig_fluid_noalloc_forget_device afterwards.
int scratch_on_current_device(Scratch* out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(WIG_E_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || (uint32_t)dev >= MAX_DEVICES) return set_error(WIG_E_ARG, "device ordinal past the ones this entry point keeps");
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_scratch_of[dev].partials) {
        void *p = nullptr, *n = nullptr;
        e = cudaGetSymbolAddress(&p, g_block_partials);
        if (e == cudaSuccess) e = cudaGetSymbolAddress(&n, g_done);
        if (e != cudaSuccess) return set_error(WIG_E_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        g_scratch_of[dev] = Scratch{static_cast<double*>(p), static_cast<uint32_t*>(n)};
    }
    *out = g_scratch_of[dev];
    return WIG_OK;
}

// The word a call on stream s counts its CTAs in, 0 by the time its kernel runs.
cudaError_t counter_of(cudaStream_t s, uint32_t* done, uint32_t** out) {
    const uint32_t k = g_calls.fetch_add(1u) % COUNTERS;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    // (the legacy stream cannot be asked while another is captured; nor can
    // it be launched on, as the launch then says)
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
        cudaGetLastError();
        cs = cudaStreamCaptureStatusNone;
    }
    if (cs == cudaStreamCaptureStatusNone) {
        *out = done + k;
        return cudaSuccess;
    }
    *out = done + COUNTERS + k;
    return cudaMemsetAsync(*out, 0, sizeof(uint32_t), s);
}

}  // namespace

extern "C" {

int wig_fluid_residual_norm2_noalloc(const wig_world_desc* d, const void* field, const void* blocks, const void* cg,
                                     double* out, void* stream) {
    if (!d || !field || !blocks || !cg || !out) return set_error(WIG_E_ARG, "null argument");
    if (d->width == 0 || d->height == 0 || d->width > 32768 || d->height > 32768)
        return set_error(WIG_E_ARG, "world size out of range (1..32768 per side)");
    const uint32_t BW = (d->width + 7u) / 8u, BH = (d->height + 7u) / 8u;
    const uint64_t B = (uint64_t)BW * BH;
    if (B > WIG_NOALLOC_MAX_BLOCKS)
        return set_error(WIG_E_ARG, "world has " + std::to_string(B) + " blocks; the allocation-free entry point holds at most " +
                                        std::to_string(WIG_NOALLOC_MAX_BLOCKS) + " (a 1024 x 1024 world)");
    Scratch scratch{};
    int rc = scratch_on_current_device(&scratch);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t* done = nullptr;
    cudaError_t e = counter_of(s, scratch.done, &done);
    if (e != cudaSuccess) return set_error(WIG_E_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
    const unsigned need = (unsigned)((B + NORM_WARPS - 1u) / NORM_WARPS), grid = need < 148u * 2u ? need : 148u * 2u;
    k_r2<<<grid, NORM_THREADS, 0, s>>>(d->width, d->height, (uint32_t)B, BW, (const uint32_t*)blocks, (const float4*)field,
                                       (const float4*)cg, scratch.partials, done, out);
    e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(WIG_E_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    return WIG_OK;
}

int wig_fluid_noalloc_forget_device(void) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(WIG_E_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || (uint32_t)dev >= MAX_DEVICES) return set_error(WIG_E_ARG, "device ordinal past the ones this entry point keeps");
    std::lock_guard<std::mutex> lock(g_mutex);
    g_scratch_of[dev] = Scratch{};
    return WIG_OK;
}

}  // extern "C"
