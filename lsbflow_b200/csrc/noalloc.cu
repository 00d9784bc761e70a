// lsb_solve_helmholtz_noalloc: the Helmholtz / Poisson solve of solve_helmholtz for
// callers that are not allowed to allocate GPU memory.
//
// Who needs it: a host program whose device memory is owned by someone else -- a
// pool allocator or framework that hands out every byte and forbids direct
// cudaMalloc -- or a time-stepping loop that cannot afford cudaMalloc / cudaFree,
// which synchronize the whole device.  Such a caller can pass device pointers it
// already holds, but cannot let the library create a handle (lsb_create allocates).
//
// How: the solve is the handle's one-launch form (gemm_kernels.cu), whose intermediate stays
// on the SM; its two matrices are read zero-padded to a multiple of 16, and those copies live
// in one file-scope __device__ array of LSB_NOALLOC_SCRATCH_BYTES, written by a small kernel on
// each call.  Every GPU that loads the library keeps that array for the life of the process.
// The grid size is limited only through nz (nzp <= 129).  At 256 x 64 x 129: 246 us in three
// column chunks of two separate contractions each, 61 us in one launch.
//
// Set-up: the first call on a device looks up the array's device address with
// cudaGetSymbolAddress while that device is current and caches it; make that first
// call outside any stream capture.  Calls share the array and it keeps the last
// call's contents: calls that overlap on the GPU (two streams, or two host threads
// on one device) race on it and must be serialised by the caller.
#include <cuda_runtime.h>

#include <exception>
#include <mutex>
#include <string>

#include "lsb_internal.cuh"
#include "lsbgpu.h"

namespace lsb {
void set_last_error(const std::string& m);  // lsbgpu.cu
}

namespace {

constexpr long long kScratchDoubles = LSB_NOALLOC_SCRATCH_BYTES / 8;
constexpr int kMaxNzp = 129;
constexpr int kMaxP = 128;                // padded nzm
static_assert(2LL * kMaxP * kMaxP <= kScratchDoubles, "two padded matrices fit the scratch");

static __device__ __align__(256) double g_noalloc_scratch[kScratchDoubles];

std::mutex g_mu;
double* g_scratch_ptr[64] = {nullptr};    // device address per device ordinal

// Zero-padded copies [kp][kp] of E^-1 and E (nzm x nzm), written into the scratch (every entry,
// each call).
__global__ void k_pad_mats(const double* __restrict__ e, const double* __restrict__ ei, int nzm, int kp,
                           double* __restrict__ a1, double* __restrict__ a2) {
    const int n = kp * kp;
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < 2 * n; x += gridDim.x * blockDim.x) {
        const int y = x < n ? x : x - n;
        const int r = y / kp, k = y % kp;
        const double* m = x < n ? ei : e;
        (x < n ? a1 : a2)[y] = (r < nzm && k < nzm) ? m[(long long)r * nzm + k] : 0.0;
    }
}

int fail(int code, const std::string& m) {
    lsb::set_last_error(m);  // reported by lsb_last_error()
    return code;
}

}  // namespace

extern "C" int lsb_solve_helmholtz_noalloc(int nx, int ny, int nz, const double* rhs, double* out, const double* lam,
                                           const double* e, const double* ei, const double* wavx,
                                           const double* wavy, double dtnui, void* stream) {
    if (!rhs || !out || !lam || !e || !ei || !wavx || !wavy) return fail(LSB_ERR_ARG, "null pointer argument");
    if (rhs == out) return fail(LSB_ERR_ARG, "rhs and out must not alias");
    if (nx < 2 || nx % 2 || ny < 1 || nz < 3) return fail(LSB_ERR_ARG, "bad grid size");
    const int nzp = nz + 1, nzm = nz - 1;
    if (nzp > kMaxNzp)
        return fail(LSB_ERR_UNSUPPORTED, "nz = " + std::to_string(nz) + " exceeds the no-allocation limit nzp <= " +
                                             std::to_string(kMaxNzp));
    const int kp = ((nzm + 15) / 16) * 16;
    int dev = 0;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce != cudaSuccess) return fail(LSB_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(ce));
    if (dev < 0 || dev >= 64) return fail(LSB_ERR_UNSUPPORTED, "device ordinal out of range");
    double* base = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_scratch_ptr[dev] == nullptr) {
            // once per device, with that device current: the device address of the array
            void* p = nullptr;
            ce = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (ce != cudaSuccess)
                return fail(LSB_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(ce));
            g_scratch_ptr[dev] = (double*)p;
        }
        base = g_scratch_ptr[dev];
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (s != nullptr) {
        // the scratch address above belongs to the current device: the stream must too
        int sdev = -1;
        ce = cudaStreamGetDevice(s, &sdev);
        if (ce != cudaSuccess) return fail(LSB_ERR_CUDA, std::string("cudaStreamGetDevice: ") + cudaGetErrorString(ce));
        if (sdev != dev)
            return fail(LSB_ERR_ARG, "the stream belongs to device " + std::to_string(sdev) + ", not the current device " +
                                         std::to_string(dev));
    }
    double* a1 = base;                           // padded E^-1
    double* a2 = base + (long long)kMaxP * kMaxP;  // padded E
    { lsb::note_launch(); k_pad_mats<<<64, 256, 0, s>>>(e, ei, nzm, kp, a1, a2); }
    // out[1..nz-1] = E (E^-1 rhs[1..nz-1] / (lam - k^2 - dtnui)); rows 0 and nz are exactly 0
    lsb::GemmArgs g1{};
    g1.A = a1;
    g1.M = g1.K = nzm;
    g1.Mp = g1.Kp = kp;
    g1.in = rhs;
    g1.koff = 1;
    g1.C = (long long)nx * ny;
    g1.nfields = 1;
    g1.epi = lsb::EPI_HELM_SCALE;
    g1.sigma = dtnui;
    g1.lam = lam;
    g1.wavx = wavx;
    g1.wavy = wavy;
    g1.nx = nx;
    lsb::GemmArgs g2 = g1;
    g2.A = a2;
    g2.in = nullptr;
    g2.koff = 0;
    g2.out = out;
    g2.roff = 1;
    g2.epi = lsb::EPI_LIFT_ADD;
    try {
        if (!lsb::launch_helm_fused(g1, g2, s)) return fail(LSB_ERR_CUDA, "the device refused the solve's shared memory");
    } catch (const std::exception& ex) {
        return fail(LSB_ERR_STATE, ex.what());
    }
    ce = cudaGetLastError();
    if (ce != cudaSuccess) return fail(LSB_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(ce));
    return LSB_OK;
}
