// noalloc.cu -- an allocation-free variant of the stand-alone CSR solve.
//
// fp_solve_csr_upper_noalloc solves the same system as fp_solve_csr_upper (an
// SPD matrix given by its upper-triangle CSR, Jacobi-preconditioned CG with
// FP64 vectors), with two differences: the matrix, right-hand side and
// solution are device buffers owned by the caller, and every work vector lives
// in g_csr_scratch, one file-scope device array of fixed size.  The call makes
// no cudaMalloc, no cudaFree and no call into an allocating library.
//
// It is meant for callers that must not allocate device memory while they
// run: a host application whose own pool allocator owns the GPU memory (a
// stray cudaMalloc there can fail once the pool has reserved the device, and
// it synchronises the whole device), and time-bounded loops that cannot afford
// the unbounded latency of cudaMalloc/cudaFree between steps.
//
// Rules that follow from the fixed scratch:
//   * it holds systems of at most FP_NOALLOC_MAX_N unknowns (6 double vectors
//     of that length, 12 MiB); larger systems are rejected with FP_ERR_ARG
//     before any GPU work;
//   * every call on a device uses the same array, so the calls on one device
//     take turns: each holds that device's host mutex from its first launch
//     until its stream has drained (the call is synchronous; on an error path
//     the stream is synchronised before the mutex is released), and calls
//     from several host threads, on any streams, are serialised in-process
//     (separate processes have separate contexts, each with its own array);
//   * the solve is one cooperative launch (k_csr_cg) of up to one block per SM
//     on the caller's stream.  It starts when all of its blocks fit on the GPU
//     together, so a resident kernel of the host that holds the SMs delays it
//     until that kernel ends, where a solve of separate kernels could run on
//     whatever SMs were free; a resident kernel that waits for the solution
//     would wait for good.  Hosts with such a kernel keep SMs free for it: a
//     system of n rows needs ceil(n / 512) blocks of 512 threads, at most one
//     per SM;
//   * each call clears the scratch it relies on before use: the control
//     block, the product vector, the first direction; x starts at zero;
//   * the first call on each device, with that device current, looks up the
//     array's device address with cudaGetSymbolAddress (the host-side symbol
//     is not a device address) and caches it; make that first call before any
//     stream capture begins on that device.
#include <cmath>
#include <cstdio>
#include <mutex>

#include "../../include/fluidprjct.h"
#include "kernels.hpp"

namespace {

constexpr int kMaxN = FP_NOALLOC_MAX_N;
constexpr int kMaxDevices = 64;
// Layout in doubles: the work vectors of launch_csr_cg (kMaxN each), its
// partial sums (kCsrPartials doubles), its control block.
constexpr size_t kScratchDoubles = size_t(fp::kCsrVectors) * kMaxN + fp::kCsrPartials +
                                   (sizeof(fp::CsrCtl) + sizeof(double) - 1) / sizeof(double);

static __device__ __align__(256) double g_csr_scratch[kScratchDoubles];

std::mutex g_setup_mutex;
double* g_scratch_ptr[kMaxDevices] = {nullptr};  // device address of g_csr_scratch, per device ordinal
std::mutex g_call_mutex[kMaxDevices];            // held by the one call that owns a device's scratch

int current_device(int* dev) {
    return cudaGetDevice(dev) == cudaSuccess && *dev >= 0 && *dev < kMaxDevices ? FP_OK : FP_ERR_CUDA;
}

int scratch_for_device(int dev, double** out) {
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_csr_scratch);
        if (e != cudaSuccess || !p) {
            std::fprintf(stderr, "fp_solve_csr_upper_noalloc: cudaGetSymbolAddress failed on device %d: %s\n", dev,
                         cudaGetErrorString(e));
            return FP_ERR_CUDA;
        }
        g_scratch_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_scratch_ptr[dev];
    return FP_OK;
}

// The solve proper (launch_csr_cg, with the checks that fp_solve_csr_upper
// makes on the host made on the device), run by one call at a time per device
// on scratch base.
int solve_on_scratch(double* base, int n, const int* d_offsets, const int* d_cols, const double* d_vals,
                     const double* d_b, double* d_x, double tol, int max_iters, int* iters, double* relres,
                     cudaStream_t st) {
    double* part = base + size_t(fp::kCsrVectors) * kMaxN;
    auto* ctl = reinterpret_cast<fp::CsrCtl*>(part + fp::kCsrPartials);
    if (fp::launch_csr_cg(n, d_offsets, d_cols, d_vals, d_b, d_x, base, kMaxN, part, ctl, 1, tol, max_iters, st))
        return FP_ERR_CUDA;
    fp::CsrCtl h{};
    if (cudaMemcpyAsync(&h, ctl, sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return FP_ERR_CUDA;
    if (h.status == fp::DEV_TIMEOUT) return FP_ERR_TIMEOUT;
    if (h.bad_off || h.bad_col) {
        std::fprintf(stderr, "fp_solve_csr_upper_noalloc: malformed CSR (offsets or column indices)\n");
        return FP_ERR_ARG;
    }
    if (iters) *iters = h.iters;
    if (relres) *relres = h.bb > 0.0 ? std::sqrt(h.rr / h.bb) : 0.0;
    return FP_OK;
}

}  // namespace

extern "C" int fp_solve_csr_upper_noalloc(int n, const int* d_offsets, const int* d_cols, const double* d_vals,
                                          const double* d_b, double* d_x, double tol, int max_iters, int* iters,
                                          double* relres, void* stream) {
    if (n <= 0 || !d_offsets || !d_cols || !d_vals || !d_b || !d_x) return FP_ERR_ARG;
    if (n > kMaxN) {
        std::fprintf(stderr, "fp_solve_csr_upper_noalloc: n = %d exceeds the scratch limit of %d unknowns\n", n,
                     kMaxN);
        return FP_ERR_ARG;
    }
    int dev = 0;
    double* base = nullptr;
    if (const int rc = current_device(&dev)) return rc;
    if (const int rc = scratch_for_device(dev, &base)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lock(g_call_mutex[dev]);
    // A launch error of this call is one that appears during it: an error the
    // calling thread left pending before the call is neither reported as this
    // call's failure nor cleared.
    const bool clean_before = cudaPeekAtLastError() == cudaSuccess;
    int rc = solve_on_scratch(base, n, d_offsets, d_cols, d_vals, d_b, d_x, tol, max_iters, iters, relres, st);
    // An early error return may leave launches queued on st: let them finish
    // before the next call takes the scratch.
    if (rc != FP_OK) cudaStreamSynchronize(st);
    if (clean_before && cudaPeekAtLastError() != cudaSuccess) {
        cudaGetLastError();  // this call's launch error: report it and clear it
        if (rc == FP_OK) rc = FP_ERR_CUDA;
    }
    return rc;
}
