// Block-tridiagonal FP64 solve that allocates no memory.
//
// For callers that cannot call cudaMalloc: code running where a host-side
// allocation is not allowed or not wanted -- inside a framework that owns all
// device memory through its own pool, or a plugin handed pre-allocated
// buffers by its host -- and that still need the solver's scratch space.  The
// scratch (block inverses and the forward-sweep vector) lives in one
// file-scope __device__ array of fixed size, so nothing is allocated at call
// time; every GPU that loads the library holds that array until the process
// exits.  Each call waits for its stream to finish (it reads the status word
// back to report a singular or non-finite block).
//
// Solves, for one column of nz layers with ni species,
//     lower[j] o x[j-1] + D[j] x[j] + upper[j] o x[j+1] = b[j]
// (D dense ni x ni, lower/upper diagonal vectors) with the FP64 solver's
// two-sided block-Thomas (vk_lu64.cu): a cluster of eight CTAs per half of the
// column.  A column of 150 layers of 69 species: 28.1 -> 3.7 ms (one CTA from
// one end before).  Where the two-sided order meets a block without a finite
// non-zero pivot, or a Schur term from the top that would cost the block its
// digits (k_solve64_growth), the column is solved from its bottom alone, whose answer or
// failure is the call's (10.8 ms for such a column).
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>
#include <string>

#include "vk_internal.cuh"

// Scratch capacity in doubles: nz*ni*ni (inverses) + nz*ni (sweep vector) + 1
// must fit.  2^21 doubles = 16 MiB, e.g. nz = 200 at ni = 100.
#define VK_NOALLOC_MAX_DOUBLES (1u << 21)

static __device__ __align__(256) double g_noalloc_scratch[VK_NOALLOC_MAX_DOUBLES];
static __device__ int g_noalloc_words[vk::kSolve64Words];      // the column, its status, the queues

namespace {

std::mutex g_setup_mu;
constexpr int kMaxDevices = 64;
struct Scratch { double *p; int *words; };
Scratch g_scratch_dev[kMaxDevices] = {};   // device addresses of the arrays, per device
int noalloc_fail(int code, const std::string &msg) {
    vk::set_global_error(msg);        // read back with vk_last_error(NULL)
    return code;
}

// Once per device, with that device current: resolve the arrays' device
// addresses (host code must not use the symbols themselves) and opt the
// kernels into the shared memory that blocks of 160 species need.
int noalloc_setup(int dev, Scratch *out) {
    std::lock_guard<std::mutex> lock(g_setup_mu);
    if (!g_scratch_dev[dev].p) {
        Scratch t = {};
        cudaError_t e = cudaGetSymbolAddress((void **)&t.p, g_noalloc_scratch);
        if (e == cudaSuccess) e = cudaGetSymbolAddress((void **)&t.words, g_noalloc_words);
        if (e != cudaSuccess || !t.p || !t.words)
            return noalloc_fail(VK_ECUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        e = vk::init_solve64(VK_MAX_NI);
        if (e != cudaSuccess)
            return noalloc_fail(VK_ECUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
        g_scratch_dev[dev] = t;
    }
    *out = g_scratch_dev[dev];
    return VK_OK;
}

}  // namespace

extern "C" int vk_block_solve_noalloc(int nz, int ni, const double *D, const double *lower,
                                      const double *upper, const double *b, double *x,
                                      void *stream) {
    if (nz < 1 || ni < 1 || ni > VK_MAX_NI)
        return noalloc_fail(VK_EINVAL, "need nz >= 1 and 1 <= ni <= " + std::to_string(VK_MAX_NI));
    const unsigned long long need =
        (unsigned long long)nz * ni * ni + (unsigned long long)nz * ni + 1ull;
    if (need > VK_NOALLOC_MAX_DOUBLES)
        return noalloc_fail(VK_EINVAL, "nz*ni*ni + nz*ni + 1 = " + std::to_string(need) +
                                           " doubles exceeds the fixed scratch of " +
                                           std::to_string(VK_NOALLOC_MAX_DOUBLES) + " doubles (16 MiB)");
    if (!D || !lower || !upper || !b || !x) return noalloc_fail(VK_EINVAL, "NULL array");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return noalloc_fail(VK_ECUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(VK_EINVAL, "device ordinal out of range");
    Scratch sc = {};
    int rc = noalloc_setup(dev, &sc);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    // an error left pending by earlier, unrelated work is reported as such
    // (and cleared) rather than blamed on this launch
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return noalloc_fail(VK_ECUDA, std::string("CUDA error pending from earlier work (nothing launched): ") +
                                          cudaGetErrorString(e));
    int status = 0;
    // from both ends (of two layers the upper is the middle); from the bottom alone, as
    // small systems are, in one launch
    for (int mid = nz < 3 || vk::solve64_small(nz, ni) ? nz - 1 : -1;; mid = nz - 1) {
        e = vk::launch_solve64(nz, ni, D, lower, upper, b, x, sc.p, sc.p + (size_t)nz * ni * ni, sc.words, mid, s);
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e != cudaSuccess) return noalloc_fail(VK_ECUDA, std::string("launch: ") + cudaGetErrorString(e));
        e = cudaMemcpyAsync(&status, sc.words + 3, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return noalloc_fail(VK_ECUDA, std::string("status read: ") + cudaGetErrorString(e));
        if (status == VK_OK || status == VK_ETIMEOUT || mid >= 0) break;
    }
    if (status == VK_ESINGULAR) return noalloc_fail(VK_ESINGULAR, "singular diagonal block");
    if (status == VK_ENAN) return noalloc_fail(VK_ENAN, "non-finite pivot (NaN input)");
    if (status != VK_OK) return noalloc_fail(status, "a message between CTAs never came");
    return VK_OK;
}
