// stk_noalloc.cu -- a direct-sum entry point that allocates no device memory.
//
// Who needs it: callers that must not call cudaMalloc / cudaFree during their
// run.  cudaMalloc and cudaFree synchronise the whole device, which stalls a
// caller that keeps several streams busy; some frameworks hand the whole device
// to their own caching allocator, so memory taken behind its back can make it
// fail; and some real-time or embedded hosts forbid run-time allocation
// outright.  stk_ukernel_direct_device keeps a per-thread workspace that grows
// with cudaMalloc; this variant instead works inside one fixed scratch array
// that the library reserves when it is loaded.
//
// Mechanics: the scratch is the file-scope array g_stk_noalloc_scratch below.
// Its host-side name is only a stand-in, so the device address is fetched with
// cudaGetSymbolAddress, once per device, the first time the entry point runs on
// that device (with that device current), and cached.  That first call therefore
// does set-up work and should come before any stream capture; so should the
// first call of each (micro-kernel, precision) pair, whose list-kernel instance
// runs a one-time occupancy query (and, with lazy module loading, its module
// load).  The cached address belongs to the device's primary context: after a
// cudaDeviceReset of that device the entry point must not be used again in the
// process.  Every call shares the array and leaves its contents behind: two calls
// whose work overlaps on the GPU (different streams, or host threads, at the
// same time) race on the array.
#include <mutex>

#include <cuda_runtime.h>

#include "../../include/stkfmm_b200.h"
#include "stk_p2p.cuh"
#include "stk_tree.hpp"

namespace {

// Fixed scratch capacity: 8 MiB, held by every GPU that loads the library.
constexpr size_t kNoAllocScratchBytes = size_t(8) << 20;
constexpr int kNoAllocMaxDevices = 64;
constexpr int kItemTargets = 64;

static __device__ __align__(256) unsigned char g_stk_noalloc_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mu;
void *g_noalloc_addr[kNoAllocMaxDevices] = {};

inline size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Device address of the scratch array for the current device.
int noalloc_scratch(void **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return STK_ERR_NO_DEVICE;
    }
    if (dev < 0 || dev >= kNoAllocMaxDevices) return STK_ERR_NOT_SUPPORTED;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_stk_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return STK_ERR_CUDA;
        }
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return STK_OK;
}

}  // namespace

extern "C" int stk_ukernel_direct_device_noalloc(int ukernel, int nsrc, const double *d_src_coord,
                                                 const double *d_src_value, int ntrg, const double *d_trg_coord,
                                                 double *d_trg_value, int precision, void *stream) {
    // every micro-kernel the allocating direct sum takes without per-target values
    // (the adjoint kernels, which need them, go through stk_ukernel_direct_aux_device)
    int sdim = 0, tdim = 0;
    if (stk_ukernel_dims(ukernel, &sdim, &tdim) != STK_OK || stk::uk_tvdim_host(ukernel) > 0 || nsrc < 0 || ntrg < 0)
        return STK_ERR_INVALID_ARG;
    if (precision != STK_FP64 && precision != STK_MIXED) return STK_ERR_INVALID_ARG;
    if (nsrc == 0 || ntrg == 0) return STK_OK;
    if (!d_src_coord || !d_src_value || !d_trg_coord || !d_trg_value) return STK_ERR_INVALID_ARG;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return STK_ERR_NO_DEVICE;
    }
    // The sizes this entry takes are its interface's, not what is needed below: 24 bytes per 64
    // targets x chunk of sources (>= 256 points), 12 per chunk, and a record per source.
    const long long nchunk = (ntrg + kItemTargets - 1) / kItemTargets;
    const long long want_items = (long long)(sms > 0 ? sms : 1) * 64;
    long long nsc = (want_items + nchunk - 1) / nchunk;
    if (nsc < 1) nsc = 1;
    if (nsc > (nsrc / 256 > 1 ? nsrc / 256 : 1)) nsc = nsrc / 256 > 1 ? nsrc / 256 : 1;
    long long sc = (nsrc + nsc - 1) / nsc;
    sc = (sc + 31) / 32 * 32;
    nsc = (nsrc + sc - 1) / sc;
    const size_t off_sbeg = round_up(256 + (size_t)(nchunk * nsc) * 24, 256);
    const size_t off_send = round_up(off_sbeg + (size_t)nsc * sizeof(int), 256);
    const size_t off_ent = round_up(off_send + (size_t)nsc * sizeof(int), 256);
    const size_t off_rec = round_up(off_ent + (size_t)nsc * sizeof(int), 256);
    const size_t need = off_rec + (size_t)nsrc * ((3 + sdim + 1) & ~1) * sizeof(double);
    if (need > kNoAllocScratchBytes) return STK_ERR_SIZE;  // beyond the fixed 8 MiB scratch

    void *base = nullptr;
    int rc = noalloc_scratch(&base);
    if (rc) return rc;
    // the direct form of the list kernel reads the caller's arrays; the chunks' sums are kept in
    // the scratch and added in order, or by atomics where they do not fit
    stk::ListP2PArgs a{};
    a.src_xyz = d_src_coord;
    a.src_val = d_src_value;
    a.nsrc = nsrc;
    a.ntrg = ntrg;
    stk::direct_chunks(ukernel, precision, ntrg, nsrc, sms, a.src_chunk, a.n_chunk);
    a.trg_xyz = d_trg_coord;
    a.trg_out = d_trg_value;
    // the work counter of mixed items: the array's end (the limit above leaves room for it)
    constexpr size_t room = kNoAllocScratchBytes - 256;
    a.counter = reinterpret_cast<unsigned int *>(static_cast<unsigned char *>(base) + room);
    const bool fits = (size_t)a.n_chunk * ntrg * tdim * sizeof(double) <= room;
    const bool in_place = stk::direct_in_place(ukernel, a, d_trg_value);
    if (fits && (a.n_chunk > 1 || in_place)) {
        a.parts = static_cast<double *>(base);
    } else if (in_place) {  // a copy of the sources, which fits by the limit above
        double *x = static_cast<double *>(base), *v = x + 3 * (size_t)nsrc;
        if (cudaMemcpyAsync(x, d_src_coord, sizeof(double) * 3 * nsrc, cudaMemcpyDefault, (cudaStream_t)stream) != cudaSuccess ||
            cudaMemcpyAsync(v, d_src_value, sizeof(double) * sdim * nsrc, cudaMemcpyDefault, (cudaStream_t)stream) != cudaSuccess)
            return STK_ERR_CUDA;
        a.src_xyz = x;
        a.src_val = v;
    }
    if (stk::launch_direct_p2p(ukernel, precision, a, fits ? 1 : 2, sms, (cudaStream_t)stream) != cudaSuccess)
        return STK_ERR_CUDA;
    return STK_OK;
}
