// stk_plan.cu -- a reusable, asynchronous list P2P plan (C ABI stk_p2p_plan_*).
//
// stk_p2p_lists validates a CSR interaction list, builds its cost-sorted work
// items on the host, uploads them and waits for the result on every call.  A
// caller that evaluates the same list many times (PVFMM's list loops call
// ker_poten for the same U/W/X lists at every evaluation; an autograd forward
// and its two adjoint passes share one U list) builds a plan once instead:
// stk_p2p_plan_create validates the list, builds the items and uploads the list
// and the items into device memory owned by the plan; stk_p2p_plan_execute then
// queues the pack and list kernels on the caller's stream and returns without a
// host wait.
#include <algorithm>
#include <new>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/stkfmm_b200.h"
#include "stk_p2p.cuh"
#include "stk_tree.hpp"
#include "stk_ukernels.cuh"
#include "stk_work.hpp"

struct stk_p2p_plan {
    int device = -1;
    int num_sms = 1;
    int nsrc = 0, ntrg = 0;
    int n_src_box = 0;
    double period = 1.0;
    long long pairs = 0;
    int n_items[2] = {0, 0};  // FP64 (split), mixed
    int n_groups = 0;
    long long part_targets = 0;
    int *d_sbeg = nullptr, *d_send = nullptr, *d_ent = nullptr;
    stk::WorkItem *d_items[2] = {nullptr, nullptr};
    stk::PartGroup *d_groups = nullptr;
    double *d_parts[2] = {nullptr, nullptr};  // sums of split sources, 8 and 16 doubles per slot
    unsigned int *d_counter = nullptr;
    double *d_rec = nullptr;  // packed source records, grown to the largest record stride used (at least 8)
    size_t rec_cap = 0;       // doubles
    size_t parts_bytes(int wide) const { return (size_t)part_targets * (wide ? 16 : 8) * sizeof(double); }
    ~stk_p2p_plan() {
        cudaFree(d_sbeg);
        cudaFree(d_send);
        cudaFree(d_ent);
        cudaFree(d_items[0]);
        cudaFree(d_items[1]);
        cudaFree(d_groups);
        cudaFree(d_parts[0]);
        cudaFree(d_parts[1]);
        cudaFree(d_counter);
        cudaFree(d_rec);
    }
};

namespace {

int validate_lists(int n_trg_box, const int *trg_begin, const int *trg_end, const int *list_off,
                   const int *list_ent, int n_src_box, const int *src_begin, const int *src_end, int nsrc,
                   int ntrg) {
    if (n_trg_box < 0 || n_src_box < 0 || nsrc < 0 || ntrg < 0) return STK_ERR_INVALID_ARG;
    if (n_trg_box > 0 && (!trg_begin || !trg_end || !list_off)) return STK_ERR_INVALID_ARG;
    if (n_trg_box > 0 && list_off[0] != 0) return STK_ERR_INVALID_ARG;
    if (n_src_box > 0 && (!src_begin || !src_end)) return STK_ERR_INVALID_ARG;
    for (int b = 0; b < n_trg_box; b++) {
        if (trg_begin[b] < 0 || trg_end[b] < trg_begin[b] || trg_end[b] > ntrg) return STK_ERR_INVALID_ARG;
        if (list_off[b + 1] < list_off[b]) return STK_ERR_INVALID_ARG;
    }
    for (int s = 0; s < n_src_box; s++)
        if (src_begin[s] < 0 || src_end[s] < src_begin[s] || src_end[s] > nsrc) return STK_ERR_INVALID_ARG;
    const int nent = n_trg_box > 0 ? list_off[n_trg_box] : 0;
    if (nent > 0 && !list_ent) return STK_ERR_INVALID_ARG;
    for (int e = 0; e < nent; e++) {
        const int sb = list_ent[e] >> 5, code = list_ent[e] & 31;
        if (list_ent[e] < 0 || sb >= n_src_box || code > 26) return STK_ERR_INVALID_ARG;
    }
    return STK_OK;
}

template <class T> cudaError_t upload(T **dst, const T *src, size_t n) {
    if (n == 0) return cudaSuccess;
    cudaError_t e = cudaMalloc(dst, n * sizeof(T));
    if (e != cudaSuccess) return e;
    return cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice);
}

}  // namespace

extern "C" stk_p2p_plan *stk_p2p_plan_create(int n_trg_box, const int *trg_begin, const int *trg_end,
                                             const int *list_off, const int *list_ent, int n_src_box,
                                             const int *src_begin, const int *src_end, int nsrc, int ntrg,
                                             double period, int *status) {
    int dummy = 0;
    int &st = status ? *status : dummy;
    st = validate_lists(n_trg_box, trg_begin, trg_end, list_off, list_ent, n_src_box, src_begin, src_end, nsrc, ntrg);
    if (st) return nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        st = STK_ERR_NO_DEVICE;
        return nullptr;
    }
    auto *p = new (std::nothrow) stk_p2p_plan();
    if (!p) {
        st = STK_ERR_CUDA;
        return nullptr;
    }
    p->nsrc = nsrc;
    p->ntrg = ntrg;
    p->n_src_box = n_src_box;
    p->period = period;
    const int nent = n_trg_box > 0 ? list_off[n_trg_box] : 0;
    bool ok = cudaGetDevice(&p->device) == cudaSuccess &&
              cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, p->device) == cudaSuccess;
    // The two item lists on host threads of their own, and meanwhile, on this one, the device's
    // arrays and the records of most executions (eight doubles a source).  One after the other the
    // lists alone took 2.6 ms for 262k points, and buffers that the first execution allocated made it
    // wait: creation and first FP64 pass 4.3 ms, 2.8 before there were two lists.  (Small lists: here.)
    std::vector<stk::WorkItem> items[2];
    std::vector<stk::PartGroup> groups;
    const size_t records = (size_t)std::max(nsrc, 1) * 8;
    bool host_ok = true;
    try {
        stk::parallel_ranges(ok ? 3 : 0, nent > 16384 ? 1 : 3, [&](size_t i0, size_t i1) {
            for (size_t i = i0; i < i1; i++) {
                if (i == 0) {
                    ok = cudaMalloc(&p->d_counter, 64) == cudaSuccess && upload(&p->d_sbeg, src_begin, n_src_box) == cudaSuccess &&
                         upload(&p->d_send, src_end, n_src_box) == cudaSuccess && upload(&p->d_ent, list_ent, nent) == cudaSuccess;
                    if (ok && nent > 0 && cudaMalloc(&p->d_rec, records * sizeof(double)) == cudaSuccess) p->rec_cap = records;
                } else if (n_trg_box > 0 && i == 1) {
                    stk::build_list_items(n_trg_box, trg_begin, trg_end, list_off, list_ent, src_begin, src_end, items[1],
                                          p->pairs);
                } else if (n_trg_box > 0) {
                    stk::build_split_items(n_trg_box, trg_begin, trg_end, list_off, list_ent, src_begin, src_end,
                                           p->num_sms * 15, items[0], groups, p->part_targets);
                }
            }
        });
    } catch (...) {  // host memory
        host_ok = false;
    }
    ok = ok && host_ok;
    p->n_items[0] = (int)items[0].size();
    p->n_items[1] = (int)items[1].size();
    p->n_groups = (int)groups.size();
    ok = ok && upload(&p->d_items[0], items[0].data(), items[0].size()) == cudaSuccess &&
         upload(&p->d_items[1], items[1].data(), items[1].size()) == cudaSuccess &&
         upload(&p->d_groups, groups.data(), groups.size()) == cudaSuccess;
    // the slots of FP64 sums of up to eight components (an execution without them tries again)
    if (ok && p->n_groups > 0 && cudaMalloc(&p->d_parts[0], p->parts_bytes(0)) != cudaSuccess) p->d_parts[0] = nullptr;
    cudaGetLastError();
    if (!ok) {
        cudaGetLastError();
        delete p;
        st = STK_ERR_CUDA;
        return nullptr;
    }
    return p;
}

extern "C" void stk_p2p_plan_destroy(stk_p2p_plan *plan) {
    if (!plan) return;
    int cur = -1;
    cudaGetDevice(&cur);
    const int dev = plan->device;
    if (dev >= 0 && dev != cur) cudaSetDevice(dev);
    cudaDeviceSynchronize();  // work queued on any stream may still read the plan's buffers
    delete plan;
    if (cur >= 0 && dev >= 0 && dev != cur) cudaSetDevice(cur);
}

extern "C" long long stk_p2p_plan_pairs(const stk_p2p_plan *plan) { return plan ? plan->pairs : -1; }

extern "C" int stk_p2p_plan_execute(stk_p2p_plan *plan, int ukernel, int precision, const double *d_src_coord,
                                    const double *d_src_value, const double *d_trg_coord, const double *d_trg_aux,
                                    double *d_trg_value, void *stream) {
    if (!plan || ukernel < 0 || ukernel >= stk::UK_COUNT) return STK_ERR_INVALID_ARG;
    if (precision != stk::PREC_FP64 && precision != stk::PREC_MIXED) return STK_ERR_INVALID_ARG;
    if ((stk::uk_tvdim_host(ukernel) > 0) != (d_trg_aux != nullptr)) return STK_ERR_INVALID_ARG;
    const bool mixed = precision == stk::PREC_MIXED;
    if (plan->n_items[mixed] == 0) return STK_OK;
    if ((plan->nsrc > 0 && (!d_src_coord || !d_src_value)) || !d_trg_coord || !d_trg_value) return STK_ERR_INVALID_ARG;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != plan->device) return STK_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const int sd = stk::uk_sdim_host(ukernel), rs = stk::uk_record_stride(ukernel);
    // records: the plan's own hold eight doubles each (a forward pass and its adjoints: 3 to 5 values)
    const size_t n = std::max(plan->nsrc, 1), need = n * rs;
    if (plan->rec_cap < need) {
        // grow the record buffer: earlier executions may still read it on any stream
        if (plan->d_rec) {
            cudaDeviceSynchronize();
            cudaFree(plan->d_rec);
            plan->d_rec = nullptr;
            plan->rec_cap = 0;
        }
        size_t cap = n * std::max(rs, 8);
        if (cudaMalloc(&plan->d_rec, cap * sizeof(double)) != cudaSuccess) {
            cudaGetLastError();
            cap = need;
            if (cudaMalloc(&plan->d_rec, cap * sizeof(double)) != cudaSuccess) {
                cudaGetLastError();
                return STK_ERR_CUDA;
            }
        }
        plan->rec_cap = cap;
    }
    // The split sums' slots: one buffer for up to eight components and one beyond, each allocated
    // once and kept, so that a captured execution keeps its buffer; during a capture, too (relaxed:
    // an allocation is no part of the stream's work).  Without memory for them the mixed path's
    // items are taken, which split no sources.
    const int td = stk::uk_tdim_host(ukernel);
    double **parts = &plan->d_parts[td > 8];
    int list = mixed;
    if (!mixed && plan->n_groups > 0 && !*parts) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (cudaMalloc(parts, plan->parts_bytes(td > 8)) != cudaSuccess) {
            cudaGetLastError();
            *parts = nullptr;
            list = 1;
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    if (stk::launch_pack_records(ukernel, plan->nsrc, nullptr, d_src_coord, d_src_value, sd, nullptr, plan->d_rec, s) !=
        cudaSuccess)
        return STK_ERR_CUDA;
    stk::ListP2PArgs a{};
    a.src_rec = plan->d_rec;
    a.src_box_begin = plan->d_sbeg;
    a.src_box_end = plan->d_send;
    a.list_ent = plan->d_ent;
    a.items = plan->d_items[list];
    a.n_items = plan->n_items[list];
    if (list == 0) {
        a.groups = plan->d_groups;
        a.n_groups = plan->n_groups;
        a.parts = *parts;
    }
    a.counter = plan->d_counter;
    a.trg_xyz = d_trg_coord;
    a.trg_out = d_trg_value;
    a.box_centre = nullptr;
    a.period = plan->period;
    a.atomic_out = 0;
    a.trg_aux = d_trg_aux;
    if (stk::launch_list_p2p(ukernel, precision, a, plan->num_sms, s) != cudaSuccess) return STK_ERR_CUDA;
    return STK_OK;
}
