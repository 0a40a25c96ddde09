// stk_p2p.cuh -- host-side interface of the sm_100a P2P kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace stk {

enum Precision : int { PREC_FP64 = 0, PREC_MIXED = 1 };

// One unit of P2P work: up to 64 targets of one target box against source-list
// entries [e0, e1).  A warp has 64 target slots (two per lane); glog =
// log2(slots per target) <= 5: the lanes that share a target split the source
// tile and are reduced with warp shuffles.
struct WorkItem {
    int trg_box;
    int t0;   // first target (leaf-sorted index)
    int nt;   // number of targets (1..64)
    int glog; // lanes per target = 1 << glog
    int e0;   // first list entry
    int e1;   // one past the last list entry
    // FP64 items (build_split_items): the range of the entries' sources, from source `skip` of
    // the first entry to source `stop` (exclusive) of the last, and where the sums of a
    // part go (target slot in ListP2PArgs::parts; -1: added to trg_out)
    int skip = 0, stop = 0x7fffffff;
    int part = -1;
};

// Targets whose sources were split over several items: n_parts runs of nt target slots from
// slot part0 on, added to trg_out in order.
struct PartGroup {
    int t0, nt, part0, n_parts;
};

// Device-resident description of one list evaluation.
struct ListP2PArgs {
    const double *src_rec;     // source records (launch_pack_records), uk_record_stride doubles each
    const int *src_box_begin;  // per source box: first record
    const int *src_box_end;    // per source box: one past the last record
    const int *list_ent;       // per entry: (source box << 5) | periodic shift code (0..26, 13 = none)
    const WorkItem *items;     // cost-sorted work items
    int n_items;
    unsigned int *counter;     // work counter, zero at launch
    const double *trg_xyz;     // targets, 3 doubles each
    double *trg_out;           // outputs, TDIM doubles each, accumulated
    const double *box_centre;  // per target box: local origin for the mixed path (3 doubles)
    double period;             // periodic image length (1 for the unit box)
    int atomic_out;            // direct sums only: 0 trg_out or parts =, 1 +=, 2 += by atomics (lists: 0, +=)
    const double *trg_aux;     // per-target values (TV doubles each) of the adjoint kernels, else null
    int coincident_own_box;    // 1: a source can sit at a target's position only in an unshifted
                               // entry of the target's own box (lists of one octree over both
                               // point sets); the mixed path then skips the coincidence mask
                               // elsewhere.  0: every pair is masked.
    const PartGroup *groups;   // targets with split sources, their sums in `parts`
    int n_groups;
    // direct sums only (launch_direct_p2p): all sources against all targets
    const double *src_xyz, *src_val;  // 3 and SDIM doubles per source
    int nsrc, ntrg;
    int src_chunk, n_chunk;  // source points per chunk (a multiple of 32), chunks
    double *parts;           // outputs of each chunk, ntrg x TDIM each (null: one chunk)
};

// Record stride (doubles) for a micro-kernel: 3 coordinates + its staged values (or the
// source's SDIM, where those are fewer), rounded up to a 16-byte multiple; never above that of SDIM.
int uk_record_stride(int uk);
int uk_sdim_host(int uk);
int uk_tdim_host(int uk);
int uk_tvdim_host(int uk);  // per-target values read by a micro-kernel (adjoint kernels)
double uk_scale_host(int uk);

// Launch the list kernel for micro-kernel `uk` with the given precision.
cudaError_t launch_list_p2p(int uk, int prec, const ListP2PArgs &a, int num_sms, cudaStream_t stream);

// Direct sum of all sources at all targets: items of 64 targets x one chunk of sources, which
// the kernel derives from its block index; raw source arrays, nothing to set up.  With several
// chunks each writes its own sums and a second kernel adds them up in order (repeats give the
// same bits).  direct_chunks: sources per chunk (a multiple of 32) and the number of chunks.
// direct_in_place: `out` overlaps the sources, which are read while targets are written; the sums go
// through parts then, or the sources are copied.
bool direct_in_place(int uk, const ListP2PArgs &a, const double *out);
void direct_chunks(int uk, int prec, int ntrg, int nsrc, int num_sms, int &chunk, int &n_chunk);
// a: src_xyz, src_val, nsrc, ntrg, src_chunk, n_chunk, parts (n_chunk > 1, or in place), counter
// (mixed), trg_xyz, trg_aux and trg_out; add = 0: trg_out = sum, 1: +=, 2: += by atomics, without parts
cudaError_t launch_direct_p2p(int uk, int prec, const ListP2PArgs &a, int add, int num_sms, cudaStream_t stream);

// Source records of micro-kernel uk: rec[i] = (xyz[i], values, 0 padding), values = those of v1[perm[i]]
// (d1) and v2[perm[i]] (the rest of SDIM), staged where that makes no larger record; perm may be
// null (identity), v2 null.
cudaError_t launch_pack_records(int uk, int n, const int *perm, const double *xyz, const double *v1, int d1,
                                const double *v2, double *rec, cudaStream_t stream);

// Records of KIFMM surfaces: for each listed node b, rec[b n + i] = (xyz[b n + i], stage(densities
// of its point i, component c times 2^(-level[b] den_exp[c]))), i < n; level null: no factor.
cudaError_t launch_pack_surface(int uk, const int *nodes, int m, int n, const double *xyz, const double *dens,
                                const int *level, const double *den_exp, double *rec, cudaStream_t stream);

// out[perm[i] * d + k] += alpha_k * in[i * d + k]   (alpha per component; perm may be null)
cudaError_t launch_scatter_add(int n, int d, const int *perm, const double *in, const double *alpha,
                               double *out, cudaStream_t stream);

}  // namespace stk
