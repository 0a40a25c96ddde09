// stk_work.cpp -- per-thread device workspace and work-list builders.
#include "stk_work.hpp"

#include <algorithm>
#include <cmath>
#include <mutex>
#include <numeric>

#include "../../include/stkfmm_b200.h"
#include "stk_tree.hpp"

namespace stk {

namespace {

// Workspaces outlive the threads that used them: when a thread ends (for
// example torch's autograd worker at interpreter shutdown) its workspace goes
// back to this free list, with no CUDA call, and the next new thread reuses it.
// Calling cudaFree from a thread-exit destructor can run after the CUDA runtime
// has been torn down.  The pool itself is never destroyed; its device memory
// is released with the CUDA context when the process ends.
class WorkspacePool {
  public:
    Workspace *acquire() {
        std::lock_guard<std::mutex> lock(mu_);
        if (!free_.empty()) {
            Workspace *w = free_.back();
            free_.pop_back();
            return w;
        }
        return new Workspace();
    }
    void release(Workspace *w) {
        std::lock_guard<std::mutex> lock(mu_);
        free_.push_back(w);
    }

  private:
    std::mutex mu_;
    std::vector<Workspace *> free_;
};

WorkspacePool &pool() {
    static WorkspacePool *p = new WorkspacePool();
    return *p;
}

struct WorkspaceHolder {
    Workspace *ws = pool().acquire();
    ~WorkspaceHolder() { pool().release(ws); }
};

}  // namespace

Workspace &Workspace::thread_local_ws() {
    static thread_local WorkspaceHolder holder;
    return *holder.ws;
}

Workspace::~Workspace() = default;

int Workspace::ensure_device() {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        cudaGetLastError();
        return STK_ERR_NO_DEVICE;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return STK_ERR_CUDA;
    Dev &d = devs_[dev];
    cur_ = &d;
    if (!d.stream) {
        if (cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking) != cudaSuccess) return STK_ERR_CUDA;
        if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return STK_ERR_CUDA;
        if (cudaMalloc(&d.counter, 64) != cudaSuccess) return STK_ERR_CUDA;
        if (cudaEventCreateWithFlags(&d.done, cudaEventDisableTiming) != cudaSuccess) return STK_ERR_CUDA;
    }
    return STK_OK;
}

int Workspace::begin(cudaStream_t s) {
    if (!cur_) return STK_ERR_CUDA;
    if (cur_->recorded && cudaStreamWaitEvent(s, cur_->done, 0) != cudaSuccess) return STK_ERR_CUDA;
    return STK_OK;
}

int Workspace::end(cudaStream_t s) {
    if (!cur_) return STK_ERR_CUDA;
    if (cudaEventRecord(cur_->done, s) != cudaSuccess) return STK_ERR_CUDA;
    cur_->recorded = true;
    return STK_OK;
}

void *Workspace::raw(int slot, size_t bytes) {
    if (!cur_ || slot < 0 || slot >= kNumSlots) return nullptr;
    if (bytes == 0) bytes = 16;
    if (cur_->cap[slot] < bytes) {
        const size_t want = std::max(bytes, cur_->cap[slot] * 3 / 2);
        if (cur_->ptr[slot]) {
            // the previous contents may still be read by work queued on any stream
            cudaDeviceSynchronize();
            cudaFree(cur_->ptr[slot]);
        }
        cur_->ptr[slot] = nullptr;
        cur_->cap[slot] = 0;
        if (cudaMalloc(&cur_->ptr[slot], want) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        cur_->cap[slot] = want;
    }
    return cur_->ptr[slot];
}

void *Workspace::pinned(size_t bytes) {
    if (bytes > kPinnedBytes) return nullptr;
    if (pin_cap_ < bytes) {
        size_t want = 64u << 10;
        while (want < bytes) want *= 2;
        if (pin_) cudaFreeHost(pin_);  // its last call has waited for its copies
        pin_ = nullptr;
        pin_cap_ = 0;
        if (cudaHostAlloc(&pin_, want, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            pin_ = nullptr;
            return nullptr;
        }
        pin_cap_ = want;
    }
    return pin_;
}

unsigned int *Workspace::counter() { return cur_ ? cur_->counter : nullptr; }
int Workspace::num_sms() { return cur_ ? cur_->sms : 1; }
cudaStream_t Workspace::stream() { return cur_ ? cur_->stream : nullptr; }

// A warp has 64 target slots (two per lane); items hold at most kItemTargets targets.
constexpr int kItemTargets = 64;

static inline int lanes_log2(int m) {
    // largest g = 2^glog <= 32 with m * g <= 64 slots
    int glog = 0;
    while (glog < 5 && (m << (glog + 1)) <= kItemTargets) glog++;
    return glog;
}

// Indices by falling cost, equal ones in their order (radix: comparing 12k items of 262k points
// took 0.8 ms of a plan's creation).
static void longest_first(const std::vector<long long> &cost, std::vector<int> &idx) {
    long long top = 0;
    for (long long c : cost) top = std::max(top, c);
    int shift = 0;
    while (shift < 59 && (top >> (59 - shift)) == 0) shift++;  // the largest key fills 60 bits
    std::vector<uint64_t> key(cost.size());
    for (size_t i = 0; i < cost.size(); i++) key[i] = (uint64_t)(top - cost[i]) << shift;
    sort_keys(key, idx);
}

void build_list_items(int n_trg_box, const int *trg_begin, const int *trg_end, const int *list_off,
                      const int *list_ent, const int *src_begin, const int *src_end, std::vector<WorkItem> &items,
                      long long &pairs, int balance_warps, int shard_rank, int shard_n) {
    items.clear();
    pairs = 0;
    std::vector<long long> box_ns(n_trg_box, 0);
    for (int b = 0; b < n_trg_box; b++) {
        const int nt = trg_end[b] - trg_begin[b];
        if (nt <= 0) continue;
        long long ns = 0;
        for (int e = list_off[b]; e < list_off[b + 1]; e++) {
            const int sb = list_ent[e] >> 5;
            ns += src_end[sb] - src_begin[sb];
        }
        box_ns[b] = ns;
        pairs += (long long)nt * ns;
    }
    // Load balance: no item above ~half of one warp's share of the pairs, so a
    // box with very many sources (a long W list) is not a single long item that
    // finishes after every other warp.  Items keep at least 8 targets (64 slots
    // filled with 8 lanes per target).
    const long long cap = balance_warps > 0 ? std::max(pairs / (2LL * balance_warps), 1LL) : 0;
    std::vector<long long> cost;  // in 32nds
    for (int b = 0; b < n_trg_box; b++) {
        const int nt = trg_end[b] - trg_begin[b];
        const long long ns = box_ns[b];
        if (nt <= 0 || ns == 0) continue;
        int mmax = kItemTargets;
        while (cap > 0 && mmax > 8 && (long long)mmax * ns > cap) mmax /= 2;
        // Split the box into full mmax-target items, then power-of-two chunks of
        // the remainder (32, 16, 8 targets; the last < 8 targets together): a
        // chunk of m = 2^k targets fills all 64 slots with 64/m lanes per target,
        // so the box costs ~nt/64 warp passes over its sources instead of
        // ceil(nt/64).  Chunks below 8 targets would mostly re-stage sources.
        int t0 = trg_begin[b];
        int left = nt;
        while (left > 0) {
            int m = mmax;
            if (left < mmax) {
                m = 1;
                while (m * 2 <= left) m *= 2;
                if (m < 8) m = left;
            }
            const int glog = lanes_log2(m);
            items.push_back({b, t0, m, glog, list_off[b], list_off[b + 1]});
            cost.push_back(ns * (32 >> glog) + 2048LL * (list_off[b + 1] - list_off[b]));
            t0 += m;
            left -= m;
        }
    }
    std::vector<int> idx;
    longest_first(cost, idx);
    std::vector<WorkItem> sorted;
    sorted.reserve(items.size());
    if (shard_n > 1) {
        // this shard's items: the cost-sorted items dealt to the least-loaded
        // shard in turn (the same deterministic assignment on every shard)
        std::vector<int> owner;
        std::vector<double> sc;
        for (int i : idx) sc.push_back(cost[i] / 32.0);
        partition_lpt((int)sc.size(), sc.data(), shard_n, owner);
        pairs = 0;
        for (size_t i = 0; i < idx.size(); i++)
            if (owner[i] == shard_rank) {
                const WorkItem &w = items[idx[i]];
                sorted.push_back(w);
                pairs += (long long)w.nt * pair_sources(w, list_ent, src_begin, src_end);
            }
    } else {
        for (size_t i = 0; i < idx.size(); i++) sorted.push_back(items[idx[i]]);
    }
    items.swap(sorted);
}

// Targets of the next chunk of `left` remaining ones.  A chunk of m targets with g = 2^glog
// lanes each goes through every source in 1/g of a turn, and every 32-source tile costs about
// one and a half turns beside (its copy, wait and loop start): the remainder is either taken
// whole or cut at the largest power of two, whichever is cheaper in sum.
static int split_remainder(int left) {
    static const std::vector<int> next = [] {
        std::vector<int> n(kItemTargets + 1, 0);
        std::vector<double> cost(kItemTargets + 1, 0.0);
        for (int r = 1; r <= kItemTargets; r++) {
            const double tile = 1.5 / 32;
            int p = 1;
            while (p * 2 <= r) p *= 2;
            const double whole = 1.0 / (1 << lanes_log2(r)) + tile;
            const double cut = p < r ? 1.0 / (1 << lanes_log2(p)) + tile + cost[r - p] : whole;
            n[r] = cut < whole ? p : r;
            cost[r] = std::min(cut, whole);
        }
        return n;
    }();
    return next[std::min(left, kItemTargets)];
}

void build_split_items(int n_trg_box, const int *trg_begin, const int *trg_end, const int *list_off,
                       const int *list_ent, const int *src_begin, const int *src_end, int warps,
                       std::vector<WorkItem> &items, std::vector<PartGroup> &groups, long long &part_targets,
                       int shard_rank, int shard_n) {
    items.clear();
    groups.clear();
    part_targets = 0;
    struct Chunk {
        int box, t0, nt, glog;
        long long ns, turns;  // sources; sources a lane goes through
    };
    std::vector<Chunk> chunks;
    std::vector<int> size(n_trg_box > 0 ? list_off[n_trg_box] : 0);  // sources per entry
    long long total = 0;
    for (int b = 0; b < n_trg_box; b++) {
        const int nt = trg_end[b] - trg_begin[b];
        if (nt <= 0) continue;
        long long ns = 0;
        for (int e = list_off[b]; e < list_off[b + 1]; e++) {
            const int sb = list_ent[e] >> 5;
            ns += size[e] = src_end[sb] - src_begin[sb];
        }
        if (ns == 0) continue;
        for (int t0 = trg_begin[b], left = nt; left > 0;) {
            const int m = split_remainder(left);
            const int glog = lanes_log2(m);
            const long long turns = (ns + (1 << glog) - 1) >> glog;
            chunks.push_back({b, t0, m, glog, ns, turns});
            total += turns;
            t0 += m;
            left -= m;
        }
    }
    if (shard_n > 1) {
        // chunks dealt largest first to the least-loaded shard: the same assignment on every shard
        std::vector<int> idx, owner;
        std::vector<long long> turns;
        for (const Chunk &c : chunks) turns.push_back(c.turns);
        longest_first(turns, idx);
        std::vector<double> cost;
        for (int i : idx) cost.push_back((double)chunks[i].turns);
        partition_lpt((int)cost.size(), cost.data(), shard_n, owner);
        std::vector<Chunk> own;
        total = 0;
        for (size_t i = 0; i < idx.size(); i++)
            if (owner[i] == shard_rank) {
                own.push_back(chunks[idx[i]]);
                total += own.back().turns;
            }
        chunks.swap(own);
    }
    // A quarter of a warp's share, at least 64 sources per lane (a shorter run would be mostly
    // the first tile's latency and the output): 32k Stokes points, 128 per leaf, run as 4600
    // items of 64 x 384 pairs instead of 4096 of 8 x 1700.
    const long long cap = std::max(total / (4LL * std::max(warps, 1)), 64LL);
    std::vector<long long> cost;
    for (const Chunk &c : chunks) {
        const int g = 1 << c.glog;
        long long np = std::max(1LL, std::min(c.turns / std::max(cap / 2, 1LL), (c.turns + cap - 1) / cap));
        const long long len = ((c.ns + np - 1) / np + 31) / 32 * 32;
        np = (c.ns + len - 1) / len;
        int e = list_off[c.box];
        long long at = 0;  // sources of the entries before e
        const int part0 = (int)part_targets;
        for (long long j = 0; j < np; j++) {
            const long long a = j * len, z = std::min(c.ns, a + len);
            while (at + size[e] <= a) at += size[e++];  // the entry that holds source a
            WorkItem w{c.box, c.t0, c.nt, c.glog, e, e + 1};
            w.skip = (int)(a - at);
            long long end = at + size[e];
            while (end < z) end += size[w.e1++];
            w.stop = (int)(z - (end - size[w.e1 - 1]));
            if (np > 1) {
                w.part = (int)part_targets;
                part_targets += c.nt;
            }
            cost.push_back((z - a) / g);
            items.push_back(w);
        }
        if (np > 1) groups.push_back({c.t0, c.nt, part0, (int)np});
    }
    std::vector<int> idx;
    longest_first(cost, idx);
    std::vector<WorkItem> sorted;
    sorted.reserve(items.size());
    for (int i : idx) sorted.push_back(items[i]);
    items.swap(sorted);
}

long long pair_sources(const WorkItem &w, const int *list_ent, const int *src_begin, const int *src_end) {
    long long ns = 0;
    for (int e = w.e0; e < w.e1; e++) {
        const int sb = list_ent[e] >> 5;
        ns += src_end[sb] - src_begin[sb];
    }
    return ns;
}

void morton_order(const double *xyz, int n, std::vector<int> &order, std::vector<double> &sorted) {
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int i = 0; i < n; i++)
        for (int k = 0; k < 3; k++) {
            lo[k] = std::min(lo[k], xyz[3 * (size_t)i + k]);
            hi[k] = std::max(hi[k], xyz[3 * (size_t)i + k]);
        }
    double span = 0;
    for (int k = 0; k < 3; k++) span = std::max(span, hi[k] - lo[k]);
    const double inv = span > 0 ? 1.0 / (span * (1.0 + 1e-12)) : 0.0;
    std::vector<uint64_t> key(n);
    for (int i = 0; i < n; i++) {
        double u[3];
        for (int k = 0; k < 3; k++) u[k] = std::min(std::max((xyz[3 * (size_t)i + k] - lo[k]) * inv, 0.0), 0.999999999);
        key[i] = morton_key(u[0], u[1], u[2]);
    }
    sort_keys(key, order);
    sorted.resize(3 * (size_t)n);
    for (int i = 0; i < n; i++)
        for (int k = 0; k < 3; k++) sorted[3 * (size_t)i + k] = xyz[3 * (size_t)order[i] + k];
}

}  // namespace stk
