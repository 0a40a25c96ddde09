// stk_tree.cpp -- adaptive octree and KIFMM interaction lists (host C++).
#include "stk_tree.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>
#include <mutex>
#include <numeric>
#include <thread>

namespace stk {

namespace {

inline uint64_t spread3(uint64_t v) {
    v &= 0x1fffffULL;
    v = (v | (v << 32)) & 0x1f00000000ffffULL;
    v = (v | (v << 16)) & 0x1f0000ff0000ffULL;
    v = (v | (v << 8)) & 0x100f00f00f00f00fULL;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ULL;
    v = (v | (v << 2)) & 0x1249249249249249ULL;
    return v;
}

inline uint64_t interleave(uint64_t x, uint64_t y, uint64_t z) { return spread3(x) | (spread3(y) << 1) | (spread3(z) << 2); }

inline uint32_t quantize(double x) {
    const double s = (double)(1u << kMaxDepth);
    double q = std::floor(x * s);
    if (q < 0) q = 0;
    if (q > s - 1) q = s - 1;
    return (uint32_t)q;
}

// unique key of a node: a marker bit above the 3l Morton bits
inline uint64_t node_key(int l, uint64_t x, uint64_t y, uint64_t z) { return (1ULL << (3 * l)) | interleave(x, y, z); }

}  // namespace

uint64_t morton_key(double x, double y, double z) { return interleave(quantize(x), quantize(y), quantize(z)); }

void parallel_ranges(size_t n, size_t grain, const std::function<void(size_t, size_t)> &f) {
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t nt = std::min<size_t>({hw, 16, n / std::max<size_t>(grain, 1)});
    if (nt < 2) {
        f(0, n);
        return;
    }
    std::vector<std::thread> th;
    std::vector<std::exception_ptr> err(nt);
    auto run = [&](size_t i) {
        try {
            f(n * i / nt, n * (i + 1) / nt);
        } catch (...) {
            err[i] = std::current_exception();
        }
    };
    th.reserve(nt);
    size_t started = 1;
    try {
        for (; started < nt; started++) th.emplace_back(run, started);
    } catch (...) {  // no more threads, or no memory for one: the rest runs here
    }
    run(0);
    for (size_t i = started; i < nt; i++) run(i);
    for (auto &t : th) t.join();
    for (auto &e : err)
        if (e) std::rethrow_exception(e);
}

// Least-significant-digit radix sort of the leading 32 bits, 8 bits a pass (a Morton key of 10
// of its 20 levels: few keys agree that far), then the runs of equal leading bits by the whole
// key.  Every range of the keys counts its digits, and the counts of all ranges in digit order are
// where each range writes: equal keys keep their order on any number of threads.
void sort_keys(std::vector<uint64_t> &keys, std::vector<int> &perm) {
    const size_t n = keys.size();
    perm.resize(n);
    std::iota(perm.begin(), perm.end(), 0);
    if (n < 2) return;
    constexpr int kBits = 8, kBins = 1 << kBits, kTop = 28;  // four passes, from bit 28 of 60
    std::vector<uint64_t> keys2(n);
    std::vector<int> perm2(n);
    const size_t nr = n < (1u << 18) ? 1 : std::min<size_t>(16, n >> 16);  // ranges
    std::vector<size_t> count(nr * kBins);
    for (int shift = kTop; shift < 60; shift += kBits) {
        auto begin = [&](size_t r) { return n * r / nr; };
        parallel_ranges(nr, 1, [&](size_t r0, size_t r1) {
            for (size_t r = r0; r < r1; r++) {
                size_t *c = &count[r * kBins];
                std::fill(c, c + kBins, (size_t)0);
                for (size_t i = begin(r); i < begin(r + 1); i++) c[(keys[i] >> shift) & (kBins - 1)]++;
            }
        });
        size_t at = 0;
        bool one = false;  // every key has the same digit
        for (int d = 0; d < kBins; d++) {
            const size_t from = at;
            for (size_t r = 0; r < nr; r++) {
                const size_t c = count[r * kBins + d];
                count[r * kBins + d] = at;
                at += c;
            }
            one = one || at - from == n;
        }
        if (one) continue;
        parallel_ranges(nr, 1, [&](size_t r0, size_t r1) {
            for (size_t r = r0; r < r1; r++) {
                size_t *c = &count[r * kBins];
                for (size_t i = begin(r); i < begin(r + 1); i++) {
                    const size_t to = c[(keys[i] >> shift) & (kBins - 1)]++;
                    keys2[to] = keys[i];
                    perm2[to] = perm[i];
                }
            }
        });
        keys.swap(keys2);
        perm.swap(perm2);
    }
    std::vector<std::pair<uint64_t, int>> run;
    for (size_t i = 0; i < n;) {
        size_t j = i + 1;
        bool sorted = true;
        for (; j < n && (keys[j] >> kTop) == (keys[i] >> kTop); j++) sorted = sorted && keys[j - 1] <= keys[j];
        if (!sorted) {
            run.clear();
            for (size_t q = i; q < j; q++) run.push_back({keys[q], perm[q]});  // perm ascends within equal keys
            std::sort(run.begin(), run.end());
            for (size_t q = i; q < j; q++) {
                keys[q] = run[q - i].first;
                perm[q] = run[q - i].second;
            }
        }
        i = j;
    }
}

namespace {

// keys, permutation and coordinates of a point set in Morton order; false: a point outside [0,1)
bool sort_points(const double *xyz, int n, PointSet &ps) {
    ps.n = n;
    ps.key.resize(n);
    std::vector<char> bad(1, 0);
    parallel_ranges(n, 32768, [&](size_t a, size_t z) {
        for (size_t i = a; i < z; i++) {
            const double *p = xyz + 3 * i;
            if (!(p[0] >= 0.0 && p[0] < 1.0 && p[1] >= 0.0 && p[1] < 1.0 && p[2] >= 0.0 && p[2] < 1.0)) {
                __atomic_store_n(&bad[0], 1, __ATOMIC_RELAXED);
                return;
            }
            ps.key[i] = morton_key(p[0], p[1], p[2]);
        }
    });
    if (bad[0]) return false;
    sort_keys(ps.key, ps.perm);
    ps.xyz.resize(3 * (size_t)n);
    parallel_ranges(n, 32768, [&](size_t a, size_t z) {
        for (size_t i = a; i < z; i++) std::memcpy(&ps.xyz[3 * i], xyz + 3 * (size_t)ps.perm[i], 3 * sizeof(double));
    });
    return true;
}

}  // namespace

double Octree::side(int i) const { return std::ldexp(1.0, -level[i]); }

void Octree::corner(int i, double c[3]) const {
    const double h = side(i);
    c[0] = ix[i] * h;
    c[1] = iy[i] * h;
    c[2] = iz[i] * h;
}

void Octree::centre(int i, double c[3]) const {
    const double h = side(i);
    c[0] = (ix[i] + 0.5) * h;
    c[1] = (iy[i] + 0.5) * h;
    c[2] = (iz[i] + 0.5) * h;
}

int Octree::find(int l, int64_t x, int64_t y, int64_t z) const {
    auto it = lookup_.find(node_key(l, (uint64_t)x, (uint64_t)y, (uint64_t)z));
    return it == lookup_.end() ? -1 : it->second;
}

bool Octree::adjacent(int a, int shift, int b) const {
    const int L = std::max(level[a], level[b]);
    const int sa = L - level[a], sb = L - level[b];
    const int64_t n = 1LL << L;
    const int64_t s[3] = {shift % 3 - 1, (shift / 3) % 3 - 1, shift / 9 - 1};
    const uint32_t ac[3] = {ix[a], iy[a], iz[a]};
    const uint32_t bc[3] = {ix[b], iy[b], iz[b]};
    for (int k = 0; k < 3; k++) {
        const int64_t alo = ((int64_t)ac[k] << sa) + s[k] * n, ahi = alo + (1LL << sa);
        const int64_t blo = (int64_t)bc[k] << sb, bhi = blo + (1LL << sb);
        if (alo > bhi || blo > ahi) return false;
    }
    return true;
}

std::string Octree::build(const double *pts, int n, int max_pts, int max_depth, int pbc_) {
    if (n < 0 || (n > 0 && !pts)) return "invalid tree points";
    if (max_pts < 1) return "max_pts must be >= 1";
    if (pbc_ < 0 || pbc_ > 3) return "pbc must be 0..3";
    pbc = pbc_;
    max_depth = std::max(0, std::min(max_depth, kMaxDepth));
    if (!sort_points(pts, n, tree_)) return "tree point outside the unit box after scaling";
    const std::vector<uint64_t> &keys = tree_.key;

    level.assign(1, 0);
    parent.assign(1, -1);
    first_child.assign(1, -1);
    ix.assign(1, 0);
    iy.assign(1, 0);
    iz.assign(1, 0);
    key_lo_.assign(1, 0);
    std::vector<int> pbeg(1, 0), pend(1, n);
    for (size_t i = 0; i < level.size(); i++) {
        const int l = level[i];
        if (pend[i] - pbeg[i] <= max_pts || l >= max_depth) continue;
        first_child[i] = (int)level.size();
        const int cs = 3 * (kMaxDepth - l - 1);
        for (int c = 0; c < 8; c++) {
            const uint64_t lo = key_lo_[i] + ((uint64_t)c << cs);
            const uint64_t hi = lo + (1ULL << cs);
            level.push_back(l + 1);
            parent.push_back((int)i);
            first_child.push_back(-1);
            ix.push_back(2 * ix[i] + (c & 1));
            iy.push_back(2 * iy[i] + ((c >> 1) & 1));
            iz.push_back(2 * iz[i] + ((c >> 2) & 1));
            key_lo_.push_back(lo);
            pbeg.push_back((int)(std::lower_bound(keys.begin() + pbeg[i], keys.begin() + pend[i], lo) - keys.begin()));
            pend.push_back((int)(std::lower_bound(keys.begin() + pbeg[i], keys.begin() + pend[i], hi) - keys.begin()));
        }
    }
    const int nn = (int)level.size();
    max_level = level.back();
    level_begin.assign(max_level + 2, nn);
    for (int i = nn - 1; i >= 0; i--) level_begin[level[i]] = i;
    level_begin[max_level + 1] = nn;
    lookup_.clear();
    lookup_.reserve(nn * 2);
    for (int i = 0; i < nn; i++) lookup_[node_key(level[i], ix[i], iy[i], iz[i])] = i;
    leaves.clear();
    for (int i = 0; i < nn; i++)
        if (first_child[i] < 0) leaves.push_back(i);
    std::sort(leaves.begin(), leaves.end(), [&](int a, int b) { return key_lo_[a] < key_lo_[b]; });
    for (auto &s : sets) s = PointSet();
    U = V = W = X = NodeList();
    return "";
}

std::string Octree::assign(int set, const double *xyz, int n) {
    if (set < 0 || set > 2) return "invalid point set";
    if (n < 0 || (n > 0 && !xyz)) return "invalid points";
    PointSet &ps = sets[set];
    // the tree points themselves (sources and targets at the same points): sorted already.  The
    // coordinates in the caller's order are compared through the permutation.
    bool same = n == tree_.n && n > 0;
    if (same) {
        std::vector<char> differ(1, 0);
        parallel_ranges(n, 65536, [&](size_t a, size_t z) {
            for (size_t i = a; i < z; i++)
                if (std::memcmp(&tree_.xyz[3 * i], xyz + 3 * (size_t)tree_.perm[i], 3 * sizeof(double))) {
                    __atomic_store_n(&differ[0], 1, __ATOMIC_RELAXED);
                    return;
                }
        });
        same = !differ[0];
    }
    if (same)
        ps = tree_;
    else if (!sort_points(xyz, n, ps))
        return "point outside the unit box after scaling";
    const int nn = num_nodes();
    ps.node_begin.resize(nn);
    ps.node_end.resize(nn);
    for (int i = 0; i < nn; i++) {  // within the parent's range
        const uint64_t lo = key_lo_[i];
        const uint64_t hi = lo + (1ULL << (3 * (kMaxDepth - level[i])));
        const auto b = ps.key.begin() + (i ? ps.node_begin[parent[i]] : 0);
        const auto e = i ? ps.key.begin() + ps.node_end[parent[i]] : ps.key.end();
        ps.node_begin[i] = (int)(std::lower_bound(b, e, lo) - ps.key.begin());
        ps.node_end[i] = (int)(std::lower_bound(b, e, hi) - ps.key.begin());
    }
    return "";
}

namespace {
NodeList to_csr(const std::vector<std::vector<int>> &v) {
    NodeList L;
    L.off.resize(v.size() + 1, 0);
    for (size_t i = 0; i < v.size(); i++) L.off[i + 1] = L.off[i] + (int)v[i].size();
    L.ent.reserve(L.off.back());
    for (auto &x : v) L.ent.insert(L.ent.end(), x.begin(), x.end());
    return L;
}
}  // namespace

void Octree::build_lists() {
    const int nn = num_nodes();
    std::vector<std::vector<int>> Ul(nn), Vl(nn), Wl(nn), Xl(nn);
    const bool per[3] = {pbc >= 1, pbc >= 2, pbc >= 3};

    // Visit the 27 same-level neighbour positions of node b at level l, wrapping
    // periodic axes; calls f(node_or_-1, shift_code, wrapped position).
    auto neighbours = [&](int b, auto &&f) {
        const int l = level[b];
        const int64_t ns = 1LL << l;
        for (int dz = -1; dz <= 1; dz++)
            for (int dy = -1; dy <= 1; dy++)
                for (int dx = -1; dx <= 1; dx++) {
                    int64_t p[3] = {(int64_t)ix[b] + dx, (int64_t)iy[b] + dy, (int64_t)iz[b] + dz};
                    int s[3] = {0, 0, 0};
                    bool ok = true;
                    for (int k = 0; k < 3; k++) {
                        if (p[k] < 0 || p[k] >= ns) {
                            if (!per[k]) {
                                ok = false;
                                break;
                            }
                            s[k] = p[k] < 0 ? -1 : 1;
                            p[k] -= s[k] * ns;
                        }
                    }
                    if (!ok) continue;
                    f(find(l, p[0], p[1], p[2]), shift_code(s[0], s[1], s[2]), p, l);
                }
    };

    // every entry once, in ascending order
    auto finish = [](std::vector<int> &x) {
        std::sort(x.begin(), x.end());
        x.erase(std::unique(x.begin(), x.end()), x.end());
    };
    // nodes are independent of each other (U, W, V): spread over the host's threads
    constexpr size_t kGrain = 128;
    parallel_ranges(leaves.size(), kGrain, [&](size_t first, size_t last) {
    std::vector<int> stack;
    for (size_t li = first; li < last; li++) {
        const int b = leaves[li];
        if (trg_count(b) == 0) continue;
        auto addU = [&](int node, int code) {
            if (src_count(node) > 0) Ul[b].push_back((node << 5) | code);
        };
        auto addW = [&](int node, int code) {
            if (src_count(node) > 0) Wl[b].push_back((node << 5) | code);
        };
        neighbours(b, [&](int node, int code, const int64_t *p, int l) {
            if (node >= 0) {
                if (is_leaf(node)) {
                    addU(node, code);
                    return;
                }
                stack.assign(1, node);
                while (!stack.empty()) {
                    const int m = stack.back();
                    stack.pop_back();
                    for (int c = first_child[m]; c < first_child[m] + 8; c++) {
                        if (src_count(c) == 0) continue;
                        if (adjacent(c, code, b)) {
                            if (is_leaf(c))
                                addU(c, code);
                            else
                                stack.push_back(c);
                        } else {
                            addW(c, code);
                        }
                    }
                }
            } else {
                // the position is covered by a coarser leaf
                int a = -1;
                for (int ll = l - 1; ll >= 0 && a < 0; ll--)
                    a = find(ll, p[0] >> (l - ll), p[1] >> (l - ll), p[2] >> (l - ll));
                if (a >= 0) addU(a, code);
            }
        });
        finish(Ul[b]);
        finish(Wl[b]);
    }
    });

    // V: children of the parent's colleagues that are not adjacent
    parallel_ranges(nn, kGrain, [&](size_t first, size_t last) {
    for (int b = std::max(1, (int)first); b < (int)last; b++) {
        if (trg_count(b) == 0) continue;
        const int P = parent[b];
        neighbours(P, [&](int node, int code, const int64_t *, int) {
            if (node < 0 || is_leaf(node)) return;
            for (int c = first_child[node]; c < first_child[node] + 8; c++) {
                if (src_count(c) == 0) continue;
                if (!adjacent(c, code, b)) Vl[b].push_back((c << 5) | code);
            }
        });
        std::sort(Vl[b].begin(), Vl[b].end());
    }
    });

    // X: the W relation seen from the source side.  For every leaf a with
    // sources, the nodes with targets that are descendants of a's colleagues,
    // not adjacent to a, with a parent adjacent to a, gain a (with the inverse
    // shift).  Walking from the source leaves also covers source leaves that hold
    // no targets, which have no W list of their own.
    std::mutex x_mutex;
    parallel_ranges(leaves.size(), kGrain, [&](size_t first, size_t last) {
    std::vector<std::pair<int, int>> found;  // (node, entry)
    std::vector<int> stack;
    for (size_t li = first; li < last; li++) {
        const int a = leaves[li];
        if (src_count(a) == 0) continue;
        neighbours(a, [&](int node, int code, const int64_t *, int) {
            if (node < 0 || is_leaf(node)) return;
            stack.assign(1, node);
            while (!stack.empty()) {
                const int m = stack.back();
                stack.pop_back();
                for (int c = first_child[m]; c < first_child[m] + 8; c++) {
                    if (trg_count(c) == 0) continue;
                    if (adjacent(c, code, a)) {
                        if (!is_leaf(c)) stack.push_back(c);
                    } else {
                        found.push_back({c, (a << 5) | shift_negate(code)});
                    }
                }
            }
        });
    }
    std::lock_guard<std::mutex> lock(x_mutex);
    for (const auto &f : found) Xl[f.first].push_back(f.second);
    });
    for (auto &x : Xl) finish(x);

    U = to_csr(Ul);
    V = to_csr(Vl);
    W = to_csr(Wl);
    X = to_csr(Xl);
}

void partition_lpt(int n, const double *cost, int nparts, std::vector<int> &owner) {
    owner.assign(n, 0);
    if (nparts <= 1) return;
    std::vector<double> load(nparts, 0.0);
    for (int i = 0; i < n; i++) {
        int best = 0;
        for (int r = 1; r < nparts; r++)
            if (load[r] < load[best]) best = r;
        owner[i] = best;
        load[best] += cost[i];
    }
}

// Owners of the M2L / S2L target nodes when the far field is split over nranks:
// the nodes of complete levels (all 8^l boxes, l >= 1) by parity type
// ((ix & 1) | (iy & 1) << 1 | (iz & 1) << 2) mod nranks -- the dense M2L splits
// its work by target type -- and every other node, largest first by its V-list
// and X-list size, to the least loaded rank (LPT).  Host only, deterministic.
std::vector<int> far_owners(const Octree &T, int nranks) {
    const int nn = T.num_nodes();
    std::vector<int> owner(nn, 0);
    if (nranks <= 1) return owner;
    std::vector<double> load(nranks, 0.0);
    std::vector<char> done(nn, 0);
    auto cost = [&](int b) { return 1.0 + (T.V.off[b + 1] - T.V.off[b]) + (T.X.off[b + 1] - T.X.off[b]); };
    for (int l = 1; l <= T.depth(); l++) {
        const long long cnt = (long long)T.level_begin[l + 1] - T.level_begin[l];
        if (cnt != (1LL << (3 * l))) continue;
        for (int b = T.level_begin[l]; b < T.level_begin[l + 1]; b++) {
            const int c = (int)((T.ix[b] & 1) | (T.iy[b] & 1) << 1 | (T.iz[b] & 1) << 2);
            owner[b] = c % nranks;
            load[owner[b]] += cost(b);
            done[b] = 1;
        }
    }
    std::vector<int> rest;
    for (int b = 0; b < nn; b++)
        if (!done[b]) rest.push_back(b);
    std::stable_sort(rest.begin(), rest.end(), [&](int a, int b) { return cost(a) > cost(b); });
    for (int b : rest) {
        int best = 0;
        for (int r = 1; r < nranks; r++)
            if (load[r] < load[best]) best = r;
        owner[b] = best;
        load[best] += cost(b);
    }
    return owner;
}

}  // namespace stk
