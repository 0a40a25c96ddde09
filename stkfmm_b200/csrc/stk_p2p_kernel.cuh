// stk_p2p_kernel.cuh -- the list / direct P2P kernel of every micro-kernel (instances: stk_p2p_list_*.cu,
// stk_p2p_direct_*.cu; launches: stk_p2p.cu).
//
// Replaces the per-(target box, source box) ker_poten calls that PVFMM's
// PtFMM_Evaluate makes for the U-list (S2T), and the OpenMP target-chunk loop of
// FMMData::evaluateKernel (Lib/src/FMMData.cpp:252-283).
//
// Design (one warp = one work item, persistent warps):
//  * A work item is <= 64 targets of one target box plus a range of its
//    interaction-list entries.  Items are sorted by cost on the host, largest
//    first; persistent warps take them from a global counter, so uneven
//    adaptive trees balance themselves.
//  * Each lane owns two target slots (lane and lane + 32).  With fewer than 64
//    targets, 2^glog consecutive lanes share a target and split the source
//    tile; they are reduced with warp shuffles at the end.
//  * The sources of an item's list entries form one stream: each entry is a
//    segment (its source box's records, with its periodic shift), and the warp
//    walks the concatenated stream in 32-source tiles that cross segment
//    boundaries, so only the last tile of an item is padded (with one tile per
//    entry, padding was ~19% of the evaluated pairs on clustered trees).
//  * Tiles: lane i copies the record of stream position i of the next tile into
//    its own shared-memory slot with cp.async (16-byte asynchronous copies,
//    L2 -> shared) while the current tile is consumed.  Records carry the
//    per-source staged values (Uk<>::stage), computed once by the pack kernel.
//  * FP64 path: one source and two targets per step, records read as they landed
//    (16-byte broadcast loads; a lane only adds a periodic shift to its own
//    record); r = x_t - (x_s + shift) formed in double exactly as the oracle
//    forms it.  Long items are split by source ranges, their sums kept apart and
//    added in order by a second kernel (build_split_items).
//  * Mixed path: the lane splits its landed record into a column of a
//    structure-of-arrays tile (one row per component).
//  * Mixed path: at staging each source coordinate, shifted to the target
//    box's centre c in FP64, is split into FP32 hi + lo parts
//    (x - c = hi + lo to ~2^-48 relative); targets likewise.  Per pair the
//    displacement (t_hi - s_hi) + (t_lo - s_lo) is then accurate to FP32
//    relative precision even for nearly coincident points (t_hi - s_hi is exact
//    by Sterbenz' lemma when the points are close).  The kernel tensor runs in
//    Blackwell packed FP32 (fma.rn.f32x2: two sources per instruction) with
//    MUFU rsqrt + one Newton step; each tile's FP32 partial sums are added into
//    Kahan-compensated FP32 accumulators.
#pragma once
#include <algorithm>
#include <type_traits>

#include "stk_p2p.cuh"
#include "stk_ukernels.cuh"

namespace stk {

namespace {

// Warps per CTA.  Every warp works alone (warp-level synchronisation only), so
// this only sets the granularity in which registers fill an SM: one warp per CTA
// lets the FP64 kernels use every register slot (14 warps per SM at 140
// registers instead of 12 in 4-warp CTAs: the benchmark's FP64 launch 1.1%
// faster); the mixed kernels measured best at 4.
template <bool MIXED> struct Cta {
    static constexpr int warps = MIXED ? 4 : 1;
    static constexpr int threads = 32 * warps;
};
constexpr unsigned kFull = 0xffffffffu;
constexpr double kPadCoord = 1.0e4;  // offset of zero-strength padding sources
constexpr int kShiftNoneCode = 13;   // list-entry shift code of the unshifted source box
constexpr int kMayCoincide = 32;     // segment-table flag above the 5-bit shift code

// Number of staged per-output-point values of a micro-kernel (1 as a dummy
// array size when it has none).
template <class K, class = void> struct NtvOf {
    static constexpr int value = 1;
};
template <class K> struct NtvOf<K, std::void_t<decltype(K::NTV)>> {
    static constexpr int value = K::NTV;
};

template <int UK> struct Rec {
    static constexpr int SDIM = Uk<UK>::SDIM;
    // doubles (16-byte multiples) of a record with the source's values, and with its staged values
    static constexpr int RAW = (3 + SDIM + 1) & ~1, STAGED = (3 + Uk<UK>::NV + 1) & ~1;
    // Records carry staged values unless that makes them larger (laplace_pgrad, the Hessian and
    // gradient kernels); those, and a direct sum's sources, are staged in every tile that reads
    // them (262k points, lists of 1728 sources, mixed: laplace_dipolepgradgrad 10 doubles staged
    // 1032 us, 6 raw 970; stokes_pvellaplacian 10 857, 8 814; FP64 the same to 1%).
    static constexpr bool kStaged = STAGED <= RAW;
    static constexpr int RS = kStaged ? STAGED : RAW;  // doubles per record
    static constexpr int SLOT = STAGED > RAW ? STAGED : RAW;  // landing slot of values staged in place
};

// Resident CTAs per SM requested from the register allocator (1: no
// constraint; forcing 5 measured slower for the FP64 path and neutral for the
// mixed path).  STK_MINB_OVERRIDE builds tuning variants.
template <int UK, bool MIXED> struct MinBlocks {
#ifdef STK_MINB_OVERRIDE
    static constexpr int value = STK_MINB_OVERRIDE;
#else
    static constexpr int value = 1;
#endif
};

// How the mixed path forms the displacement (STK_MIXED_DISP selects at build time):
//   kDispHiLo: FP32 hi + lo parts of the centre-relative coordinates, 3 FP32
//              operations per coordinate and pair on the FP32 pipe;
//   kDispF64:  centre-relative coordinates kept in FP64 in shared memory, one
//              FP64 subtraction and one FP64->FP32 rounding per coordinate and
//              pair, on the otherwise idle FP64 pipe.
constexpr int kDispHiLo = 0, kDispF64 = 1;
#ifdef STK_MIXED_DISP
constexpr int kMixedDisp = STK_MIXED_DISP;
#else
constexpr int kMixedDisp = kDispHiLo;
#endif
static_assert(kMixedDisp == kDispHiLo || kMixedDisp == kDispF64, "STK_MIXED_DISP must be 0 or 1");

// Unroll of the source loop (tuning builds override it)
#ifndef STK_P2P_UNROLL_MIXED
#define STK_P2P_UNROLL_MIXED 2
#endif
#ifndef STK_P2P_UNROLL_FP64
#define STK_P2P_UNROLL_FP64 2
#endif
#define STK_PRAGMA(x) _Pragma(#x)
#define STK_UNROLL(n) STK_PRAGMA(unroll n)

// Target slots per lane: 2 (a warp holds 64 targets), or 4 for small micro-kernels
// in builds with STK_P2P_TPL4 (twice the targets per staged source pair, the
// host's lanes-per-target doubled to keep every target covered).
#ifndef STK_P2P_TPL4
#define STK_P2P_TPL4 0
#endif
template <class K> struct TargetsPerLane {
    static constexpr int value = (STK_P2P_TPL4 && K::TDIM <= 4 && K::NV <= 8 && K::TV == 0) ? 4 : 2;
};

// Mixed path: the packed FP32 partial sums go into the Kahan accumulators every
// kKahanTiles * g tiles, i.e. after ~32 kKahanTiles sources per lane whatever
// the lanes per target g (STK_KAHAN_TILES overrides; the step costs ~5 FP32
// operations per output, which per 32-source tile was ~7% of the instructions
// when g > 1).
#ifndef STK_KAHAN_TILES
#define STK_KAHAN_TILES 1
#endif
constexpr int kKahanTiles = STK_KAHAN_TILES;

// cp.async (Ampere+ asynchronous global -> shared copy, 16 bytes per lane and
// instruction, L2 only): the next tile's raw source records land in shared memory
// while the current tile is consumed, so no register holds a prefetched record.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// wait until at most N of this thread's most recent groups are still in flight
template <int N> __device__ __forceinline__ void cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Tiles in flight per warp (STK_P2P_DEPTH builds deeper pipelines where the landing
// zones fit the 48 KB of static shared memory per block).  One tile ahead is the
// default: two measured 0.5% slower on the clustered 1M-point LapPGrad U list
// (3.100 against 3.084 ms mixed, 4.446 against 4.409 ms FP64), so the L2 round
// trip is hidden behind one tile's consumption even for items of 8 targets.
#ifndef STK_P2P_DEPTH
#define STK_P2P_DEPTH 1
#endif
template <int RS> struct StageDepth {
    static constexpr int value = RS <= 10 ? STK_P2P_DEPTH : 1;
};

// FP32 hi part of a double by truncation: the top 24 significant bits (the low
// 29 mantissa bits cleared), so (float)hi is exact and d - hi is exact in FP64.
__device__ __forceinline__ double trunc_to_f32_bits(double d) {
    return __hiloint2double(__double2hiint(d), __double2loint(d) & (int)0xE0000000u);
}

// Shared-memory stride (doubles) of a raw record: an odd number of 16-byte units,
// so the 8 lanes of a quarter-warp reading their own records with 16-byte loads
// hit 8 distinct bank groups.
template <int RS> struct RawStride {
    static constexpr int value = ((RS / 2) & 1) ? RS : RS + 2;
};

// One component of a source record from the caller's own arrays (8 bytes, no alignment
// beyond a double's).
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

// DIRECT: a direct sum (launch_direct_p2p).  Item it is targets [64 c, ...) against source chunk
// k, c the fast index: the warps of an SM read the same sources.  Sources come straight from
// the caller's arrays, and there are no lists to read or to set up.
template <int UK, bool MIXED, bool DIRECT>
__global__ void __launch_bounds__(Cta<MIXED>::threads, MinBlocks<UK, MIXED>::value)
    list_p2p_kernel(const __grid_constant__ ListP2PArgs a) {
    constexpr int kWarpsPerCta = Cta<MIXED>::warps;
    using K = Uk<UK>;
    constexpr int TDIM = K::TDIM;
    constexpr int NV = K::NV;
    constexpr int TV = K::TV;  // per-output-point values (adjoint kernels)
    constexpr int NTV = NtvOf<K>::value;
    constexpr int RS = Rec<UK>::RS;
    constexpr bool STAGE = DIRECT || !Rec<UK>::kStaged;  // values are staged here
    constexpr int RSS = RawStride<STAGE ? Rec<UK>::SLOT : RS>::value;
    constexpr int TPL = TargetsPerLane<K>::value;
    constexpr bool HILO = MIXED && kMixedDisp == kDispHiLo;
    // shared tile, one row per component: coordinates (FP64, or FP32 hi x3 + lo x3)
    // and staged values (FP64 path: double, mixed path: float)
    constexpr int NCC = HILO ? 6 : 3;
    using CT = typename std::conditional<HILO, float, double>::type;
    using S = typename std::conditional<MIXED, float, double>::type;

    // (mixed path only: the FP64 path reads the landed records as they are)
    __shared__ __align__(16) CT tcoord[kWarpsPerCta][MIXED ? NCC : 1][MIXED ? 32 : 1];
    __shared__ __align__(16) S tval[kWarpsPerCta][MIXED ? NV : 1][MIXED ? 32 : 1];
    constexpr int DEPTH = MIXED ? StageDepth<RS>::value : 2;  // FP64: one zone read, one landing
    // cp.async landing zones, one record per lane and tile in flight
    __shared__ __align__(16) double traw[kWarpsPerCta][DEPTH][32][RSS];
    // the item's list entries (up to 32 at a time) as segments of one source stream
    __shared__ int sg_end[kWarpsPerCta][32];   // stream position one past the segment
    __shared__ int sg_src[kWarpsPerCta][32];   // first record of the segment minus its stream start
    __shared__ int sg_code[kWarpsPerCta][32];  // periodic shift code
    const int wid = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    auto &mc = tcoord[wid];
    auto &mv = tval[wid];
    int *s_end = sg_end[wid];
    int *s_src = sg_src[wid];
    int *s_code = sg_code[wid];

    for (int turn = 0;; turn++) {
        int it = 0;
        WorkItem w;
        if constexpr (DIRECT) {
            // Equal items.  FP64: dealt in turn (direct_chunks fills whole turns).  Mixed: taken from the
            // counter, as their number fills the last turn anyhow (50k x 50k points, dealt: rpy_u 3.30
            // ms, 3.02 taken; stokes_regftvel 4.73, 4.49).
            if constexpr (MIXED) {
                if (lane == 0) it = (int)atomicAdd(a.counter, 1u);
                it = __shfl_sync(kFull, it, 0);
            } else {
                it = (turn * gridDim.x + blockIdx.x) * kWarpsPerCta + wid;
            }
            if (it >= a.n_items) break;
            const int nc = (a.ntrg + 63) >> 6, c = it % nc;
            w.trg_box = c;
            w.t0 = 64 * c;
            w.nt = min(64, a.ntrg - w.t0);
            w.glog = w.nt > 32 ? 0 : min(5, __clz(w.nt - 1) - 26);  // 2^glog <= 64 / nt
            w.e0 = it / nc;
            w.e1 = w.e0 + 1;
        } else {
            if (lane == 0) it = (int)atomicAdd(a.counter, 1u);
            it = __shfl_sync(kFull, it, 0);
            if (it >= a.n_items) break;
            w = a.items[it];
        }
        // the host sizes glog for 64 slots; 4 slots per lane give twice the lanes per target
        const int glog = TPL == 4 ? min(5, w.glog + 1) : w.glog;
        const int g = 1 << glog;
        const int sub = lane & (g - 1);
        bool act[TPL];
        int tt[TPL];
#pragma unroll
        for (int h = 0; h < TPL; h++) {
            const int ti = (lane + 32 * h) >> glog;
            act[h] = ti < w.nt;
            tt[h] = w.t0 + (act[h] ? ti : 0);
        }

        double c[3] = {0.0, 0.0, 0.0};
        if constexpr (MIXED) {
            // local origin: the target box centre, or the item's first target
            const double *o = a.box_centre ? a.box_centre + 3 * (size_t)w.trg_box : a.trg_xyz + 3 * (size_t)w.t0;
            c[0] = o[0];
            c[1] = o[1];
            c[2] = o[2];
        }
        double xt[TPL][3];
#pragma unroll
        for (int h = 0; h < TPL; h++)
#pragma unroll
            for (int k = 0; k < 3; k++) xt[h][k] = a.trg_xyz[3 * (size_t)tt[h] + k];

        // per-output-point values, staged once per item
        using V = typename std::conditional<MIXED, F2, double>::type;
        V ta[TPL][NTV];
        if constexpr (TV > 0) {
#pragma unroll
            for (int h = 0; h < TPL; h++) {
                double r0[TV], s0[NTV];
#pragma unroll
                for (int q = 0; q < TV; q++) r0[q] = a.trg_aux[(size_t)tt[h] * TV + q];
                K::stage_aux(r0, s0);
#pragma unroll
                for (int q = 0; q < NTV; q++) {
                    if constexpr (MIXED)
                        ta[h][q] = splat((float)s0[q]);
                    else
                        ta[h][q] = s0[q];
                }
            }
        }
        auto eval = [&](auto &u, auto dx, auto dy, auto dz, const auto *sv, const auto *tav) {
            if constexpr (TV > 0)
                K::eval(u, dx, dy, dz, sv, tav);
            else
                K::eval(u, dx, dy, dz, sv);
        };

        // accumulators: FP64 path sums directly; mixed path keeps Kahan sum + compensation
        S acc[TPL][TDIM], cmp[TPL][TDIM];
#pragma unroll
        for (int h = 0; h < TPL; h++)
#pragma unroll
            for (int k = 0; k < TDIM; k++) acc[h][k] = cmp[h][k] = S(0);
        // mixed path: packed FP32 partial sums, added into the Kahan accumulators in steps
        F2 pp[TPL][TDIM];
#pragma unroll
        for (int h = 0; h < TPL; h++)
#pragma unroll
            for (int k = 0; k < TDIM; k++) pp[h][k] = splat(0.0f);
        int kahan_tiles = 0;
        auto kahan_step = [&]() {
            if constexpr (MIXED) {
#pragma unroll
                for (int h = 0; h < TPL; h++)
#pragma unroll
                    for (int k = 0; k < TDIM; k++) {
                        const float y = (pp[h][k].v.x + pp[h][k].v.y) - cmp[h][k];
                        const float t = acc[h][k] + y;
                        cmp[h][k] = (t - acc[h][k]) - y;
                        acc[h][k] = t;
                        pp[h][k] = splat(0.0f);
                    }
            }
            kahan_tiles = 0;
        };
        F2 th[TPL][3], tl[TPL][3];  // hi/lo targets (HILO)
        double tr[TPL][3];          // centre-relative targets (FP64 displacement)
#pragma unroll
        for (int h = 0; h < TPL; h++)
#pragma unroll
            for (int k = 0; k < 3; k++) tr[h][k] = xt[h][k] - c[k];
        if constexpr (HILO) {
#pragma unroll
            for (int h = 0; h < TPL; h++)
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const float hv = (float)tr[h][k];
                    th[h][k] = splat(hv);
                    tl[h][k] = splat((float)(tr[h][k] - (double)hv));
                }
        }

        // ---- the item's sources as one stream: its list entries, 32 at a time, in
        // order, each a segment of its source box's records; tiles of 32 stream
        // positions cross segment boundaries, so only a chunk's last tile is padded ----
        for (int ec = w.e0; ec < w.e1; ec += 32) {
            const int ne = min(32, w.e1 - ec);
            int sz = 0, sbeg = 0, code = kShiftNoneCode;
            if constexpr (!DIRECT) if (lane < ne) {
                const int ent = a.list_ent[ec + lane];
                const int sb = ent >> 5;
                code = ent & 31;
                sbeg = a.src_box_begin[sb];
                sz = a.src_box_end[sb] - sbeg;
                // mixed items hold whole entries; looking for parts of them cost 4 registers, and
                // the adjoint and dipole kernels a CTA per SM (262k points: regvel_adjoint_trg 777 ->
                // 824 us)
                if constexpr (!MIXED) {
                    if (ec + lane == w.e1 - 1) sz = min(sz, w.stop);
                    if (ec + lane == w.e0) {
                        sbeg += w.skip;
                        sz -= w.skip;
                    }
                }
                // bit 5: the segment may hold a source at a target's position (always,
                // unless the lists guarantee coincidence only in the unshifted own box)
                if (!a.coincident_own_box || sb == w.trg_box || code != kShiftNoneCode) code |= kMayCoincide;
            }
            int total;
            if constexpr (DIRECT) {
                sbeg = w.e0 * a.src_chunk;
                total = min(a.src_chunk, a.nsrc - sbeg);
            } else {
                int incl = sz;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += v;
                }
                total = __shfl_sync(kFull, incl, 31);
                __syncwarp();  // the previous chunk's segment table is no longer read
                s_end[lane] = lane < ne ? incl : 0x7fffffff;
                s_src[lane] = sbeg - (incl - sz);
                s_code[lane] = code;
                __syncwarp();
                if (total == 0) continue;
            }

            // per-lane cursor into the segment table; positions only grow
            int seg = 0;
            // segment of the record in each landing zone, oldest first (registers:
            // every index below is a compile-time constant)
            int zseg[DEPTH];
            // cp.async the record at stream position p into this lane's slot of zone z,
            // or nothing past the stream's end; one commit group per call either way,
            // so every lane counts the same groups
            auto fetch = [&](int p, int z, int &zs) {
                if constexpr (DIRECT) {
                    if (p < total) {
                        const double *x = a.src_xyz + 3 * (size_t)(sbeg + p), *v = a.src_val + (size_t)K::SDIM * (sbeg + p);
                        double *dst = traw[wid][z][lane];
#pragma unroll
                        for (int q = 0; q < 3; q++) cp_async8(dst + q, x + q);
#pragma unroll
                        for (int q = 0; q < K::SDIM; q++) cp_async8(dst + 3 + q, v + q);
                    }
                } else if (p < total) {
                    while (p >= s_end[seg]) seg++;
                    const double *src = a.src_rec + (size_t)(s_src[seg] + p) * RS;
                    double *dst = traw[wid][z][lane];
#pragma unroll
                    for (int q = 0; q < RS / 2; q++) cp_async16(dst + 2 * q, src + 2 * q);
                    zs = seg;
                }
                cp_async_commit();
            };
            if constexpr (!MIXED) {
                // ---- FP64: tiles are read straight from their landing zone (records carry
                // staged values; a lane's record is broadcast to the lanes of a target group) ----
                fetch(lane, 0, zseg[0]);
                int zone = 0;
                for (int p0 = 0; p0 < total; p0 += 32, zone ^= 1) {
                    const int n = min(32, total - p0);
                    cp_async_wait_group<0>();
                    if (lane < n) {  // fix up this lane's own record in place
                        double *raw = traw[wid][zone][lane];
                        if constexpr (STAGE) {
                            double f[K::SDIM], v[NV];
#pragma unroll
                            for (int q = 0; q < K::SDIM; q++) f[q] = raw[3 + q];
                            K::stage(f, v);
#pragma unroll
                            for (int q = 0; q < NV; q++) raw[3 + q] = v[q];
                        }
                        if constexpr (!DIRECT) {
                            const int cd = s_code[zseg[0]] & 31;
                            if (cd != kShiftNoneCode) {  // periodic image
                                raw[0] += (cd % 3 - 1) * a.period;
                                raw[1] += ((cd / 3) % 3 - 1) * a.period;
                                raw[2] += (cd / 9 - 1) * a.period;
                            }
                        }
                    }
                    __syncwarp();  // the tile is complete, and the previous one no longer read
                    fetch(p0 + 32 + lane, zone ^ 1, zseg[0]);
                    const double(*tile)[RSS] = traw[wid][zone];
STK_UNROLL(STK_P2P_UNROLL_FP64)
                    for (int j = sub; j < n; j += g) {
                        constexpr int RN = Rec<UK>::STAGED;
                        double rn[RN];
#pragma unroll
                        for (int q = 0; q < RN / 2; q++) {
                            const double2 t2 = *reinterpret_cast<const double2 *>(&tile[j][2 * q]);
                            rn[2 * q] = t2.x;
                            rn[2 * q + 1] = t2.y;
                        }
#pragma unroll
                        for (int h = 0; h < TPL; h++)
                            eval(acc[h], xt[h][0] - rn[0], xt[h][1] - rn[1], xt[h][2] - rn[2], rn + 3, ta[h]);
                    }
                }
                __syncwarp();  // the last tile has been read
                continue;
            }
#pragma unroll
            for (int z = 0; z < DEPTH; z++) fetch(32 * z + lane, z, zseg[z]);
            int p0 = 0, zone = 0;
            while (p0 < total) {
                const int n = min(32, total - p0);
                // ---- stage: lane i turns stream position p0 + i (its landed record)
                // into tile column i, or writes zero-strength padding ----
                cp_async_wait_group<DEPTH - 1>();  // this tile's group; later ones may still fly
                __syncwarp();  // every lane has finished reading the previous tile
                int may_coincide = 0;
                {
                    double v[NV];
                    double x[3];
                    if (lane < n) {
                        const double *raw = traw[wid][zone][lane];
                        constexpr int RR = STAGE ? Rec<UK>::RAW : RS;
                        double rn[RR];
#pragma unroll
                        for (int q = 0; q < RR / 2; q++) {
                            const double2 t2 = *reinterpret_cast<const double2 *>(raw + 2 * q);
                            rn[2 * q] = t2.x;
                            rn[2 * q + 1] = t2.y;
                        }
                        x[0] = rn[0];
                        x[1] = rn[1];
                        x[2] = rn[2];
                        if constexpr (DIRECT) {
                            may_coincide = 1;
                        } else {
                            const int cdf = s_code[zseg[0]];
                            may_coincide = cdf & kMayCoincide;
                            const int cd = cdf & 31;
                            if (cd != kShiftNoneCode) {  // periodic image
                                x[0] += (cd % 3 - 1) * a.period;
                                x[1] += ((cd / 3) % 3 - 1) * a.period;
                                x[2] += (cd / 9 - 1) * a.period;
                            }
                        }
                        if constexpr (STAGE) {
                            K::stage(rn + 3, v);
                        } else {
#pragma unroll
                            for (int q = 0; q < NV; q++) v[q] = rn[3 + q];
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 3; k++) x[k] = c[k] + kPadCoord;
#pragma unroll
                        for (int q = 0; q < NV; q++) v[q] = 0.0;
                    }
                    if constexpr (HILO) {
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            const double d = x[k] - c[k];
                            const double hd = trunc_to_f32_bits(d);
                            mc[k][lane] = (float)hd;
                            mc[3 + k][lane] = (float)(d - hd);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 3; k++) mc[k][lane] = x[k] - c[k];
                    }
#pragma unroll
                    for (int q = 0; q < NV; q++) mv[q][lane] = (S)v[q];
                }
                // ---- prefetch the tile DEPTH ahead into the zone just staged ----
#pragma unroll
                for (int z = 0; z + 1 < DEPTH; z++) zseg[z] = zseg[z + 1];
                fetch(p0 + 32 * DEPTH + lane, zone, zseg[DEPTH - 1]);
                p0 += 32;
                zone = DEPTH > 1 ? (zone + 1 == DEPTH ? 0 : zone + 1) : 0;
                __syncwarp();

                // ---- consume the tile ----
                if constexpr (MIXED) {
                    // sources j, j+1 in one packed pair; entries [n, n+1] are zero-strength padding.
                    // P: F2 (rsqrt masks coincident pairs) or F2U (no source of the tile can sit
                    // at a target's position)
                    auto consume = [&](auto proto) {
                        using P = decltype(proto);
STK_UNROLL(STK_P2P_UNROLL_MIXED)
                        for (int j = 2 * sub; j < n; j += 2 * g) {
                            P sv[NV];
#pragma unroll
                            for (int q = 0; q < NV; q++) sv[q].v = *reinterpret_cast<const float2 *>(&mv[q][j]);
                            P dxyz[TPL][3];
                            if constexpr (HILO) {
                                F2 sh[3], sl[3];
#pragma unroll
                                for (int k = 0; k < 3; k++) {
                                    sh[k].v = *reinterpret_cast<const float2 *>(&mc[k][j]);
                                    sl[k].v = *reinterpret_cast<const float2 *>(&mc[3 + k][j]);
                                }
#pragma unroll
                                for (int h = 0; h < TPL; h++)
#pragma unroll
                                    for (int k = 0; k < 3; k++)
                                        dxyz[h][k].v = ((th[h][k] - sh[k]) + (tl[h][k] - sl[k])).v;
                            } else {
                                double2 sx[3];
#pragma unroll
                                for (int k = 0; k < 3; k++) sx[k] = *reinterpret_cast<const double2 *>(&mc[k][j]);
#pragma unroll
                                for (int h = 0; h < TPL; h++)
#pragma unroll
                                    for (int k = 0; k < 3; k++)
                                        dxyz[h][k].v = make_float2((float)(tr[h][k] - sx[k].x),
                                                                   (float)(tr[h][k] - sx[k].y));
                            }
#pragma unroll
                            for (int h = 0; h < TPL; h++) {
                                P u[TDIM], tv[NTV];
#pragma unroll
                                for (int k = 0; k < TDIM; k++) u[k].v = pp[h][k].v;
#pragma unroll
                                for (int q = 0; q < NTV; q++) tv[q].v = ta[h][q].v;
                                eval(u, dxyz[h][0], dxyz[h][1], dxyz[h][2], sv, tv);
#pragma unroll
                                for (int k = 0; k < TDIM; k++) pp[h][k].v = u[k].v;
                            }
                        }
                    };
                    if (__any_sync(kFull, may_coincide))
                        consume(F2{});
                    else
                        consume(F2U{});
                    // Kahan-compensated accumulation of the partial sums once a lane has
                    // evaluated ~32 sources since the last step (every g tiles)
                    if (++kahan_tiles >= kKahanTiles * g) kahan_step();
                }
            }
        }
        __syncwarp();
        if (kahan_tiles > 0) kahan_step();

        // ---- reduce the lanes that share a target, then accumulate ----
        double o[TPL][TDIM];
#pragma unroll
        for (int h = 0; h < TPL; h++)
#pragma unroll
            for (int k = 0; k < TDIM; k++) {
                if constexpr (MIXED)
                    o[h][k] = double(acc[h][k]) - double(cmp[h][k]);
                else
                    o[h][k] = acc[h][k];
            }
        for (int off = 1; off < g; off <<= 1) {
#pragma unroll
            for (int h = 0; h < TPL; h++)
#pragma unroll
                for (int k = 0; k < TDIM; k++) o[h][k] += __shfl_xor_sync(kFull, o[h][k], off);
        }
        if (sub == 0) {
#pragma unroll
            for (int h = 0; h < TPL; h++) {
                if (!act[h]) continue;
                double *dst = a.trg_out + (size_t)tt[h] * TDIM;
                bool store = false;  // a part's own slot
                if constexpr (DIRECT) {
                    store = a.atomic_out == 0;
                    if (a.parts) dst = a.parts + ((size_t)w.e0 * a.ntrg + tt[h]) * TDIM;
                } else if constexpr (!MIXED) {
                    if (w.part >= 0) {
                        store = true;
                        dst = a.parts + (size_t)(w.part + tt[h] - w.t0) * TDIM;
                    }
                }
#pragma unroll
                for (int k = 0; k < TDIM; k++) {
                    const double val = K::SCALE * K::comp_scale(k) * o[h][k];
                    if (store)
                        dst[k] = val;
                    else if (DIRECT && a.atomic_out == 2)  // (in lists, unused, it cost kernels of 7 to 16
                                                           // components 2 to 3%)
                        atomicAdd(dst + k, val);
                    else
                        dst[k] += val;
                }
            }
        }
    }
}

// resident CTAs per SM of a kernel instance
template <int UK, bool MIXED, bool DIRECT> cudaError_t occupancy(int &n) {
    static int blocks_per_sm = 0;
    if (blocks_per_sm == 0) {
        int v = 0;
        const cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, list_p2p_kernel<UK, MIXED, DIRECT>,
                                                                              Cta<MIXED>::threads, 0);
        if (err != cudaSuccess) return err;
        blocks_per_sm = std::max(v, 1);
    }
    n = blocks_per_sm;
    return cudaSuccess;
}

template <int UK, bool MIXED, bool DIRECT>
cudaError_t launch_impl(const ListP2PArgs &a, int num_sms, cudaStream_t stream) {
    int blocks_per_sm = 1;
    cudaError_t err = occupancy<UK, MIXED, DIRECT>(blocks_per_sm);
    if (err != cudaSuccess) return err;
    constexpr int kWarpsPerCta = Cta<MIXED>::warps;
    long long want = ((long long)a.n_items + kWarpsPerCta - 1) / kWarpsPerCta;
    int grid = (int)std::max(1LL, std::min<long long>((long long)num_sms * blocks_per_sm, want));
    if ((!DIRECT || MIXED) && (err = cudaMemsetAsync(a.counter, 0, sizeof(unsigned int), stream)) != cudaSuccess) return err;
    list_p2p_kernel<UK, MIXED, DIRECT><<<grid, Cta<MIXED>::threads, 0, stream>>>(a);
    return cudaGetLastError();
}

// f(integral_constant<int, UK>) for the micro-kernel uk
template <int UK = 0, class F> cudaError_t with_uk(int uk, const F &f) {
    if constexpr (UK < UK_COUNT) {
        if (uk == UK) return f(std::integral_constant<int, UK>());
        return with_uk<UK + 1>(uk, f);
    } else {
        return cudaErrorInvalidValue;
    }
}

}  // namespace

// The instances of the kernel, in a translation unit per precision and form: the driver loads a unit's
// code at its first launch, and a program mostly uses one of them (all in one unit: 15 ms for the
// first launch of a process).
#define STK_P2P_UNIT(NAME, MIXED, DIRECT)                                                             \
    cudaError_t NAME(int uk, const ListP2PArgs &a, int num_sms, cudaStream_t stream) {                \
        return with_uk(uk, [&](auto id) {                                                             \
            return launch_impl<decltype(id)::value, MIXED, DIRECT>(a, num_sms, stream);               \
        });                                                                                           \
    }
cudaError_t list_p2p_fp64(int uk, const ListP2PArgs &a, int num_sms, cudaStream_t stream);
cudaError_t list_p2p_mixed(int uk, const ListP2PArgs &a, int num_sms, cudaStream_t stream);
cudaError_t direct_p2p_fp64(int uk, const ListP2PArgs &a, int num_sms, cudaStream_t stream);
cudaError_t direct_p2p_mixed(int uk, const ListP2PArgs &a, int num_sms, cudaStream_t stream);
// resident warps per SM of direct_p2p_fp64's kernel (CTAs of one warp)
cudaError_t direct_p2p_fp64_occupancy(int uk, int &n);

}  // namespace stk
