// stk_i8gemm.cu -- FP64 matrix products on the sm_100a int8 tensor cores (stk_i8gemm.cuh).
//
// Pipeline of one CTA (persistent: 128 x 128 output tiles in turn):
//   warp 0  producer: per K block (32 values) one bulk copy of the A block's digit planes
//           and one of the B block's into a 4-stage shared-memory ring;
//   warp 1  TMEM owner and MMA issuer: tcgen05.mma kind::i8, M = 128, K = 32, N the tile's
//           columns rounded up to 16 (partly filled M2L chunks hold 82 on average);
//   warps 2-17 drain: tcgen05.ld, the digit groups put together in int64, then FP64;
//   warps 18, 19 (gathered columns only) fetch B's rows in 16-byte asynchronous copies, two
//           stages in flight before a stage is handed on.
// The eight digit groups i + j = 0 .. 7 need 8 x 128 TMEM columns and there are 512, so a
// tile takes two passes over K: groups 0-3 (planes 0-3 of both operands, 10 products per K
// block) drained into an int64 per output, then groups 4-7 (all planes, 24 products).
// What bounds it (M = 636, N = 32768, K = 3584, B200): 1.58 ms, 95 TFLOP/s of FP64 work (cuBLAS:
// 29.9); tensor pipe active 80% of the time at 1.68 GHz (power), L2 6.2 TB/s.  By shared memory alone, the
// 34 MMAs of a K block read 8 KB each and the copies write 88 KB: 2800 clocks for 34 x 64 of MMA.
// 128 x 64 tiles (all groups resident, one pass) would read 6 KB per MMA of half the work; CTA
// pairs (256 x 128 tiles, 2110 clocks by the same count) measured 1.71 ms beside 1.55.
// Short K (M2L's P_d, 4 K blocks): the chain of the two passes, 18000 clocks a tile, 5900 of
// them MMA: the second pass's MMAs 6200, the drains 1800 and 6000, the wait for the first 2000;
// a third of the L2 traffic less (blocks kept for the second pass, used rows only) changed nothing.
// Every mbarrier wait has an iteration limit: on expiry the kernel records an error code,
// stops issuing work, waits (bounded) for what it issued, frees its TMEM and returns.
#include <algorithm>
#include <type_traits>

#include <cooperative_groups.h>

#include "stk_i8gemm.cuh"
#include "stk_umma_ptx.cuh"

namespace cg = cooperative_groups;

namespace stk {

namespace {

constexpr int kBM = kI8Rows, kBN = kI8Rows;
constexpr int kStages = 4;
constexpr int kStageBytes = 2 * kI8BlockBytes;  // A planes, then B planes
// 16 drain warps: 32 output columns each, so that the 64-bit sums of the first pass (64
// registers) fit beside the TMEM loads at 112 registers per thread
constexpr int kDrainWarps = 16;
constexpr int kDrainCols = kBN / (kDrainWarps / 4);
constexpr int kGatherWarps = 2;
template <class Job> constexpr int kThreads = 32 * (2 + kDrainWarps + (Job::kGather ? kGatherWarps : 0));
constexpr uint32_t kTmemCols = 512;
constexpr int kBarBytes = 2944;  // barriers, column scales
constexpr int kSmemBytes = kStages * kStageBytes + kBarBytes + 128 /* alignment */;
static_assert(kSmemBytes <= 232448, "shared memory of one CTA");

struct Bars {
    unsigned long long full[kStages], empty[kStages], accf, acce;
    uint32_t tmem;
    double col_scale[2][kBN / kDrainCols][kDrainCols];
    short col_rest[2][kBN / kDrainCols][kDrainCols];
    double ones[kDrainCols];
};
static_assert(sizeof(Bars) <= kBarBytes, "Bars fit their place");

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
                 : "memory");
}

// shared-memory matrix descriptor of one digit plane: K-major, no swizzle, core matrices of
// 8 rows x 16 bytes, 128 bytes apart along K, 256 bytes apart along the rows
__device__ __forceinline__ uint64_t plane_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)(128 >> 4) << 16;  // leading byte offset (along K)
    d |= (uint64_t)(256 >> 4) << 32;  // stride byte offset (row groups)
    d |= (uint64_t)1 << 46;           // version
    return d;
}

// instruction descriptor: D S32, A and B S8, both K-major, M = 128, N columns (a multiple of 16)
__device__ __forceinline__ uint32_t idesc_i8(int N) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(__cvta_generic_to_global(src)) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// this thread's shared-memory writes become visible to the tensor core's reads
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, int (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}

struct DenseJob {
    static constexpr bool kGather = false;
    int M, N, add, gm, gn, ntiles, seg_kb, nkb;  // K part p: blocks [p seg_kb, ...)
    bool m_fast;
    double *C;
    long long ldc, part_ld;  // elements between the parts' outputs
    const int *cols;
    struct Tile {
        int a_blk, b_blk, kb0, nkb, m_valid, n_valid, part;
    };
    __device__ Tile tile(int i) const {
        // neighbouring CTAs share the operand block of the slow index
        const int part = i / (gm * gn), j = i - part * gm * gn;
        const int m = m_fast ? j % gm : j / gn, n = m_fast ? j / gm : j % gn;
        const int kb0 = part * seg_kb;
        return {m, n, kb0, min(seg_kb, nkb - kb0), min(kBM, M - m * kBM), min(kBN, N - n * kBN), part};
    }
    // output column c0 of the tile, and column n from the running pointer of column n - 1
    __device__ double *first(const Tile &t, int c0) const {
        return C + t.part * part_ld + (cols ? 0 : (size_t)(t.b_blk * kBN + c0) * ldc) + t.a_blk * kBM;
    }
    __device__ double *at(double *p, const Tile &t, int n) const {
        return cols ? p + (size_t)cols[t.b_blk * kBN + n] * ldc : p;
    }
    __device__ long long step(const Tile &) const { return cols ? 0 : ldc; }
    __device__ int scale(const int *sb, const Tile &t, int n) const { return sb[t.b_blk * kBN + n]; }
};

template <bool GATHER> struct GroupJob {
    static constexpr bool kGather = GATHER;
    const I8Tile *tiles;
    int ntiles, add;
    double *C;
    const int *rows;  // gathered columns
    struct Tile {
        int a_blk, b_blk, kb0, nkb, m_valid, n_valid, ldc;
        double *c;
    };
    __device__ Tile tile(int i) const {
        const I8Tile &t = tiles[i];
        return {t.a_blk, t.b_blk, 0, t.nkb, t.m_valid, t.n_valid, t.ldc, C + t.c_off};
    }
    __device__ double *first(const Tile &t, int c0) const { return t.c + (size_t)c0 * t.ldc; }
    __device__ double *at(double *p, const Tile &, int) const { return p; }
    __device__ long long step(const Tile &t) const { return t.ldc; }
    __device__ int scale(const int *sb, const Tile &t, int n) const {
        const int c = t.b_blk * kBN + n;
        return sb[GATHER ? rows[c] : c];
    }
};

__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }  // normal range only

// A scale 2^e as a factor of up to 2^+-500, so that a sum of digit products (below 2^88) takes two
// of them without leaving the range of a double, and the exponent that is left (rare)
constexpr int kCoreExp = 500;
__device__ __forceinline__ double core_scale(int e) {
    return e == kI8NonFinite ? __longlong_as_double(0x7ff8000000000000ll) : pow2(min(max(e, -kCoreExp), kCoreExp));
}
__device__ __forceinline__ int rest_exp(int e) {
    return e == kI8NonFinite ? 0 : e - min(max(e, -kCoreExp), kCoreExp);
}
// v 2^r; a rest has the sign of its factor's exponent, so that v, which has been multiplied by both
// factors, is out of range only where v 2^r is
__device__ __forceinline__ double scale_rest(double v, int r) { return v * pow2(r >> 1) * pow2(r - (r >> 1)); }

template <class Job>
__global__ void __launch_bounds__(kThreads<Job>, 1)
    i8_gemm_kernel(const I8Operand A, const I8Operand B, const Job job, int *err) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = saddr(smem_raw);
    uint8_t *ring = smem_raw + ((128u - (raw & 127u)) & 127u);
    Bars *bars = reinterpret_cast<Bars *>(ring + kStages * kStageBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(saddr(&bars->full[s]), Job::kGather ? 1 + 32 * kGatherWarps : 1);
            mbar_init(saddr(&bars->empty[s]), 1);
        }
        mbar_init(saddr(&bars->accf), 1);
        mbar_init(saddr(&bars->acce), kDrainWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < kDrainCols) bars->ones[threadIdx.x] = 1.0;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&bars->tmem)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem;
    bool ok = true;

    if (warp == 0) {
        // ---- producer ----
        if (lane == 0) {
            unsigned g = 0;  // stages issued so far
            for (int t = blockIdx.x; t < job.ntiles && ok; t += gridDim.x) {
                const auto ts = job.tile(t);
                const uint8_t *pa = A.dig + ((size_t)ts.a_blk * A.nkb + ts.kb0) * kI8BlockBytes;
                const uint8_t *pb = B.dig + ((size_t)ts.b_blk * B.nkb + ts.kb0) * kI8BlockBytes;
                for (int k0 = 0; k0 < ts.nkb && ok; k0 += kI8MaxSegment) {
                    const int k1 = min(ts.nkb, k0 + kI8MaxSegment);
                    for (int pass = 0; pass < 2 && ok; pass++) {
                        const uint32_t bytes = (pass ? kI8Planes : 4) * kI8PlaneBytes;
                        for (int kb = k0; kb < k1; kb++, g++) {
                            const unsigned s = g % kStages;
                            if (!mbar_wait(saddr(&bars->empty[s]), ((g / kStages) & 1u) ^ 1u)) {
                                ok = false;
                                break;
                            }
                            const uint32_t fb = saddr(&bars->full[s]);
                            const uint32_t st = saddr(ring + s * kStageBytes);
                            mbar_expect_tx(fb, Job::kGather ? bytes : 2 * bytes);
                            bulk_load(st, pa + (size_t)kb * kI8BlockBytes, bytes, fb);
                            if constexpr (!Job::kGather)
                                bulk_load(st + kI8BlockBytes, pb + (size_t)kb * kI8BlockBytes, bytes, fb);
                        }
                    }
                }
            }
            if (!ok) {
                atomicExch(err, 11);
                // the copies already issued land before the CTA exits
                for (unsigned i = g > kStages ? g - kStages : 0; i < g; i++)
                    mbar_wait(saddr(&bars->full[i % kStages]), (i / kStages) & 1u);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer ----
        if (lane == 0) {
            unsigned g = 0, a = 0;  // stages consumed, accumulations started
            for (int t = blockIdx.x; t < job.ntiles && ok; t += gridDim.x) {
                const auto ts = job.tile(t);
                const int nkb = ts.nkb;
                const uint32_t idesc = idesc_i8((max(ts.n_valid, 1) + 15) & ~15);
                for (int k0 = 0; k0 < nkb && ok; k0 += kI8MaxSegment) {
                    const int n = min(nkb - k0, kI8MaxSegment);
                    for (int pass = 0; pass < 2 && ok; pass++, a++) {
                        if (!mbar_wait(saddr(&bars->acce), (a & 1u) ^ 1u)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        for (int kb = 0; kb < n; kb++, g++) {
                            const unsigned s = g % kStages;
                            if (!mbar_wait(saddr(&bars->full[s]), (g / kStages) & 1u)) {
                                ok = false;
                                break;
                            }
                            tc_fence_after();
                            const uint32_t st = saddr(ring + s * kStageBytes);
                            const uint64_t da = plane_desc(st), db = plane_desc(st + kI8BlockBytes);
                            constexpr uint64_t step = kI8PlaneBytes >> 4;
                            const uint32_t first = kb > 0 ? 1u : 0u;
                            if (pass == 0) {
#pragma unroll
                                for (int gr = 0; gr < 4; gr++)
#pragma unroll
                                    for (int i = 0; i <= gr; i++)
                                        mma_i8(tmem + gr * kBN, da + i * step, db + (gr - i) * step, idesc,
                                               i ? 1u : first);
                            } else {
#pragma unroll
                                for (int gr = 4; gr < 8; gr++)
#pragma unroll
                                    for (int i = gr > 6; i <= min(gr, 6); i++)
                                        mma_i8(tmem + (gr - 4) * kBN, da + i * step, db + (gr - i) * step, idesc,
                                               i > (gr > 6) ? 1u : first);
                            }
                            mma_commit(saddr(&bars->empty[s]));
                        }
                        mma_commit(saddr(&bars->accf));
                    }
                }
            }
            if (!ok) {
                atomicExch(err, 12);
                // one more commit tracks every MMA issued: complete before the TMEM is freed
                // (accf's phase count is then off, but no one waits for it any more than boundedly)
                mma_commit(saddr(&bars->accf));
                mbar_wait(saddr(&bars->accf), a & 1u);
            } else if (a > 0) {
                mbar_wait(saddr(&bars->accf), (a - 1) & 1u);
            }
        }
        __syncwarp();
    } else if (Job::kGather && warp >= 2 + kDrainWarps) {
        // ---- gathered columns ----
        if constexpr (Job::kGather) {
            // A copy instruction takes four 16-byte pieces of eight rows: the eight rows of a piece are
            // one core matrix, 128 bytes of shared memory without bank conflicts (the MMAs alone
            // read close to what it can give).  A thread keeps the numbers of its 16 rows of the
            // tile, so that a copy is an address and an instruction.
            constexpr int kTurns = kBN / 8;
            static_assert(kGatherWarps == 2 && kI8Planes == 7, "14 pieces: 4 + 4 of planes 0-3, 3 + 3 of the others");
            const int w = warp - 2 - kDrainWarps, r = lane & 7, q = lane >> 3;
            const int j = 4 * w + q, j2 = 8 + 3 * w + q;
            auto place = [&](int piece) {
                return (uint32_t)(kI8BlockBytes + (piece >> 1) * kI8PlaneBytes + (piece & 1) * 128 + r * 16);
            };
            const uint32_t d = place(j), d2 = place(j2);
            unsigned g = 0;
            const size_t pitch = (size_t)B.nkb * (kI8Planes * kI8K);
            for (int t = blockIdx.x; t < job.ntiles && ok; t += gridDim.x) {
                const auto ts = job.tile(t);
                const int turns = (ts.n_valid - r + 7) >> 3;
                int row[kTurns];
#pragma unroll
                for (int i = 0; i < kTurns; i++) row[i] = i < turns ? job.rows[ts.b_blk * kBN + r + 8 * i] : 0;
                for (int k0 = 0; k0 < ts.nkb && ok; k0 += kI8MaxSegment) {
                    const int k1 = min(ts.nkb, k0 + kI8MaxSegment);
                    for (int pass = 0; pass < 2 && ok; pass++)
                        for (int kb = k0; kb < k1; kb++, g++) {
                            const unsigned s = g % kStages;
                            if (!__all_sync(0xffffffffu, mbar_wait(saddr(&bars->empty[s]), ((g / kStages) & 1u) ^ 1u))) {
                                ok = false;
                                break;
                            }
                            const uint32_t st = saddr(ring + s * kStageBytes);
                            const uint8_t *src = B.dig + (size_t)kb * (kI8Planes * kI8K);
#pragma unroll
                            for (int i = 0; i < kTurns; i++)
                                if (i < turns) cp_async16(st + d + i * 256, src + row[i] * pitch + j * 16);
                            if (pass == 1 && q < 3) {
#pragma unroll
                                for (int i = 0; i < kTurns; i++)
                                    if (i < turns) cp_async16(st + d2 + i * 256, src + row[i] * pitch + j2 * 16);
                            }
                            cp_async_commit();
                            if (g >= 2) {  // the stage issued two before has landed
                                cp_async_wait<2>();
                                fence_async_smem();
                                mbar_arrive(saddr(&bars->full[(g - 2) % kStages]));
                            }
                        }
                }
                if (!ok) break;
            }
            cp_async_wait<0>();
            fence_async_smem();
            for (unsigned i = g > 2 ? g - 2 : 0; i < g; i++) mbar_arrive(saddr(&bars->full[i % kStages]));
            if (!ok && lane == 0) atomicExch(err, 14);
        }
        __syncwarp();
    } else {
        // ---- drain: warp w reads TMEM lanes 32 (w % 4) .. + 31, columns kDrainCols ((w - 2) / 4) .. ----
        const int q = warp & 3, c0 = ((warp - 2) >> 2) * kDrainCols;
        const int row = q * 32 + lane;
        const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
        unsigned a = 0;  // accumulations drained so far
        int buf = 0;
        // scales of this thread's row and of column c0 + lane of a tile, read a tile ahead (read at
        // the tile's start they took 3000 clocks, two dependent L2 latencies and a third for gathered
        // columns; read per column inside the drain, its length again)
        int ea = 0, eb = 0;
        static_assert(kDrainCols == 32, "a lane per column");
        auto read_scales = [&](int t) {
            if (t >= job.ntiles) return;
            const auto ts = job.tile(t);
            ea = row < ts.m_valid ? A.scale[ts.a_blk * kBM + row] : 0;
            eb = c0 + lane < ts.n_valid ? job.scale(B.scale, ts, c0 + lane) : 0;
        };
        read_scales(blockIdx.x);
        for (int t = blockIdx.x; t < job.ntiles && ok; t += gridDim.x) {
            const int nkb = job.tile(t).nkb;
            const double sr = core_scale(ea);
            // the four warps of these columns write the same values, and none is two tiles ahead
            double *sn = bars->col_scale[buf][c0 / kDrainCols];
            buf ^= 1;
            sn[lane] = core_scale(eb);
            bars->col_rest[buf ^ 1][c0 / kDrainCols][lane] = (short)rest_exp(eb);
            const bool wide = __any_sync(0xffffffffu, rest_exp(ea) | rest_exp(eb));
            __syncwarp();
            for (int k0 = 0; k0 < nkb && ok; k0 += kI8MaxSegment) {
                const bool add = job.add || k0 > 0;
                // groups 0-3: hi = sum_g acc_g 256^(3 - g)
                if (!__all_sync(0xffffffffu, mbar_wait(saddr(&bars->accf), a & 1u))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                long long hi[kDrainCols];
#pragma unroll
                for (int c = 0; c < kDrainCols; c += 8) {
                    int g0[8], g1[8], g2[8], g3[8];
                    tmem_ld8(tb + c, g0);
                    tmem_ld8(tb + kBN + c, g1);
                    tmem_ld8(tb + 2 * kBN + c, g2);
                    tmem_ld8(tb + 3 * kBN + c, g3);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        hi[c + j] = (long long)g0[j] * (1 << 24) + (long long)g1[j] * (1 << 16) +
                                    (long long)g2[j] * (1 << 8) + (long long)g3[j];
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(saddr(&bars->acce));
                a++;
                if (k0 + kI8MaxSegment >= nkb) read_scales(t + gridDim.x);
                // groups 4-7: lo = sum_g acc_g 256^(7 - g); value = hi 2^32 + lo
                if (!__all_sync(0xffffffffu, mbar_wait(saddr(&bars->accf), a & 1u))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                // first all values, so that the next tile's MMAs run while these are scaled and stored
#pragma unroll
                for (int c = 0; c < kDrainCols; c += 4) {
                    int g4[4], g5[4], g6[4], g7[4];
                    tmem_ld4(tb + c, g4);
                    tmem_ld4(tb + kBN + c, g5);
                    tmem_ld4(tb + 2 * kBN + c, g6);
                    tmem_ld4(tb + 3 * kBN + c, g7);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const long long lo = (long long)g4[j] * (1 << 24) + (long long)g5[j] * (1 << 16) +
                                             (long long)g6[j] * (1 << 8) + (long long)g7[j];
                        hi[c + j] = __double_as_longlong(fma((double)hi[c + j], 4294967296.0, (double)lo));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(saddr(&bars->acce));
                a++;
                asm volatile("" ::: "memory");  // the tile is read again: kept, it would spill
                const auto ts = job.tile(t);
                double *pc = job.first(ts, c0) + row;
                const long long step = job.step(ts);
                const double *fn = sn;
                double fr = sr;
                if (wide) {
                    // scales at the ends of the range (rare): all of it here, so that the stores below
                    // stay as they are (a predicate in them cost 4 to 12 % of a short product)
                    const short *rn = bars->col_rest[buf ^ 1][c0 / kDrainCols];
                    const int ra = row < ts.m_valid ? rest_exp(A.scale[ts.a_blk * kBM + row]) : 0;
#pragma unroll
                    for (int c = 0; c < kDrainCols; c++) {
                        hi[c] = __double_as_longlong(scale_rest(__longlong_as_double(hi[c]) * sn[c] * sr, ra + rn[c]));
                        asm volatile("" ::: "memory");
                    }
                    fn = bars->ones;
                    fr = 1.0;
                }
#pragma unroll
                for (int c = 0; c < kDrainCols; c++) {
                    // four columns at a time: pointers and scales of all 32 at once would spill
                    if (c % 4 == 0) asm volatile("" : "+l"(pc)::"memory");
                    if (row < ts.m_valid && c0 + c < ts.n_valid) {
                        double *p = job.at(pc, ts, c0 + c);
                        const double v = __longlong_as_double(hi[c]) * fn[c] * fr;
                        *p = add ? *p + v : v;
                    }
                    pc += step;
                }
            }
        }
        if (!ok && lane == 0) atomicExch(err, 13);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// ---- FP64 rows -> digit blocks ---------------------------------------------------
// Source of four consecutive K values of a row (values beyond K are zero) and their exponents.
struct RowLoad {
    const double *src;
    long long ld;
    const int *idx;
    int K;
    const int *ks;
    const int *kof, *kset, *nof;  // per 128-row block, or null
    int kld;
    const double *rmul;
    __device__ int mul(long long r) const { return rmul ? ((__double2hiint(rmul[r]) >> 20) & 0x7ff) - 1023 : 0; }
    __device__ int used_blocks(long long blk, int nkb) const { return kof ? (kof[blk] + kI8K - 1) / kI8K : nkb; }
    __device__ int len(long long r) const {
        return kof ? (r % kI8Rows < nof[r / kI8Rows] ? kof[r / kI8Rows] : 0) : K;
    }
    __device__ void load4(long long r, int k, int n, double (&v)[4], int (&e)[4]) const {
        const long long i = idx ? idx[r] : r;
        const int *f = ks && kset ? ks + (size_t)kset[r / kI8Rows] * kld : ks;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = i >= 0 && k + q < n ? src[i * ld + k + q] : 0.0;
            e[q] = f && k + q < n ? f[k + q] : 0;
        }
    }
};
struct GatherLoad {
    I8Gather g;
    __device__ int mul(long long) const { return 0; }
    __device__ int used_blocks(long long blk, int) const { return (g.K[(blk * kI8Rows) >> g.lg] + kI8K - 1) / kI8K; }
    __device__ int len(long long r) const { return g.K[r >> g.lg]; }
    __device__ void load4(long long r, int k, int n, double (&v)[4], int (&e)[4]) const {
        const int c = (int)(r >> g.lg);
        const int *t = g.tab + g.tab_off[c] + (r & ((1ll << g.lg) - 1)) * g.nq[c];
        // the tables are padded to multiples of 4
        const int4 q4 = *reinterpret_cast<const int4 *>(g.rowq + g.row_off[c] + k);
        const int4 s4 = *reinterpret_cast<const int4 *>(g.srow + g.row_off[c] + k);
        const int4 e4 = *reinterpret_cast<const int4 *>(g.kexp + g.row_off[c] + k);
        const int rq[4] = {q4.x, q4.y, q4.z, q4.w}, sr[4] = {s4.x, s4.y, s4.z, s4.w};
        e[0] = e4.x, e[1] = e4.y, e[2] = e4.z, e[3] = e4.w;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = 0.0;
            if (k + q < n) {
                const int pos = t[rq[q]];
                if (pos >= 0) v[q] = g.z[(size_t)pos * g.ldz + sr[q]];
            }
        }
    }
};

// Magnitude of x 2^ke (|ke| <= kI8KExp) in an order-preserving integer: exponent and six leading
// fraction bits of x, the exponent shifted by ke and made positive; 0 for zero, kMagNonFinite
// for an infinity or NaN.  (x 2^ke itself may leave the range of a double.)
constexpr unsigned kMagNonFinite = 0x7fffffffu;
constexpr int kMagBias = 2048;
__device__ __forceinline__ unsigned mag(double x, int ke) {
    const unsigned t = ((unsigned)__double2hiint(x) & 0x7fffffffu) >> 14;  // exponent, 6 bits
    if (t >= 0x7ffu << 6) return kMagNonFinite;
    return x == 0.0 ? 0u : max(t, 1u << 6) + ((unsigned)(ke + kMagBias) << 6);
}

// the exponent that takes a row's values, below 127/128 2^e, to integers below 127 2^48, whose
// top digit is at most 127, and the stored scale's exponent
struct RowScale {
    int up, s;
    bool finite;
};
__device__ __forceinline__ RowScale row_scale(unsigned m) {
    if (m == kMagNonFinite) return {0, kI8NonFinite, false};
    if (m == 0) return {0, 0, true};
    const int e = (int)(m >> 6) - kMagBias - 1022 + ((m & 0x3f) == 0x3f);  // |x| < 127/128 2^e
    return {55 - e, e - 35, true};
}

// seven balanced base-256 digits of x 2^t, |x 2^t| < 127 2^48, as the bytes of a' + 128 (256^7 - 1)
// / 255, each with its top bit flipped (digit = byte - 128); byte 6 is the most significant.
// t = f + ke + rest, f + ke within +-1000: the first factor takes x to where rest (zero but at the
// ends of the range) can neither over- nor underflow what the digits hold.
__device__ __forceinline__ unsigned long long digits(double x, int e, int rest) {
    double y = x * pow2(e);
    if (rest) y *= pow2(rest);
    const long long v = __double2ll_rn(y);
    return (unsigned long long)(v + 0x0080808080808080ll) ^ 0x0080808080808080ull;
}

// A cluster of CTAs per 8 rows (one row group of the block layout), each a slice of K, one
// warp per row: the row's largest magnitude (over the cluster through distributed shared
// memory), then 128 values at a time into a shared tile that is written out as whole 128-byte
// core matrices (blocks) or 224-byte pieces (rows).  Bound by memory: 8 bytes read (twice, the
// second time from L1 / L2) and 7 written per value.  The slices matter where rows are few and
// long: 512 rows of 15616 values took 191 us as 64 CTAs.
template <class Load, bool ROWS>
__global__ void __launch_bounds__(256) i8_digits_kernel(const __grid_constant__ Load ld, long long rows, long long groups,
                                                        int nkb, int slice, uint8_t *__restrict__ dig,
                                                        int *__restrict__ scale) {
    // [plane][16-value core][row][16 bytes], cores padded by one row against bank conflicts
    constexpr int kCore = 9 * 16;
    __shared__ __align__(16) uint8_t tile[kI8Planes][8][kCore];
    __shared__ unsigned part[8];  // this CTA's largest magnitudes
    cg::cluster_group cluster = cg::this_cluster();
    const int nsl = (int)cluster.num_blocks(), sl = (int)cluster.block_rank();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ka = sl * slice;
    for (long long grp = blockIdx.x / nsl; grp < groups; grp += gridDim.x / nsl) {
        const long long r = grp * 8 + w;
        const int n = r < rows ? min(ld.len(r), nkb * kI8K) : 0;
        // the row block's K blocks in use (the whole pitch, or fewer where K goes by blocks)
        const int kz = min(min(nkb, ld.used_blocks(grp / 16, nkb)) * kI8K, ka + slice);
        unsigned m = 0;
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        int e[4] = {0, 0, 0, 0};
        for (int k = ka + 4 * lane; k < min(n, kz); k += 128) {
            ld.load4(r, k, n, v, e);
#pragma unroll
            for (int q = 0; q < 4; q++) m = max(m, mag(v[q], e[q]));
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (nsl > 1) {
            if (lane == 0) part[w] = m;
            cluster.sync();
            for (int i = 0; i < nsl; i++) m = max(m, cluster.map_shared_rank(part, i)[w]);
            cluster.sync();  // everyone has read part before the next group writes it
        }
        const RowScale sc = row_scale(m);
        if (lane == 0 && sl == 0 && (!ROWS || r < rows)) scale[r] = r < rows ? sc.s + (sc.finite ? ld.mul(r) : 0) : 0;
        const int up = min(max(sc.up, -900), 900), rest = sc.up - up;
        uint8_t *blk = dig + (size_t)(grp / 16) * nkb * kI8BlockBytes + (size_t)(grp % 16) * 256;
        for (int k0 = ka; k0 < kz; k0 += 128) {
            if (kz - ka > 128 || !sc.finite) {  // one turn: still in registers
#pragma unroll
                for (int q = 0; q < 4; q++) v[q] = 0.0, e[q] = 0;
                if (sc.finite && k0 + 4 * lane < n) ld.load4(r, k0 + 4 * lane, n, v, e);
            }
            unsigned lo[4], hi[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const unsigned long long d = digits(v[q], up + e[q], rest);
                lo[q] = (unsigned)d;
                hi[q] = (unsigned)(d >> 32);
            }
#pragma unroll
            for (int p = 0; p < kI8Planes; p++) {
                const int b = 6 - p;  // byte of this plane
                const unsigned sel = (b & 3) | ((b & 3) + 4) << 4;
                const unsigned *x = b < 4 ? lo : hi;
                const unsigned v01 = __byte_perm(x[0], x[1], sel), v23 = __byte_perm(x[2], x[3], sel);
                *reinterpret_cast<unsigned *>(&tile[p][lane >> 2][w * 16 + (lane & 3) * 4]) =
                    __byte_perm(v01, v23, 0x5410);
            }
            __syncthreads();
            for (int u = threadIdx.x; u < kI8Planes * 64; u += 256) {
                int p, c, row;
                uint8_t *dst;
                if constexpr (ROWS) {
                    // (row, K block, plane, half): 14 pieces of 16 bytes in a run
                    row = u / 56;
                    const int i = u - row * 56, kq = i / 14, j = i - kq * 14;
                    p = j >> 1;
                    c = 2 * kq + (j & 1);
                    dst = dig + (((size_t)(grp * 8 + row) * nkb + (k0 >> 5) + kq) * kI8Planes + p) * kI8K + (c & 1) * 16;
                    if (grp * 8 + row >= rows) continue;
                } else {
                    p = u >> 6, c = (u >> 3) & 7, row = u & 7;
                    dst = blk + (size_t)((k0 >> 5) + (c >> 1)) * kI8BlockBytes + p * kI8PlaneBytes + (c & 1) * 128 + row * 16;
                }
                if ((k0 >> 5) * kI8K + (c >> 1) * kI8K < kz)
                    *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(&tile[p][c][row * 16]);
            }
            __syncthreads();
        }
    }
}

// The transpose, x(r, k) = src[k ld + r]: one CTA per 8 rows again; the eight rows of one k
// are 64 contiguous bytes.  Operators only, once per tree set-up.
struct TransLoad {
    const double *src;
    long long ld;
    int K;
    const int *ks;
    __device__ int mul(long long) const { return 0; }
    __device__ int used_blocks(long long, int nkb) const { return nkb; }
    __device__ int len(long long) const { return K; }
    __device__ void load4(long long r, int k, int n, double (&v)[4], int (&e)[4]) const {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = k + q < n ? src[(k + q) * ld + r] : 0.0;
            e[q] = ks && k + q < n ? ks[k + q] : 0;
        }
    }
};

// 2^up > the magnitude m (0 for zero or a non-finite one), down = -up
__device__ __forceinline__ void k_scale(unsigned m, int &up, int &down) {
    const int e = m == 0 || m == kMagNonFinite ? 0 : (int)(m >> 6) - kMagBias - 1022;
    up = min(max(e, -kI8KExp), kI8KExp);
    down = -up;
}

__global__ void __launch_bounds__(256) column_scales_kernel(const double *__restrict__ src, long long ld, long long rows,
                                                            int K, int *__restrict__ up, int *__restrict__ down) {
    __shared__ unsigned red[8];
    for (int k = blockIdx.x; k < K; k += gridDim.x) {
        unsigned m = 0;
        for (long long r = threadIdx.x; r < rows; r += 256) m = max(m, mag(src[(size_t)k * ld + r], 0));
        m = __reduce_max_sync(0xffffffffu, m);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int i = 1; i < 8; i++) m = max(m, red[i]);
            k_scale(m, up[k], down[k]);
        }
        __syncthreads();
    }
}

__global__ void row_mag_kernel(const double *__restrict__ src, long long ld, long long rows, int K,
                               unsigned *__restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    unsigned m = 0;
    for (long long r = blockIdx.y; r < rows; r += gridDim.y) m = max(m, mag(src[r * ld + k], 0));
    atomicMax(out + k, m);
}

__global__ void row_scales_kernel(const unsigned *__restrict__ m, int K, int *__restrict__ up, int *__restrict__ down) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < K) k_scale(m[k], up[k], down[k]);
}

template <bool ROWS = false, class Load>
cudaError_t launch_digits(const Load &ld, long long rows, int nkb, uint8_t *dig, int *scale, cudaStream_t s) {
    if (rows <= 0 || nkb <= 0) return cudaSuccess;
    const long long groups = (ROWS ? rows + 7 : i8_pad_rows(rows)) / 8;
    // slices of at least 512 values until ~4 CTAs per SM run
    int nsl = 1;
    while (nsl < 8 && groups * nsl < 148 * 4 && nkb * kI8K >= 1024 * nsl) nsl *= 2;
    const int slice = ((nkb * kI8K + nsl - 1) / nsl + 127) / 128 * 128;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(std::min<long long>(groups, 148 * 64) * nsl));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)nsl, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, i8_digits_kernel<Load, ROWS>, ld, rows, groups, nkb, slice, dig, scale);
}

// C[m + ldc col(n)] (=|+=) the parts' sum, in order
__global__ void sum_parts_kernel(const double *__restrict__ parts, int np, int M, int N, int add,
                                 const int *__restrict__ cols, double *__restrict__ C, long long ldc) {
    const long long total = (long long)M * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int n = (int)(i / M), m = (int)(i - (long long)n * M);
        double v = parts[i];
        for (int p = 1; p < np; p++) v += parts[i + p * total];
        double *c = C + (size_t)(cols ? cols[n] : n) * ldc + m;
        *c = add ? *c + v : v;
    }
}

int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return n > 0 ? n : 1;
}

template <class Job> cudaError_t launch_gemm(const I8Operand &A, const I8Operand &B, const Job &job, int *err, cudaStream_t s) {
    // for the current device
    const cudaError_t e = cudaFuncSetAttribute(i8_gemm_kernel<Job>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    i8_gemm_kernel<Job><<<std::min(job.ntiles, sm_count()), kThreads<Job>, kSmemBytes, s>>>(A, B, job, err);
    return cudaGetLastError();
}

bool operand_ok(const I8Operand &o) {
    return o.dig && o.scale && o.nkb > 0 && (reinterpret_cast<uintptr_t>(o.dig) & 15u) == 0;
}

}  // namespace

cudaError_t i8_column_scales(const double *src, long long ld, long long rows, int K, int *up, int *down,
                             cudaStream_t s) {
    if (K <= 0) return cudaSuccess;
    column_scales_kernel<<<std::min(K, 148 * 8), 256, 0, s>>>(src, ld, rows, K, up, down);
    return cudaGetLastError();
}
cudaError_t i8_row_scales(const double *src, long long ld, long long rows, int K, unsigned *mag, int *up, int *down,
                          cudaStream_t s) {
    if (K <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(mag, 0, sizeof(unsigned) * K, s);
    if (e != cudaSuccess) return e;
    const dim3 grid((K + 255) / 256, (unsigned)std::max<long long>(1, std::min<long long>(rows, 512)));
    row_mag_kernel<<<grid, 256, 0, s>>>(src, ld, rows, K, mag);
    row_scales_kernel<<<(K + 255) / 256, 256, 0, s>>>(mag, K, up, down);
    return cudaGetLastError();
}
cudaError_t i8_digits(const double *src, long long ld, const int *idx, long long rows, int K, int nkb, const int *kexp,
                      const double *rmul, uint8_t *dig, int *scale, cudaStream_t s) {
    return launch_digits(RowLoad{src, ld, idx, K, kexp, nullptr, nullptr, nullptr, 0, rmul}, rows, nkb, dig, scale, s);
}
cudaError_t i8_digits_rows(const double *src, long long ld, long long rows, int K, int nkb, const int *kexp,
                           uint8_t *dig, int *scale, cudaStream_t s) {
    return launch_digits<true>(RowLoad{src, ld, nullptr, K, kexp, nullptr, nullptr, nullptr, 0, nullptr}, rows, nkb, dig, scale, s);
}
cudaError_t i8_digits_blocks(const double *src, long long ld, long long rows, const int *kof, const int *nof, int nkb,
                             const int *kexp, const int *kset, int kld, uint8_t *dig, int *scale, cudaStream_t s) {
    return launch_digits(RowLoad{src, ld, nullptr, 0, kexp, kof, kset, nof, kld, nullptr}, rows, nkb, dig, scale, s);
}
cudaError_t i8_digits_trans(const double *src, long long ld, long long rows, int K, int nkb, const int *kexp,
                            uint8_t *dig, int *scale, cudaStream_t s) {
    return launch_digits(TransLoad{src, ld, K, kexp}, rows, nkb, dig, scale, s);
}
cudaError_t i8_digits_gather(const I8Gather &g, int nkb, uint8_t *dig, int *scale, cudaStream_t s) {
    return launch_digits(GatherLoad{g}, 8ll << g.lg, nkb, dig, scale, s);
}

// K parts of a product with fewer tiles than half the SMs: as many as keep every part at
// least 16 K blocks long (~23 us against ~3 us for its drain and ~1 us per part of the sum)
int i8_gemm_parts(long long M, long long N, int nkb) {
    const long long nt = ((M + kBM - 1) / kBM) * ((N + kBN - 1) / kBN);
    if (nt > 74) return 1;
    return (int)std::max<long long>(1, std::min<long long>(148 / nt, nkb / 16));
}

cudaError_t i8_gemm(int M, int N, I8Operand A, I8Operand B, int add, double *C, long long ldc, const int *cols,
                    double *parts, int *err, cudaStream_t s) {
    if (M <= 0 || N <= 0) return cudaSuccess;
    if (!operand_ok(A) || !operand_ok(B) || A.nkb != B.nkb || !C || !err || ldc < M) return cudaErrorInvalidValue;
    const int gm = (M + kBM - 1) / kBM, gn = (N + kBN - 1) / kBN;
    int np = parts ? i8_gemm_parts(M, N, A.nkb) : 1;
    const int seg = (A.nkb + np - 1) / np;
    np = (A.nkb + seg - 1) / seg;
    const long long nt = (long long)gm * gn * np;
    if (nt > 0x7fffffff) return cudaErrorInvalidValue;
    // the operand with fewer blocks is walked fastest: it stays in L2 while the other streams
    DenseJob job{M, N, add, gm, gn, (int)nt, seg, A.nkb, gm <= gn, C, ldc, 0, cols};
    if (np > 1) {
        job.add = 0;
        job.C = parts;
        job.ldc = M;
        job.part_ld = (long long)M * N;
        job.cols = nullptr;
    }
    const cudaError_t e = launch_gemm(A, B, job, err, s);
    if (e != cudaSuccess || np == 1) return e;
    const int grid = (int)std::min<long long>(((long long)M * N + 255) / 256, 148 * 16);
    sum_parts_kernel<<<grid, 256, 0, s>>>(parts, np, M, N, add, cols, C, ldc);
    return cudaGetLastError();
}

cudaError_t i8_grouped(I8Operand A, I8Operand B, const I8Tile *tiles, int ntiles, int add, double *C, int *err,
                       cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    if (!operand_ok(A) || !operand_ok(B) || !tiles || !C || !err) return cudaErrorInvalidValue;
    return launch_gemm(A, B, GroupJob<false>{tiles, ntiles, add, C, nullptr}, err, s);
}

cudaError_t i8_grouped_gather(I8Operand A, I8Rows B, const int *rows, const I8Tile *tiles, int ntiles, int add, double *C,
                              int *err, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    const I8Operand b{B.dig, B.scale, B.nkb};
    if (!operand_ok(A) || !operand_ok(b) || !rows || !tiles || !C || !err) return cudaErrorInvalidValue;
    return launch_gemm(A, b, GroupJob<true>{tiles, ntiles, add, C, rows}, err, s);
}

}  // namespace stk
