// stk_p2p.cu -- P2P launches, source records and the sums of split sources (the kernel:
// stk_p2p_kernel.cuh).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "stk_p2p_kernel.cuh"
#include "stk_ukernels.cuh"

namespace stk {

namespace {

// trg_out += the parts of targets whose sources were split over items: blockIdx.y takes columns of
// the groups blockIdx.x, ....  Groups of many parts (a leaf with a long list: hundreds) are summed
// in eight runs of parts side by side, 32 columns per CTA, the runs' sums then in order: as one
// chain of all parts per thread, the longest groups took 140 us of a 131k-point wall evaluation.
// The order depends on the lists alone, so repeats give the same bits.
constexpr int kPartThreads = 256, kPartRuns = 8, kPartWide = kPartThreads / kPartRuns;

__global__ void __launch_bounds__(kPartThreads)
    add_parts_kernel(const PartGroup *__restrict__ groups, int n, int d, const double *__restrict__ parts,
                     double *__restrict__ out) {
    __shared__ double red[kPartRuns][kPartWide];
    const int run = threadIdx.x / kPartWide, jj = threadIdx.x - run * kPartWide;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const PartGroup g = groups[i];
        const int m = g.nt * d;
        const double *p = parts + (size_t)g.part0 * d;
        double *o = out + (size_t)g.t0 * d;
        if (g.n_parts <= 2 * kPartRuns) {
            const int j = blockIdx.y * kPartThreads + threadIdx.x;
            if (j < m) {
                double v = 0.0;
#pragma unroll 4
                for (int k = 0; k < g.n_parts; k++) v += p[(size_t)k * m + j];
                o[j] += v;
            }
            continue;
        }
        const int j = blockIdx.y * kPartWide + jj;
        if (blockIdx.y * kPartWide >= m) continue;
        const int k0 = (int)((long long)g.n_parts * run / kPartRuns), k1 = (int)((long long)g.n_parts * (run + 1) / kPartRuns);
        double v = 0.0;
        if (j < m) {
#pragma unroll 8
            for (int k = k0; k < k1; k++) v += p[(size_t)k * m + j];
        }
        red[run][jj] = v;
        __syncthreads();
        if (run == 0 && j < m) {
            double t = 0.0;
#pragma unroll
            for (int r = 0; r < kPartRuns; r++) t += red[r][jj];
            o[j] += t;
        }
        __syncthreads();
    }
}

// out[i] (=|+=) the chunks' sums, in order
__global__ void sum_chunks_kernel(const double *__restrict__ parts, int n_chunk, long long n, int add,
                                  double *__restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double v = parts[i];
#pragma unroll 8
        for (int k = 1; k < n_chunk; k++) v += parts[k * n + i];
        out[i] = add ? out[i] + v : v;
    }
}

// a record's values from its source's: staged or as they are, zeros behind
template <int UK> __device__ __forceinline__ void record_values(const double (&f)[Uk<UK>::SDIM], double (&r)[Rec<UK>::RS]) {
    using K = Uk<UK>;
    constexpr int n = Rec<UK>::kStaged ? K::NV : K::SDIM;
    double v[n];
    if constexpr (Rec<UK>::kStaged) {
        K::stage(f, v);
    } else {
#pragma unroll
        for (int k = 0; k < n; k++) v[k] = f[k];
    }
#pragma unroll
    for (int k = 3; k < Rec<UK>::RS; k++) r[k] = k - 3 < n ? v[k - 3 < n ? k - 3 : 0] : 0.0;
}

// One thread per source: its values staged once here instead of in every tile that reads it
// (Rec<>::kStaged).
template <int UK>
__global__ void pack_records_kernel(int n, const int *__restrict__ perm, const double *__restrict__ xyz,
                                    const double *__restrict__ v1, int d1, const double *__restrict__ v2,
                                    double *__restrict__ rec) {
    using K = Uk<UK>;
    constexpr int RS = Rec<UK>::RS;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = perm ? perm[i] : i;
        double f[K::SDIM], r[RS];
#pragma unroll
        for (int k = 0; k < K::SDIM; k++)
            f[k] = k < d1 ? v1[(size_t)p * d1 + k] : v2[(size_t)p * (K::SDIM - d1) + k - d1];
        record_values<UK>(f, r);
#pragma unroll
        for (int k = 0; k < 3; k++) r[k] = xyz[3 * (size_t)i + k];
        double2 *o = reinterpret_cast<double2 *>(rec + (size_t)i * RS);
#pragma unroll
        for (int k = 0; k < RS / 2; k++) o[k] = make_double2(r[2 * k], r[2 * k + 1]);
    }
}

struct DensExp {
    double v[4];
};

template <int UK>
__global__ void pack_surface_kernel(const int *__restrict__ nodes, int m, int n, const double *__restrict__ xyz,
                                    const double *__restrict__ dens, const int *__restrict__ level, DensExp e,
                                    double *__restrict__ rec) {
    using K = Uk<UK>;
    constexpr int RS = Rec<UK>::RS;
    const long long total = (long long)m * n;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(idx / n), j = (int)(idx - (long long)i * n), b = nodes[i];
        const size_t p = (size_t)b * n + j;
        double f[K::SDIM], r[RS];
#pragma unroll
        for (int k = 0; k < K::SDIM; k++) f[k] = dens[p * K::SDIM + k];
        if (level) {
#pragma unroll
            for (int k = 0; k < K::SDIM; k++)
                if (e.v[k & 3] != 0.0) f[k] *= exp2(-(double)level[b] * e.v[k & 3]);
        }
        record_values<UK>(f, r);
#pragma unroll
        for (int k = 0; k < 3; k++) r[k] = xyz[3 * p + k];
        double2 *o = reinterpret_cast<double2 *>(rec + p * RS);
#pragma unroll
        for (int k = 0; k < RS / 2; k++) o[k] = make_double2(r[2 * k], r[2 * k + 1]);
    }
}

__global__ void scatter_add_kernel(int n, int d, const int *__restrict__ perm, const double *__restrict__ in,
                                   const double *__restrict__ alpha, double *__restrict__ out) {
    const long long total = (long long)n * d;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(idx / d);
        const int k = (int)(idx - (long long)i * d);
        const int p = perm ? perm[i] : i;
        out[(size_t)p * d + k] += (alpha ? alpha[k] : 1.0) * in[idx];
    }
}

}  // namespace

int uk_sdim_host(int uk) { return uk_sdim(uk); }
int uk_tdim_host(int uk) { return uk_tdim(uk); }
int uk_tvdim_host(int uk) { return uk_tvdim(uk); }
double uk_scale_host(int uk) { return uk_scale(uk); }
int uk_record_stride(int uk) {
    int rs = 0;
    with_uk(uk, [&](auto id) {
        rs = Rec<decltype(id)::value>::RS;
        return cudaSuccess;
    });
    return rs;
}

cudaError_t launch_list_p2p(int uk, int prec, const ListP2PArgs &a, int num_sms, cudaStream_t stream) {
    if (a.n_items <= 0) return cudaSuccess;
    if (uk >= 0 && uk < UK_COUNT && uk_tvdim(uk) > 0 && !a.trg_aux) return cudaErrorInvalidValue;
    if (a.atomic_out != 0 || (a.n_groups > 0 && (!a.groups || !a.parts))) return cudaErrorInvalidValue;
    const cudaError_t e = prec == PREC_MIXED ? list_p2p_mixed(uk, a, num_sms, stream) : list_p2p_fp64(uk, a, num_sms, stream);
    if (e != cudaSuccess || a.n_groups == 0) return e;
    const int d = uk_tdim(uk);
    add_parts_kernel<<<dim3(std::min(a.n_groups, 148 * 8), (64 * d + kPartWide - 1) / kPartWide), kPartThreads, 0, stream>>>(a.groups, a.n_groups, d, a.parts,
                                                                         a.trg_out);
    return cudaGetLastError();
}

// FP64: chunks so that the equal items fill whole turns of the resident warps.  An item costs
// its sources plus ~40 more (first tile's latency, output), so many short items only pay where
// the targets alone leave warps idle: 300 x 400 points run as 65 items of 32 sources.
// Mixed: at least 256 sources per item, as its Kahan sums are formed per item.
void direct_chunks(int uk, int prec, int ntrg, int nsrc, int num_sms, int &chunk, int &n_chunk) {
    const long long nc = std::max(1, (ntrg + 63) / 64);
    num_sms = std::max(num_sms, 1);
    if (prec == PREC_MIXED) {
        n_chunk = (int)std::max(1LL, ((long long)num_sms * 64 + nc - 1) / nc);
        n_chunk = std::min(n_chunk, std::max(1, nsrc / 256));
        chunk = ((nsrc + n_chunk - 1) / n_chunk + 31) / 32 * 32;
        n_chunk = (nsrc + chunk - 1) / chunk;
        return;
    }
    int per_sm = 8;
    direct_p2p_fp64_occupancy(uk, per_sm);
    const double slots = (double)num_sms * per_sm;
    double best = 0.0;
    chunk = (nsrc + 31) / 32 * 32;
    n_chunk = 1;
    // up to eight turns of the warps, tiles of 32 sources
    const long long most = std::min<long long>((nsrc + 31) / 32, std::max<long long>(1, (long long)(8 * slots) / nc));
    for (long long n = 1; n <= most; n = n < 64 ? n + 1 : n + n / 16) {
        const int c = (int)((((nsrc + n - 1) / n) + 31) / 32 * 32);
        const long long k = (nsrc + c - 1) / c;
        const double items = (double)nc * k;
        // useful share of the time: ragged sources, ragged last turn, cost per item
        const double eff = (double)nsrc / ((double)k * c) * items / (std::ceil(items / slots) * slots) * c / (c + 40.0);
        if (eff > best * 1.001) {
            best = eff;
            chunk = c;
            n_chunk = (int)k;
        }
    }
}

bool direct_in_place(int uk, const ListP2PArgs &a, const double *out) {
    auto meets = [&](const double *p, size_t n) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(p), o = reinterpret_cast<uintptr_t>(out);
        return b < o + sizeof(double) * (size_t)a.ntrg * uk_tdim(uk) && o < b + sizeof(double) * n;
    };
    return meets(a.src_xyz, 3 * (size_t)a.nsrc) || meets(a.src_val, (size_t)uk_sdim(uk) * a.nsrc);
}

cudaError_t launch_direct_p2p(int uk, int prec, const ListP2PArgs &args, int add, int num_sms, cudaStream_t stream) {
    if (args.nsrc <= 0 || args.ntrg <= 0) return cudaSuccess;
    if (uk < 0 || uk >= UK_COUNT || (uk_tvdim(uk) > 0) != (args.trg_aux != nullptr)) return cudaErrorInvalidValue;
    const bool split = args.parts != nullptr;  // (one chunk too: targets written over the sources)
    const long long items = (long long)((args.ntrg + 63) / 64) * args.n_chunk;
    if ((prec == PREC_MIXED && !args.counter) || (args.n_chunk > 1 && add != 2 && !split) || items > 0x7fffffffll) return cudaErrorInvalidValue;
    ListP2PArgs a = args;
    a.n_items = (int)items;
    a.atomic_out = split && add != 2 ? 0 : add;
    if (add == 2) a.parts = nullptr;
    cudaError_t e = prec == PREC_MIXED ? direct_p2p_mixed(uk, a, num_sms, stream) : direct_p2p_fp64(uk, a, num_sms, stream);
    if (e != cudaSuccess || !split || add == 2) return e;
    const long long n = (long long)a.ntrg * uk_tdim(uk);
    sum_chunks_kernel<<<(int)std::min<long long>((n + 255) / 256, 148 * 16), 256, 0, stream>>>(a.parts, a.n_chunk, n, add,
                                                                                             a.trg_out);
    return cudaGetLastError();
}

cudaError_t launch_pack_records(int uk, int n, const int *perm, const double *xyz, const double *v1, int d1,
                                const double *v2, double *rec, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    if (uk < 0 || uk >= UK_COUNT || (d1 < uk_sdim(uk)) != (v2 != nullptr)) return cudaErrorInvalidValue;
    return with_uk(uk, [&](auto id) {
        const int threads = 256;
        const int grid = std::min((n + threads - 1) / threads, 148 * 16);
        pack_records_kernel<decltype(id)::value><<<grid, threads, 0, stream>>>(n, perm, xyz, v1, d1, v2, rec);
        return cudaGetLastError();
    });
}

cudaError_t launch_pack_surface(int uk, const int *nodes, int m, int n, const double *xyz, const double *dens,
                                const int *level, const double *den_exp, double *rec, cudaStream_t stream) {
    if (m <= 0) return cudaSuccess;
    if (uk < 0 || uk >= UK_COUNT || uk_sdim(uk) > 4) return cudaErrorInvalidValue;
    return with_uk(uk, [&](auto id) {
        constexpr int UK = decltype(id)::value;
        if constexpr (Uk<UK>::SDIM <= 4) {
            const DensExp e = {{den_exp[0], den_exp[1], den_exp[2], den_exp[3]}};
            const int grid = (int)std::min<long long>(((long long)m * n + 255) / 256, 148 * 16);
            pack_surface_kernel<UK><<<grid, 256, 0, stream>>>(nodes, m, n, xyz, dens, level, e, rec);
        }
        return cudaGetLastError();
    });
}

cudaError_t launch_scatter_add(int n, int d, const int *perm, const double *in, const double *alpha, double *out,
                               cudaStream_t stream) {
    if (n <= 0 || d <= 0) return cudaSuccess;
    const int threads = 256;
    const long long total = (long long)n * d;
    const int grid = (int)std::min<long long>((total + threads - 1) / threads, 148 * 16);
    scatter_add_kernel<<<grid, threads, 0, stream>>>(n, d, perm, in, alpha, out);
    return cudaGetLastError();
}

}  // namespace stk
