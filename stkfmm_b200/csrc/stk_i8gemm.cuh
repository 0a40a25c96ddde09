// stk_i8gemm.cuh -- FP64 matrix products on the sm_100a int8 tensor cores (stk_i8gemm.cu).
//
// Every row of an operand (K values) is scaled by its own power of two, 2^e > 128/127 max |x|,
// and rounded to an integer a' = x 2^(55 - e), written as seven balanced base-256 digits,
// a' = sum_i d_i 256^(6 - i) with -128 <= d_i <= 127 (the splitting of the published Ozaki
// scheme, with integer products).  A product of two rows is
//   sum_k a'_k b'_k ~ sum_{g = 0..7} 256^(12 - g) sum_{i + j = g} sum_k d_ik e_jk,
// 34 int8 dot products accumulated exactly in int32.  A value is rounded to 2^-56 of its row's
// scale, 2^e <= 2.02 max |x|, and the dropped terms i + j >= 8 add 2% to that: an element is off by
// at most 4.2 K 2^-56 max|a| max|b|, about sqrt(K) of it with mixed signs, and 2^-52 of itself (two
// conversions).  On rows of one size that is below the rounding of an FP64 sum; on graded rows it is
// not componentwise (hence the scales along K below).  (Without i + j = 7, 28 products and 15%
// faster, the dropped terms showed where a row's largest value is far above the others: the
// rounding noise of a triply periodic Laplace FMM's potential rose from 1.3e-10 to 1.9e-8.)
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace stk {

constexpr int kI8Planes = 7;     // digits per value
constexpr int kI8Rows = 128;     // rows per block
constexpr int kI8K = 32;         // K values per block
constexpr int kI8PlaneBytes = kI8Rows * kI8K;              // 4 KB
constexpr int kI8BlockBytes = kI8Planes * kI8PlaneBytes;   // 28 KB
// int32 sums stay exact up to 2^31 / (7 x 2^14) = 18724 values of K
constexpr int kI8MaxSegment = 512;  // K blocks summed before the accumulators are drained

// An operand: rows x K values as digits.  Blocks of 128 rows x 32 K, row block major, each
// block its seven planes (most significant first), each plane in the tensor core's K-major
// core matrices (8 rows x 16 bytes): a pipeline stage is one contiguous copy.
struct I8Operand {
    const uint8_t *dig = nullptr;
    const int *scale = nullptr;  // per row (padded to 128): the exponent e - 35, or kI8NonFinite
    int nkb = 0;                 // K blocks per row block
};
// Scales are kept as exponents: 2^(e - 35) itself leaves the range of a double for rows below
// 2^-987, and a product of two scales does long before the results they stand for.
constexpr int kI8NonFinite = 1 << 20;  // a row with an infinity or NaN: its products are NaN
// Rows of digits to gather from: row r is nkb x 7 x 32 bytes (K block, plane, K), so that a
// tile's columns are any rows, fetched 16 bytes at a time.
struct I8Rows {
    const uint8_t *dig = nullptr;
    const int *scale = nullptr;  // per row
    int nkb = 0;
};
inline size_t i8_row_bytes(long long rows, int nkb) { return (size_t)rows * nkb * kI8Planes * kI8K; }
inline int i8_kblocks(long long K) { return (int)((K + kI8K - 1) / kI8K); }
inline long long i8_pad_rows(long long rows) { return (rows + kI8Rows - 1) / kI8Rows * kI8Rows; }
inline size_t i8_bytes(long long rows, int nkb) {
    return (size_t)(i8_pad_rows(rows) / kI8Rows) * (size_t)nkb * kI8BlockBytes;
}

// Scales along K.  The far field's operators and densities are written in singular-vector
// coordinates whose sizes fall over eight decades, large where the other operand is small; a
// common scale per row would spend its digits on the largest.  Products are therefore formed
// as (A D^-1)(D B) with D_k a power of two, the largest |A_mk| over m rounded up: `kexp` below
// are exponents, and the values of index k are multiplied by 2^kexp[k] before they are split
// (null: 0).
// up[k] = e, 2^e > max_m |src[k ld + m]| (0 for a zero column; within +-kI8KExp), down[k] = -e
constexpr int kI8KExp = 100;
cudaError_t i8_column_scales(const double *src, long long ld, long long rows, int K, int *up, int *down,
                             cudaStream_t s);
// the same for rows of K contiguous values: max over r of |src[r ld + k]|; mag: K words of scratch
cudaError_t i8_row_scales(const double *src, long long ld, long long rows, int K, unsigned *mag, int *up, int *down,
                          cudaStream_t s);

// x(r, k) = src[(idx ? idx[r] : r) ld + k] 2^kexp[k], K contiguous; idx[r] < 0 gives a zero row.
// rmul (nullable): powers of two that multiply the rows (through their stored scales).
cudaError_t i8_digits(const double *src, long long ld, const int *idx, long long rows, int K, int nkb, const int *kexp,
                      const double *rmul, uint8_t *dig, int *scale, cudaStream_t s);
// the same as gatherable rows (I8Rows)
cudaError_t i8_digits_rows(const double *src, long long ld, long long rows, int K, int nkb, const int *kexp,
                           uint8_t *dig, int *scale, cudaStream_t s);
// the same with, per block b of 128 rows, kof[b] values (<= 32 nkb, the rest zero), nof[b] rows
// (the rest zero) and the exponents kexp + kset[b] kld
cudaError_t i8_digits_blocks(const double *src, long long ld, long long rows, const int *kof, const int *nof, int nkb,
                             const int *kexp, const int *kset, int kld, uint8_t *dig, int *scale, cudaStream_t s);
// x(r, k) = src[k ld + r] 2^kexp[k]
cudaError_t i8_digits_trans(const double *src, long long ld, long long rows, int K, int nkb, const int *kexp,
                            uint8_t *dig, int *scale, cudaStream_t s);
// rows of a gathered operand, in eight types of 2^lg rows: row r = (c, j = r mod 2^lg) has
// x(r, k) = z[pos ldz + srow[row_off[c] + k]], pos = tab[tab_off[c] + j nq[c] + rowq[row_off[c] + k]]
// (0 where pos < 0) times 2^kexp[row_off[c] + k], k < K[c]; row_off multiples of 4
struct I8Gather {
    const double *z;
    const int *tab, *rowq, *srow;
    const int *kexp;
    long long tab_off[8], row_off[8];
    int nq[8], K[8];
    int ldz, lg;
};
cudaError_t i8_digits_gather(const I8Gather &g, int nkb, uint8_t *dig, int *scale, cudaStream_t s);

// C[m + ldc col(n)] (add = 0: =, 1: +=) sum_k A[m][k] B[n][k], m < M, n < N;
// col(n) = cols ? cols[n] : n (no two n may share a column).  Products with few output tiles
// are split along K into i8_gemm_parts(M, N, nkb) parts, written to `parts` (M x N each) and
// summed in order; parts may be null when that is 1.  err: device int, set non-zero when a
// pipeline wait gave up.
int i8_gemm_parts(long long M, long long N, int nkb);
cudaError_t i8_gemm(int M, int N, I8Operand A, I8Operand B, int add, double *C, long long ldc, const int *cols,
                    double *parts, int *err, cudaStream_t s);

// One 128 x 128 output tile of a grouped product: rows of A block a_blk, columns of B
// block b_blk (row blocks of the operands), the first nkb K blocks of both.  Written (or
// added) to C[c_off + n ldc + m], m < m_valid, n < n_valid.
struct I8Tile {
    int a_blk, b_blk, nkb, m_valid, n_valid, ldc;
    long long c_off;
};
cudaError_t i8_grouped(I8Operand A, I8Operand B, const I8Tile *tiles, int ntiles, int add, double *C, int *err,
                       cudaStream_t s);

// The same with the columns gathered: column n < n_valid of tile t is row rows[128 b_blk + n]
// of B.
cudaError_t i8_grouped_gather(I8Operand A, I8Rows B, const int *rows, const I8Tile *tiles, int ntiles, int add, double *C,
                              int *err, cudaStream_t s);

}  // namespace stk
