// FP64 matrix products on the int8 tensor cores, through residues.
//
//     out[n * ldo + m] (+)= alpha * sum_k A[m, k] B[n, k]
//
// Every operand row is scaled by a power of two to integers of at most
// 2^62.1 in the 2-norm and kept as its residues modulo MG_N = 16 pairwise
// coprime moduli <= 256 (int8).  One int8 product with exact int32 sums per
// modulus (tcgen05.mma kind::i8) gives the integer product modulo each of
// them, and the Chinese remainder theorem gives the integer itself: by the
// Cauchy-Schwarz inequality it is below 2^124.2 < P / 2, P = the product of
// the moduli (Ozaki, Uchino and Imamura's "scheme II", 2025).  The errors are
// the operands' rounding to integers, |dx| <= 2^-62.1 |x| per element (an
// element above 2^-8 of its row's norm, which the typical one is up to K =
// 65535, keeps all 53 bits), the remainder theorem's 64-bit fraction and the
// last rounding to FP64: rms 2^-61 |x| |y| at most, besides that rounding.
//
// That is an error in the norm: small against a sum of FP64 products in k
// order, rms 2^-54 sum_k |x_k y_k| or more, only where sum_k |x_k y_k| is not
// far below |x| |y|.  Rows whose large elements meet their partners' small
// ones (a triangular factor's first rows, opposite slopes) can make it so.  So
// every product is guarded: for each row m of A
//     (sum_n (sum_k |A[m, k] B[n, k]|)^2)^(1/2) >= MG_GUARD |A[m]| ||B||_F
// is checked through lower bounds of its left side that need no product (the
// column sums of |B| and B^2), and the same for each row of B.  Where it holds,
// each row and each column of the result is at least as precise, in its
// 2-norm, as FP64 sums; where it does not, `bad` is raised and the caller runs
// the DMMA form.  (An element far below its row's and its column's norms has
// that absolute precision, not 53 bits of its own.)
//
// Why: FP64 arithmetic runs at 37 TFLOP/s on this chip in the FMA pipe and on
// the DMMA path alike (cuBLAS DGEMM 35 measured), int8 products at 2.4-3 POP/s
// (2400 / 16 = 150 TFLOP/s of FP64 products).  It pays where the operands'
// conversion (about 110 instructions per element) is spread over enough
// products: the callers' rules say where.
//
// Rows with a norm outside [1e-70, 1e70] (not all zero), infinities or NaN
// raise `bad` too.  The kernels of a product whose flag is up return at once.
#pragma once
#include <vector>

#include "fc_internal.cuh"

namespace fc {

constexpr int MG_N = 16;            // moduli
constexpr int MG_BM = 128, MG_BN = 256;
constexpr int MG_KT = 128;          // bytes (elements) of K per pipeline stage
constexpr int64_t MG_KMAX = 65535;  // 2^14 K < 2^30: the sums' reduction modulo p
// rms errors: operands |x| |y| 2^(-1.3 - 61.1), fraction 2^-61.3 |x| |y| at most,
// together 2^-61; 2^-54 sum_k |x_k y_k| for FP64 sums
constexpr double MG_GUARD = 1.0 / 128;

// One operand: residues of `rows` rows at pitch kp (K rounded up to MG_KT, zero
// padded), moduli `plane` rows apart, and the rows' scales (value = integer *
// scale).  slice() is a range of its rows.
struct MgOperand {
    int8_t* r = nullptr;
    const double* scale = nullptr;
    int64_t rows = 0, K = 0, kp = 0, plane = 0;
    MgOperand slice(int64_t r0, int64_t n) const { return {r + r0 * kp, scale + r0, n, K, kp, plane}; }
};
inline int64_t mg_kp(int64_t K) { return (K + MG_KT - 1) / MG_KT * MG_KT; }
inline size_t mg_bytes(int64_t rows, int64_t K) { return (size_t)MG_N * rows * mg_kp(K); }

// A matrix of n[0] rows (pitch ld) and n[1] columns, with the sums of |x| and
// x^2 along each row (axis 0) and column (axis 1) and the scales that follow
// from them (0: norm out of range).  Its rows or its columns can be operand
// rows; the other axis is then k.
struct MgMat {
    const double* p = nullptr;
    int64_t ld = 0, n[2] = {0, 0};
    double2* sum[2] = {nullptr, nullptr};  // (sum |x|, sum x^2)
    double* scale[2] = {nullptr, nullptr};
    double* f2 = nullptr;                  // partial sums of the squared Frobenius norm
    __host__ __device__ int short_axis() const { return n[0] <= n[1] ? 0 : 1; }
};
// Doubles that the sums of an R x C matrix take (mg_mat lays them out), and
// those of the partial sums that mg_stats, mg_convert and mg_guard work in.
inline int64_t mg_stat_doubles(int64_t R, int64_t C) { return 3 * (R + C) + (R < C ? R : C) / 8 + 8; }
inline int64_t mg_part_doubles(int64_t R, int64_t C) {
    return 2 * (R * ((C + 127) / 128) + C * ((R + 127) / 128));
}
MgMat mg_mat(const double* p, int64_t ld, int64_t R, int64_t C, double* stat);
fc_status mg_stats(const MgMat& x, double* part, const int* bad, cudaStream_t st);
// Operand rows = rows (axis 0) or columns (axis 1) of x -> residues at r.  *bad
// (device) is set to 1 for rows out of range and, with a partner (its rows
// along py, the same K), where the guard does not hold for x's rows.
fc_status mg_convert(const MgMat& x, int axis, int8_t* r, const MgMat* y, int py, double* part, int* bad,
                     cudaStream_t st, MgOperand* o);
// The guard alone, for an operand that was converted before.
fc_status mg_guard(const MgMat& x, int axis, const MgMat& y, int py, double* part, int* bad, cudaStream_t st);

struct MgOut {
    double* out;
    int64_t ld;
    int64_t split_stride;  // split-K: split s writes out + s * split_stride (accumulate must be 0)
    double alpha;
    int accumulate;
};

// Tiles (tm, tn) of the product, `splits` ranges of K each; upper: only tiles
// that reach m >= n.  Appended to items (or only counted: nullptr).
int64_t mg_tiles(int64_t M, int64_t N, int64_t K, bool upper, int splits, std::vector<int4>* items);
size_t mg_scratch_bytes();  // residues of the tiles in flight
// items: device copy of mg_tiles' list.  flags (device): nothing runs where the
// first is up; the second takes a wait's timeout.
fc_status mg_gemm(const MgOperand& A, const MgOperand& B, const MgOut& out, const int4* items, int64_t nitems,
                  void* scratch, int* flags, cudaStream_t st);

// A whole product of two FP64 matrices in device memory, converted here:
// operand rows are the rows of p, or its columns (cols).  Uses the residue
// slots but WS_MG_T; `splits` ranges of at most MG_KMAX each.  out.out ==
// nullptr: the result, or the splits' partials, go to WS_MG_G (*part), where
// they stay until the next residue call.
// *room = false, and nothing is launched, where all that does not fit.
// flags (two device ints, zeroed by the caller): rows out of range or the
// guard, a wait's timeout; the product is valid where both stay 0.
struct MgSrc {
    const double* p;
    int64_t ld, rows;
    bool cols;
};
fc_status mg_multiply(const MgSrc& a, const MgSrc& b, int64_t K, MgOut out, bool upper, int splits, int* flags,
                      cudaStream_t st, bool* room, double** part = nullptr);
constexpr int MG_LAUNCHES = 10, MG_LAUNCHES_SAME = 6;  // kernels of a product of two matrices, of one with itself
// Synchronises: whether the products under `flags` stand (or their DMMA form
// ran); FC_ERR_TIMEOUT where a wait ran out.
fc_status mg_outcome(const int* flags, const char* what, cudaStream_t st, bool* stands);
// out[n * ld + m] = alpha * sum of the splits' partials, in order.
fc_status mg_fold(const double* part, int splits, int64_t M, int64_t N, double alpha, double* out, int64_t ld,
                  cudaStream_t st);
// Splits of K that give the tiles of an M x N product about one wave, at least
// four k-steps each.
int mg_splits(int64_t M, int64_t N, int64_t K, bool upper);

}  // namespace fc
