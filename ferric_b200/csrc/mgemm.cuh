// FP64 matrix products on the int8 tensor cores, through residues.
//
//     out[n * ldo + m] (+)= alpha * sum_k A[m, k] B[n, k]
//
// Every operand row is scaled by a power of two to integers of at most
// 2^58.35 in the 2-norm and kept as its residues modulo MG_N = 15 pairwise
// coprime moduli <= 256 (int8).  One int8 product with exact int32 sums per
// modulus (tcgen05.mma kind::i8) gives the integer product modulo each of
// them, and the Chinese remainder theorem gives the integer itself: by the
// Cauchy-Schwarz inequality it is below 2^116.7 < P / 2, P = the product of
// the moduli (Ozaki, Uchino and Imamura's "scheme II", 2025).  The only
// errors are the operands' rounding to integers, |dx| <= 2^-58.35 |x| / 2 per
// element, and the last rounding to FP64: |error| <= 2^-58 |x| |y| on average,
// against about 2^-54.5 |x| |y| for a sum of FP64 products in k order.
//
// Why: FP64 arithmetic runs at 37 TFLOP/s on this chip in the FMA pipe and on
// the DMMA path alike (cuBLAS DGEMM 35 measured), int8 products at 2.4-3 POP/s
// (2400 / 15 = 160 TFLOP/s of FP64 products).  It pays where the operands'
// conversion (about 100 instructions per element) is spread over enough
// products: the callers' rules say where.
//
// Rows with a norm outside [1e-100, 1e100] (not 0), infinities or NaN raise
// `bad`; the caller then runs the DMMA form.
#pragma once
#include <vector>

#include "fc_internal.cuh"

namespace fc {

constexpr int MG_N = 15;            // moduli
constexpr int MG_BM = 128, MG_BN = 256;
constexpr int MG_KT = 128;          // bytes (elements) of K per pipeline stage
constexpr int64_t MG_KMAX = 65535;  // 2^14 K < 2^30: the sums' reduction modulo p

// One operand: residues of `rows` rows at pitch kp (K rounded up to MG_KT, zero
// padded), moduli `plane` rows apart, and the rows' scales (value = integer *
// scale).  slice() is a range of its rows.
struct MgOperand {
    int8_t* r = nullptr;
    double* scale = nullptr;
    int64_t rows = 0, K = 0, kp = 0, plane = 0;
    MgOperand slice(int64_t r0, int64_t n) const { return {r + r0 * kp, scale + r0, n, K, kp, plane}; }
};
inline int64_t mg_kp(int64_t K) { return (K + MG_KT - 1) / MG_KT * MG_KT; }
inline size_t mg_bytes(int64_t rows, int64_t K) { return (size_t)MG_N * rows * mg_kp(K); }

// Operand rows = rows of src (R x K, row pitch ld) -> o (buffers given in
// o->r, o->scale).  *bad (device) is set to 1 for rows out of range.
fc_status mg_convert_rows(const double* src, int64_t ld, int64_t R, int64_t K, MgOperand* o, int* bad,
                          cudaStream_t st);
// Operand rows = columns of src (K x R, row pitch ld).  `part` holds
// mg_colpart(R, K) doubles.
inline int64_t mg_colchunks(int64_t K) { return (K + 255) / 256; }
inline int64_t mg_colpart(int64_t R, int64_t K) { return R * mg_colchunks(K); }
fc_status mg_convert_cols(const double* src, int64_t ld, int64_t R, int64_t K, MgOperand* o, double* part, int* bad,
                          cudaStream_t st);

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
// items: device copy of mg_tiles' list.  *err (device) takes a wait's timeout.
fc_status mg_gemm(const MgOperand& A, const MgOperand& B, const MgOut& out, const int4* items, int64_t nitems,
                  void* scratch, int* err, cudaStream_t st);

// A whole product of two FP64 matrices in device memory, converted here:
// operand rows are the rows of p, or its columns (cols).  Uses every residue
// slot but WS_MG_T.  K beyond MG_KMAX runs in ranges that accumulate (splits
// must be 1).  *room = false, and nothing is launched, where the residues do
// not fit.  flags (two device ints, zeroed by the caller): rows out of range,
// a wait's timeout; the product is valid where both stay 0.
struct MgSrc {
    const double* p;
    int64_t ld, rows;
    bool cols;
};
fc_status mg_multiply(const MgSrc& a, const MgSrc& b, int64_t K, const MgOut& out, bool upper, int splits, int* flags,
                      cudaStream_t st, bool* room);
// out[n * ld + m] = alpha * sum of the splits' partials, in order.
fc_status mg_fold(const double* part, int splits, int64_t M, int64_t N, double alpha, double* out, int64_t ld,
                  cudaStream_t st);
// Splits of K that give the tiles of an M x N product about one wave, at least
// four k-steps each.
int mg_splits(int64_t M, int64_t N, int64_t K, bool upper);

}  // namespace fc
