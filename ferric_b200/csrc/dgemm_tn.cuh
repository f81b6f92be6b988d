// All-FP64 tile GEMM on the DMMA tensor path:
//     value(m, n) = sum_{k in split} A(m, k) * B(n, k)
// with each operand K-major (row-major M x K and N x K, the default "TN"
// form) or, with TA / TB, MN-major (stored K x M / K x N), and a functor
// epilogue, so one kernel serves the gradient's second contraction
// (Gamma = 4 B_ov Tt^T), the DF-K half-transform and rank update, the MP2
// densities and the RI response products.
//
// Tile BM x BN x 16 (128 x 64 where nothing else is said; narrower ones for
// products whose M or N would leave most of that empty), 8 warps (4 x 2);
// 3-stage cp.async pipeline; split-K over blockIdx.z.  Shared-memory rows are
// padded to 20 doubles so the fragment reads (g*20 + t) hit distinct banks.
// V16 copies 16 bytes at a time, half the copy instructions; it needs both
// operands K-major with rows on 16 bytes (dgemm_tn_launch looks).
#pragma once
#include <type_traits>

#include "dmma.cuh"

namespace fc {

constexpr int DG_BM = 128, DG_BN = 64, DG_BK = 16, DG_LDK = 20, DG_STAGES = 3;
constexpr int dg_smem(int bm, int bn) { return DG_STAGES * (bm + bn) * DG_LDK * 8; }
constexpr int DG_SMEM = dg_smem(DG_BM, DG_BN);

// The tile body.  A(m, k) = TA ? A[k*lda + m] : A[m*lda + k], and B(n, k) the
// same with TB: a transposed (MN-major) operand is read with consecutive
// threads on consecutive m (n), so its global loads stay coalesced.  The
// epilogue gets `z` (the split or the batch index).
template <class Epi, bool TA, bool TB, int BM = DG_BM, int BN = DG_BN, bool V16 = false>
__device__ __forceinline__ void dgemm_tile(const double* __restrict__ A, int64_t lda, const double* __restrict__ B,
                                           int64_t ldb, int M, int N, int64_t kbeg, int64_t kend, int upper_only,
                                           const Epi& epi, int z, int bx, int by) {
    static_assert(BM % 32 == 0 && BN % 16 == 0, "4 x 2 warps of 8 x 8 DMMA tiles");
    static_assert(!V16 || (!TA && !TB), "16-byte copies: K-major operands");
    constexpr int MT = BM / 32, NT = BN / 16;  // DMMA tiles per warp
    extern __shared__ __align__(16) double dg_smem_buf[];
    double* sA = dg_smem_buf;                               // [STAGES][BM][LDK]
    double* sB = dg_smem_buf + DG_STAGES * BM * DG_LDK;     // [STAGES][BN][LDK]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = warp & 3, wn = warp >> 2;
    const int m0 = by * BM, n0 = bx * BN;
    if (upper_only && m0 > n0 + BN - 1) return;  // tile strictly below the diagonal
    if (kbeg >= kend) return;
    const int nk = (int)((kend - kbeg + DG_BK - 1) / DG_BK);

    // rows [r0, r0 + ROWS) of a K-major operand (R rows), 16 bytes a copy
    auto load16 = [&](double* s, const double* X, int64_t ld, int r0, int R, int64_t kb, auto rows) {
        constexpr int ROWS = decltype(rows)::value;
#pragma unroll
        for (int e = 0; e < (ROWS * DG_BK / 2 + 255) / 256; ++e) {
            const int idx = tid + 256 * e, row = idx >> 3, kk = (idx & 7) * 2, gr = r0 + row;
            if (row >= ROWS) break;
            const int64_t left = kend - (kb + kk);
            const int bytes = gr < R && left > 0 ? (left > 1 ? 16 : 8) : 0;
            cp_async16n(s + row * DG_LDK + kk, bytes ? X + (int64_t)gr * ld + kb + kk : X, bytes);
        }
    };
    auto load8 = [&](double* s, const double* X, int64_t ld, int r0, int R, int64_t kb, auto rows, auto trans) {
        constexpr int ROWS = decltype(rows)::value;
        constexpr bool T = decltype(trans)::value;
#pragma unroll
        for (int e = 0; e < ROWS * DG_BK / 256; ++e) {
            const int idx = tid + 256 * e;
            const int row = T ? idx % ROWS : idx >> 4, kk = T ? idx / ROWS : idx & 15;
            const int gr = r0 + row;
            const int64_t gk = kb + kk;
            const bool ok = gr < R && gk < kend;
            cp_async8(s + row * DG_LDK + kk, ok ? (T ? X + gk * ld + gr : X + (int64_t)gr * ld + gk) : X, ok);
        }
    };
    auto load = [&](int stage, int kt) {
        const int64_t kb = kbeg + (int64_t)kt * DG_BK;
        using RA = std::integral_constant<int, BM>;
        using RB = std::integral_constant<int, BN>;
        double* a = sA + stage * BM * DG_LDK;
        double* b = sB + stage * BN * DG_LDK;
        if constexpr (V16) {
            load16(a, A, lda, m0, M, kb, RA{});
            load16(b, B, ldb, n0, N, kb, RB{});
        } else {
            load8(a, A, lda, m0, M, kb, RA{}, std::integral_constant<bool, TA>{});
            load8(b, B, ldb, n0, N, kb, RB{}, std::integral_constant<bool, TB>{});
        }
    };

    double acc[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
    for (int s = 0; s < DG_STAGES - 1; ++s) {
        if (s < nk) load(s, s);
        cp_async_commit();
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<DG_STAGES - 2>();
        __syncthreads();
        const int pf = kt + DG_STAGES - 1;
        if (pf < nk) load(pf % DG_STAGES, pf);
        cp_async_commit();
        const double* a = sA + (kt % DG_STAGES) * BM * DG_LDK;
        const double* b = sB + (kt % DG_STAGES) * BN * DG_LDK;
#pragma unroll
        for (int ks = 0; ks < DG_BK / 4; ++ks) {
            double af[MT], bf[NT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) af[mt] = a[(wm * (BM / 4) + mt * 8 + g) * DG_LDK + ks * 4 + t];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) bf[nt] = b[(wn * (BN / 2) + nt * 8 + g) * DG_LDK + ks * 4 + t];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) dmma_8x8x4(acc[mt][nt], af[mt], bf[nt]);
        }
    }
    cp_async_wait<0>();

#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = m0 + wm * (BM / 4) + mt * 8 + g;
                const int n = n0 + wn * (BN / 2) + nt * 8 + 2 * t + h;
                if (m < M && n < N) epi(m, n, acc[mt][nt][h], z);
            }
}

template <class Epi, bool TA = false, bool TB = false, int BM = DG_BM, int BN = DG_BN, bool V16 = false>
__global__ void __launch_bounds__(256) dgemm_tn_kernel(const double* __restrict__ A, int64_t lda,
                                                       const double* __restrict__ B, int64_t ldb,
                                                       int M, int N, int64_t K, int64_t k_per_split,
                                                       int upper_only, Epi epi, const int* run_if = nullptr) {
    if (run_if && !(run_if[0] | run_if[1])) return;  // the residue form's result stands (mgemm.cuh)
    const int64_t kbeg = (int64_t)blockIdx.z * k_per_split;
    const int64_t kend = kbeg + k_per_split < K ? kbeg + k_per_split : K;
    dgemm_tile<Epi, TA, TB, BM, BN, V16>(A, lda, B, ldb, M, N, kbeg, kend, upper_only, epi, (int)blockIdx.z,
                                         (int)blockIdx.x, (int)blockIdx.y);
}

// K-major product with the copies that its operands allow (k_per_split a
// multiple of DG_BK unless there is one split).  16-byte copies: the DF-K half
// transform at n 600, naux 2400, nocc 60 (and with it the JK build) 4% faster,
// the MO dressing at naux 600, n 180 5%; below eight k-steps there is nothing
// to gain (JK at n 80: 110 -> 115 us with them).
template <class Epi, int BM = DG_BM, int BN = DG_BN>
void dgemm_tn_launch(dim3 grid, cudaStream_t st, const double* A, int64_t lda, const double* B, int64_t ldb, int M,
                     int N, int64_t K, int64_t k_per_split, int upper_only, const Epi& epi,
                     const int* run_if = nullptr) {
    constexpr int smem = dg_smem(BM, BN);
    const bool aligned = !(((uintptr_t)A | (uintptr_t)B | (uintptr_t)(lda * 8) | (uintptr_t)(ldb * 8)) & 15);
    if (!aligned || K < 8 * DG_BK || k_per_split < 8 * DG_BK)
        dgemm_tn_kernel<Epi, false, false, BM, BN>
            <<<grid, 256, smem, st>>>(A, lda, B, ldb, M, N, K, k_per_split, upper_only, epi, run_if);
    else
        dgemm_tn_kernel<Epi, false, false, BM, BN, true>
            <<<grid, 256, smem, st>>>(A, lda, B, ldb, M, N, K, k_per_split, upper_only, epi, run_if);
}
template <class Epi, int BM = DG_BM, int BN = DG_BN>
cudaError_t dgemm_tn_smem() {
    const cudaError_t e = cudaFuncSetAttribute(dgemm_tn_kernel<Epi, false, false, BM, BN>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, dg_smem(BM, BN));
    return e != cudaSuccess ? e
                            : cudaFuncSetAttribute(dgemm_tn_kernel<Epi, false, false, BM, BN, true>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, dg_smem(BM, BN));
}

// Batched over blockIdx.z: operands z * sa and z * sb elements on, all of K.
template <class Epi, bool TA = false, bool TB = false>
__global__ void __launch_bounds__(256) dgemm_batched_kernel(const double* __restrict__ A, int64_t lda, int64_t sa,
                                                            const double* __restrict__ B, int64_t ldb, int64_t sb,
                                                            int M, int N, int64_t K, Epi epi) {
    const int z = (int)blockIdx.z;
    dgemm_tile<Epi, TA, TB>(A + z * sa, lda, B + z * sb, ldb, M, N, 0, K, 0, epi, z, (int)blockIdx.x,
                            (int)blockIdx.y);
}

// The tiles of an M x M product that reach the upper triangle, numbered by rows.
template <int BM, int BN>
int dgemm_upper_tiles(int64_t M) {
    const int tn = (int)((M + BN - 1) / BN);
    int t = 0;
    for (int y = 0; y * BM < M; ++y) t += tn - y * BM / BN;
    return t;
}

// Batched as above, only those tiles (blockIdx.x), each in `splits` ranges of K:
// the epilogue's z is batch * splits + range.  A grid with the tiles below the
// diagonal in it leaves the SMs that got those idle.
template <class Epi, int BM, int BN>
__global__ void __launch_bounds__(256) dgemm_upper_kernel(const double* __restrict__ A, const double* __restrict__ B,
                                                          int64_t ld, int64_t stride, int M, int64_t K, int splits,
                                                          int64_t k_per_split, Epi epi) {
    const int z = (int)blockIdx.z, b = z / splits, tn = (M + BN - 1) / BN;
    int x = (int)blockIdx.x, y = 0;
    while (x >= tn - y * BM / BN) x -= tn - y++ * BM / BN;
    const int64_t kbeg = (int64_t)(z % splits) * k_per_split;
    const int64_t kend = kbeg + k_per_split < K ? kbeg + k_per_split : K;
    dgemm_tile<Epi, false, false, BM, BN>(A + b * stride, ld, B + b * stride, ld, M, M, kbeg, kend, 0, epi, z,
                                          x + y * BM / BN, y);
}

// value * alpha -> C[m*ldc + n]
struct EpiStore {
    double* C;
    int64_t ldc;
    double alpha;
    int accumulate;  // C += alpha v instead of C = alpha v
    __device__ __forceinline__ void operator()(int m, int n, double v, int) const {
        double* c = C + (int64_t)m * ldc + n;
        *c = accumulate ? *c + alpha * v : alpha * v;
    }
};

// v -> C[z stride + m ldc + n]
struct EpiBatchStore {
    double* C;
    int64_t ldc, stride;
    __device__ __forceinline__ void operator()(int m, int n, double v, int z) const {
        C[(int64_t)z * stride + (int64_t)m * ldc + n] = v;
    }
};

// s + x[0] + x[stride] + ... (n terms, in order), sixteen loads in flight, the
// last ones too.
__device__ __forceinline__ double fold_in_order(const double* __restrict__ x, int n, int64_t stride, double s = 0.0) {
    for (int i = 0; i < n; i += 16, x += 16 * stride) {
        double v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = i + u < n ? __ldg(x + u * stride) : 0.0;
#pragma unroll
        for (int u = 0; u < 16; ++u) s += v[u];
    }
    return s;
}

// split-K partial -> P[split][m*N + n]
struct EpiSplit {
    double* P;
    int64_t split_stride;
    int N;
    __device__ __forceinline__ void operator()(int m, int n, double v, int split) const {
        P[(int64_t)split * split_stride + (int64_t)m * N + n] = v;
    }
};

}  // namespace fc
