// Residue conversion kernels and the tcgen05 GEMM of mgemm.cuh.
#include <algorithm>
#include <cmath>

#include "mgemm.cuh"
#include "tc.cuh"
#include "tmap.cuh"

namespace fc {

namespace {

// 16 pairwise coprime integers up to 256 (the largest ones but for the last
// three, which make their product P = 2^125.22 an FP64 number within 2^-59).
constexpr int MOD[MG_N] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 197, 193, 179};

constexpr int symmod(int64_t x, int p) {
    int64_t r = x % p;
    if (r < 0) r += p;
    return (int)(2 * r > p ? r - p : r);
}
// 256^b mod p for b = 0..7, symmetric (a signed byte: 256^0 mod 256 = 1, the
// others 0), four to a word
constexpr uint32_t coef(int p, int word) {
    uint32_t w = 0;
    int64_t v = 1;
    for (int b = 0; b < 8; ++b) {
        const int c = symmod(v, p);
        if (b / 4 == word) w |= (uint32_t)(c & 255) << (8 * (b % 4));
        v = (v * 256) % p;
    }
    return w;
}
constexpr int64_t powmod2(int e, int p) {
    int64_t v = 1 % p;
    for (int k = 0; k < e; ++k) v = v * 2 % p;
    return v;
}
constexpr int MAGIC = 0x4B400000;  // bits of 1.5 2^23: MAGIC + v are those of 1.5 2^23 + v, |v| < 2^22
constexpr int OFF_EXP = 63;        // integers are shifted by 2^63 to be positive

// (P / MOD[l])^-1 mod MOD[l]
constexpr int crt_inv(int l) {
    int64_t q = 1;
    for (int m = 0; m < MG_N; ++m)
        if (m != l) q = q * MOD[m] % MOD[l];
    for (int i = 1; i < MOD[l]; ++i)
        if (q * i % MOD[l] == 1) return i;
    return 0;
}

// The remainder theorem in fractions: x / P = sum_l r_l inv_l / p_l (mod 1).
// F_l = inv_l / p_l rounded to 72 bits: the sum's error, 2^-64.6 on average, and
// that of the 64 bits that are kept, 2^-65.8, are below 2^-61.3 |x| |y| / P even
// where the rows' norms are the smallest that mg_scale leaves.  Byte b of four
// F_l is a word, so four terms of the sum's byte b are one dp4a, and the sum is
// nine 20-bit integers.
// (In FP64, on pairs of moduli, the same took 30 FP64 instructions per element,
// which share their pipe with the tensor core: at K = 700 as long as a third of
// its products.)
constexpr int FB = 9;                      // bytes of F_l
constexpr int NG = MG_N / 4;               // groups of four moduli
struct Crt {
    uint32_t f[FB][NG];
    double p64;  // P / 2^64
};
constexpr Crt make_crt() {
    Crt c{};
    for (int l = 0; l < MG_N; ++l) {
        const unsigned __int128 f = (((unsigned __int128)crt_inv(l) << (8 * FB)) + MOD[l] / 2) / (unsigned)MOD[l];
        for (int b = 0; b < FB; ++b) c.f[b][l / 4] |= (uint32_t)(uint8_t)(f >> (8 * b)) << (8 * (l % 4));
    }
    unsigned __int128 P = 1;
    for (int l = 0; l < MG_N; ++l) P *= (unsigned)MOD[l];
    c.p64 = (double)(uint64_t)(P >> 64) + (double)(uint64_t)P / 18446744073709551616.0;
    return c;
}
static_assert(make_crt().p64 > 1.166 * 2305843009213693952.0 && make_crt().p64 < 1.168 * 2305843009213693952.0,
              "P = 1.167 2^125: |x| <= 2^124.2 < P / 2");
__constant__ Crt c_crt = make_crt();

// The element whose residues (unsigned bytes, any representatives) are the
// bytes of r[0..NG-1], as x / P * 2^64.
__device__ __forceinline__ double crt_element(const uint32_t (&r)[NG]) {
    uint32_t a[FB];
#pragma unroll
    for (int b = 0; b < FB; ++b) {
        a[b] = b ? 0 : 128;  // the byte that is dropped rounds to nearest
#pragma unroll
        for (int g = 0; g < NG; ++g) a[b] = __dp4a(r[g], c_crt.f[b][g], a[b]);
    }
    // (sum_b a_b 2^(8 b)) / 2^8 modulo 2^64
    const uint32_t g0 = (a[0] >> 8) + a[1] + (a[2] << 8), g1 = a[3] + (a[4] << 8);
    const uint32_t g2 = a[5] + (a[6] << 8), g3 = a[7] + (a[8] << 8);
    const uint64_t t = (uint64_t)g1 * 65536u + g0;
    const uint32_t lo = (uint32_t)t, hi = (uint32_t)(t >> 32) + g2 + (g3 << 16);
    return tc::i64_to_f64((int)hi, lo);
}

// floor(c / p) = (c * m) >> 38 with m = floor(2^38 / p) + 1 for 0 <= c < 2^30;
// for -2^30 < c < 0 it is one less where p divides c, which leaves the residue
// p instead of 0.
struct ModTab {
    int m[MG_N], p[MG_N];
};
constexpr ModTab make_modtab() {
    ModTab t{};
    for (int l = 0; l < MG_N; ++l) {
        t.m[l] = (int)((int64_t(1) << 38) / MOD[l] + (MOD[l] == 256 ? 0 : 1));
        t.p[l] = MOD[l];
    }
    return t;
}
__constant__ ModTab c_mod = make_modtab();

__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// The residue (low byte, two's complement, |r| <= p / 2) of the integer whose
// shifted form is hi:lo: the bytes' weighted sum v (|v| < 2^18.1) in two
// dp4a, then v - p rint(v / p); v / p is at least 1 / (2 p) away from a tie,
// the FP32 quotient within 2^-13.
template <int L>
__device__ __forceinline__ uint32_t residue(uint32_t lo, uint32_t hi) {
    constexpr int p = MOD[L];
    constexpr uint32_t cl = coef(p, 0), ch = coef(p, 1);
    constexpr int init = MAGIC + symmod(-powmod2(OFF_EXP, p), p);
    constexpr float inv = 1.0f / (float)p;
    const int b = dp4a_us(hi, ch, dp4a_us(lo, cl, init));
    const float t = __fmaf_rn(__int_as_float(b) - 12582912.0f, inv, 12582912.0f);
    return (uint32_t)(b - __float_as_int(t) * p);
}

template <int L>
__device__ __forceinline__ void store_residues(const uint32_t (&lo)[16], const uint32_t (&hi)[16], int8_t* dst,
                                               int64_t plane) {
    if constexpr (L < MG_N) {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t a = __byte_perm(residue<L>(lo[4 * q], hi[4 * q]), residue<L>(lo[4 * q + 1], hi[4 * q + 1]),
                                           0x0040);
            const uint32_t b = __byte_perm(residue<L>(lo[4 * q + 2], hi[4 * q + 2]),
                                           residue<L>(lo[4 * q + 3], hi[4 * q + 3]), 0x0040);
            w[q] = __byte_perm(a, b, 0x5410);
        }
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        store_residues<L + 1>(lo, hi, dst + plane, plane);
    }
}

// 16 consecutive k of one operand row: x(i) -> residues at dst (16-byte
// aligned), planes `plane` bytes apart.
template <class F>
__device__ __forceinline__ void convert16(const F& x, double inv_scale, int8_t* dst, int64_t plane) {
    uint32_t lo[16], hi[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const unsigned long long v = (unsigned long long)__double2ll_rn(x(i) * inv_scale) + (1ull << OFF_EXP);
        lo[i] = (uint32_t)v;
        hi[i] = (uint32_t)(v >> 32);
    }
    store_residues<0>(lo, hi, dst, plane);
}

// Scale of a row with squared norm n2: the power of two s with n2 / s^2 in
// (2^122.2, 2^124.2]; 0 where the row is out of range (also NaN; `abs`, the sum
// of |x|, tells a row of zeros from one whose squares underflow).
__device__ __forceinline__ double mg_scale(double abs, double n2) {
    if (abs == 0.0) return 1.0;
    if (!(n2 >= 1e-140 && n2 <= 1e140)) return 0.0;
    int k;
    const double f = frexp(n2, &k);  // n2 = f 2^k, f in [0.5, 1)
    int e = (124 - k) >> 1;          // n2 4^e < 2^124
    const int up = k + 2 * (e + 1);  // n2 4^(e+1) = f 2^up, up = 125 or 126
    if (up == 125 && f <= 0.5743) ++e;  // 0.5743 2^125 < 2^124.2
    return ldexp(1.0, -e);
}

// Sums over the lanes of a warp of eight values each: lane l gets that of
// v[l / 4], in nine exchanges instead of forty.
__device__ __forceinline__ double warp_sum8(double (&v)[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = 4, o = 16; w > 0; w >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const double send = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    double s = v[0];
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// Partial (sum |x|, sum x^2) of the rows over 128 columns, rowp[column tile][R],
// and of the columns over 128 rows, colp[row tile][C], in one read of x.
__global__ void __launch_bounds__(256) mg_stats_kernel(const double* __restrict__ x, int64_t ld, int64_t R, int64_t C,
                                                       double2* __restrict__ rowp, double2* __restrict__ colp,
                                                       const int* bad) {
    __shared__ double2 sh[8][128];
    if (*bad) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t c0 = (int64_t)blockIdx.x * 128 + lane, r0 = (int64_t)blockIdx.y * 128 + warp * 16;
    double ca[4] = {}, cq[4] = {};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        double a[8], q[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int64_t r = r0 + 8 * h + i;
            double v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = r < R && c0 + 32 * j < C ? x[r * ld + c0 + 32 * j] : 0.0;
            a[i] = q[i] = 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double w = fabs(v[j]);
                a[i] += w;
                q[i] = fma(w, w, q[i]);
                ca[j] += w;
                cq[j] = fma(w, w, cq[j]);
            }
        }
        const double sa = warp_sum8(a), sq = warp_sum8(q);
        const int64_t r = r0 + 8 * h + (lane >> 2);
        if ((lane & 3) == 0 && r < R) rowp[(int64_t)blockIdx.x * R + r] = make_double2(sa, sq);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) sh[warp][lane + 32 * j] = make_double2(ca[j], cq[j]);
    __syncthreads();
    const int64_t c = (int64_t)blockIdx.x * 128 + threadIdx.x;
    if (threadIdx.x < 128 && c < C) {
        double2 s = sh[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            s.x += sh[w][threadIdx.x].x;
            s.y += sh[w][threadIdx.x].y;
        }
        colp[(int64_t)blockIdx.y * C + c] = s;
    }
}

// Lanes that add up one entry's tiles: few tiles leave most of a warp idle.
__host__ __device__ inline int fold_lanes(int64_t tiles) { return tiles > 32 ? 32 : 4; }

// sum over the tiles of part[tile][n] for entry e (0 past the last), L lanes each.
__device__ __forceinline__ double2 fold_tiles(const double2* __restrict__ part, int64_t tiles, int64_t n, int64_t e,
                                              int L) {
    double2 s = make_double2(0.0, 0.0);
    if (e < n)
        for (int64_t t = threadIdx.x & (L - 1); t < tiles; t += L) {
            const double2 v = part[t * n + e];
            s.x += v.x;
            s.y += v.y;
        }
    for (int o = L >> 1; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    return s;
}

// The sums and scales along each axis (blockIdx.y), and from the shorter one
// the squared Frobenius norm's partial sums.
__global__ void __launch_bounds__(256) mg_stats_fold_kernel(const double2* __restrict__ rowp,
                                                            const double2* __restrict__ colp, const MgMat x,
                                                            const int* bad) {
    __shared__ double red[32];
    const int axis = blockIdx.y;
    const double2* part = axis ? colp : rowp;
    if (*bad) return;
    const int64_t tiles = (x.n[1 - axis] + 127) / 128;
    const int L = fold_lanes(tiles), t = threadIdx.x;
    const int64_t e = (int64_t)blockIdx.x * (256 / L) + t / L;
    if (e - t / L >= x.n[axis]) return;
    const double2 s = fold_tiles(part, tiles, x.n[axis], e, L);
    const bool lead = (t & (L - 1)) == 0 && e < x.n[axis];
    if (lead) {
        x.sum[axis][e] = s;
        x.scale[axis][e] = mg_scale(s.x, s.y);
    }
    if (axis != x.short_axis()) return;
    const double f = block_sum(lead ? s.y : 0.0, red);
    if (t == 0) x.f2[blockIdx.x] = f;
}

// The guard's left side for the operand rows along `axis` of x: with the
// partner's sums S_k = sum_n |y_nk|, T_k = sum_n y_nk^2,
//     sum_n (sum_k |x_k y_nk|)^2 >= max((sum_k |x_k| S_k)^2 / N, sum_k x_k^2 T_k).
// part[tile][rows]: those two sums over the k of a tile.
__global__ void __launch_bounds__(256) mg_guard_fold_kernel(const double2* __restrict__ part, int64_t tiles,
                                                            MgMat x, int axis, MgMat y, int py, int* bad) {
    __shared__ double red[32];
    double f = 0.0;
    const int64_t fa = y.short_axis(), fe = 256 / fold_lanes((y.n[1 - fa] + 127) / 128);
    for (int64_t k = threadIdx.x; k < (y.n[fa] + fe - 1) / fe; k += 256) f += y.f2[k];
    f = block_sum(f, red);
    if (threadIdx.x == 0) red[0] = f;
    __syncthreads();
    const int L = fold_lanes(tiles);
    const int64_t r = (int64_t)blockIdx.x * (256 / L) + threadIdx.x / L;
    const double2 s = fold_tiles(part, tiles, x.n[axis], r, L);
    const double low = fmax(s.x * s.x / (double)y.n[py], s.y);
    if (r < x.n[axis] && low < MG_GUARD * MG_GUARD * x.sum[axis][r].y * red[0]) *bad = 1;
}

// Rows of x -> residues (WRITE), and the guard's sums against the partner's
// (GUARD).  A warp takes 512 k of one row: coalesced loads into its
// shared-memory strip (one double of padding per 16, so the 16 k a lane then
// reads lie in other banks than its neighbours'), 16 bytes of each plane per
// lane.  Bound by the integer pipes: about 110 instructions per element.  The
// warps of a CTA take the same k of eight rows, so the partner's sums come
// from L1.
template <bool WRITE, bool GUARD>
__global__ void __launch_bounds__(256, 4) mg_rows_kernel(const MgMat x, int64_t kp, const double2* __restrict__ ys,
                                                         double2* __restrict__ part, int8_t* __restrict__ out,
                                                         int* bad) {
    __shared__ double sm[WRITE ? 8 : 1][512 + 32];
    const int64_t R = x.n[0], K = x.n[1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t r = (int64_t)blockIdx.x * 8 + warp, k0 = (int64_t)blockIdx.y * 512;
    if (*bad || r >= R) return;
    const double* row = x.p + r * x.ld;
    double* s = sm[WRITE ? warp : 0];
    double l1 = 0.0, l2 = 0.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int k = i * 32 + lane;
        const double v = k0 + k < K ? row[k0 + k] : 0.0;
        if (WRITE) s[k + (k >> 4)] = v;
        if (GUARD && k0 + k < K) {
            const double2 t = ys[k0 + k];
            l1 = fma(fabs(v), t.x, l1);
            l2 = fma(v * v, t.y, l2);
        }
    }
    if (GUARD) {
        l1 = warp_sum(l1);
        l2 = warp_sum(l2);
        if (lane == 0) part[(int64_t)blockIdx.y * R + r] = make_double2(l1, l2);
    }
    if constexpr (WRITE) {
        const double scale = x.scale[0][r];
        if (!(scale > 0.0)) {
            if (lane == 0) *bad = 1;
            return;
        }
        __syncwarp();
        const int64_t kk = k0 + lane * 16;
        if (kk >= kp) return;
        const double* mine = s + lane * 17;
        convert16([&](int i) { return mine[i]; }, 1.0 / scale, out + r * kp + kk, R * kp);
    }
}

// Columns of x (K x R) -> residues: a CTA takes 32 columns by 128 k through
// shared memory (columns rotated by 4 per 16 k against bank conflicts).
template <bool WRITE, bool GUARD>
__global__ void __launch_bounds__(256, 4) mg_cols_kernel(const MgMat x, int64_t kp, const double2* __restrict__ ys,
                                                         double2* __restrict__ part, int8_t* __restrict__ out,
                                                         int* bad) {
    __shared__ double sm[WRITE ? 128 * 32 : 1];
    __shared__ double2 sg[GUARD ? 8 : 1][32];
    if (__syncthreads_or(*bad)) return;  // (another CTA may raise it meanwhile)
    const int64_t R = x.n[1], K = x.n[0];
    const int64_t c0 = (int64_t)blockIdx.x * 32, k0 = (int64_t)blockIdx.y * 128;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double l1 = 0.0, l2 = 0.0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int k = i * 8 + warp;
        const double v = k0 + k < K && c0 + lane < R ? x.p[(k0 + k) * x.ld + c0 + lane] : 0.0;
        if (WRITE) sm[k * 32 + ((lane + 4 * (k >> 4)) & 31)] = v;
        if (GUARD && k0 + k < K) {
            const double2 t = ys[k0 + k];
            l1 = fma(fabs(v), t.x, l1);
            l2 = fma(v * v, t.y, l2);
        }
    }
    if (GUARD) sg[warp][lane] = make_double2(l1, l2);
    __syncthreads();
    if (GUARD && warp == 0 && c0 + lane < R) {
        double2 t = sg[0][lane];
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            t.x += sg[GUARD ? w : 0][lane].x;
            t.y += sg[GUARD ? w : 0][lane].y;
        }
        part[(int64_t)blockIdx.y * R + c0 + lane] = t;
    }
    if constexpr (WRITE) {
        const int c = threadIdx.x >> 3, kg = threadIdx.x & 7;
        if (c0 + c >= R) return;
        const double scale = x.scale[1][c0 + c];
        if (!(scale > 0.0)) {
            *bad = 1;
            return;
        }
        const double* mine = sm + kg * 16 * 32 + ((c + 4 * kg) & 31);
        convert16([&](int i) { return mine[i * 32]; }, 1.0 / scale, out + (c0 + c) * kp + k0 + kg * 16, R * kp);
    }
}

// ------------------------------------------------------------------ GEMM --

constexpr int S = 4;
constexpr int A_BYTES = MG_BM * MG_KT, B_BYTES = MG_BN * MG_KT;  // 16 + 32 KiB
constexpr int STAGE = A_BYTES + B_BYTES;
constexpr int SMEM = S * STAGE + 1024 + 256;
constexpr int EPI_WARPS = 16;
constexpr int EPI_THREADS = 32 * EPI_WARPS;
constexpr int EPI_COLS = MG_BN / (EPI_WARPS / 4);  // columns per thread
constexpr int THREADS = 64 + EPI_THREADS;
constexpr uint32_t IDESC = tc::idesc_i8_s32(MG_BM, MG_BN);
constexpr size_t CTA_SCRATCH = (size_t)MG_N * MG_BM * MG_BN;

struct MgArgs {
    const int4* items;  // (tm, tn, first k-step, k-steps | split << 20)
    int64_t nitems;
    int M, N, planeM, planeN;
    const double* sm;  // scales of the rows of A, B
    const double* sn;
    MgOut o;
    uint32_t* scratch;
    const int* bad;
    int* err;
    WaitHooks hooks;
};

// Persistent: a CTA takes tiles of 128 x 256; per tile it runs the 16 moduli
// one after another, each over all of K, into one of two 256-column TMEM
// accumulators, so the reduction of one modulus overlaps the products of the
// next.  Sixteen warps reduce the int32 sums modulo p and park the residue
// bytes of the tile (512 KiB per CTA: 76 MB in all, which L2 holds; twice that,
// to form a tile's results under the next one's reductions, cost 23% at K =
// 4800) until the last modulus is done; then each thread reads its own bytes
// back and forms the FP64 results.  Lanes are consecutive m, so stores to
// out[n * ld + m] are coalesced.
// Bound by the int8 products at large K (4800 x 16611 x 16611: 16.05 ms, 165
// TFLOP/s FP64-equivalent) and by the epilogue below K ~ 1000.  Sixteen epilogue
// warps with the dp4a remainder theorem instead of eight with the FP64 one: 5577^2
// x 700 0.54 -> 0.48 ms, 16384^2 x 2150 8.0 -> 7.55 (15 moduli; the sixteenth costs
// 5-7%: 2150 x 16384 x 16384 6.74 -> 7.21 ms, 700 x 5577 x 5577 0.286 -> 0.303).
__global__ void __launch_bounds__(THREADS, 1)
    mg_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const MgArgs p) {
    if (*p.bad) return;  // the product is not used
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_u32 = smem_u32(smem_raw);
    const uint32_t base_u32 = (raw_u32 + 1023u) & ~1023u;
    uint8_t* base = smem_raw + (base_u32 - raw_u32);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + S * STAGE);
    uint64_t* full = bars;
    uint64_t* empty = bars + S;
    uint64_t* tfull = bars + 2 * S;       // [2]
    uint64_t* tempty = bars + 2 * S + 2;  // [2]
    uint64_t* drain = bars + 2 * S + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 5);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&tfull[b], 1);
            tc::mbar_init(&tempty[b], EPI_THREADS);
        }
        tc::mbar_init(drain, 1);
        *abort_flag = 0;
        tc::fence_barrier_init();
    }
    if (warp == 0 && lane == 0) {
        tc::prefetch_tmap(&tmA);
        tc::prefetch_tmap(&tmB);
    }
    if (warp == 1) {
        tc::tmem_alloc(tmem_slot, 512);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t g = 0;
            const bool drop = p.hooks.drop_load && blockIdx.x == 0;  // stage g == 0 gets no load
            for (int64_t t = blockIdx.x; t < p.nitems && !*abort_flag; t += gridDim.x) {
                const int4 it = p.items[t];
                const int nk = it.w & 0xfffff;
                for (int l = 0; l < MG_N; ++l)
                    for (int kt = 0; kt < nk; ++kt, ++g) {
                        const int s = g % S;
                        if (!tc::mbar_wait(&empty[s], ((g / S) & 1) ^ 1, abort_flag, p.err)) goto prod_done;
                        if (drop && g == 0) continue;
                        tc::mbar_arrive_expect_tx(&full[s], STAGE);
                        uint8_t* st = base + s * STAGE;
                        tc::tma_load_2d(st, &tmA, &full[s], (it.z + kt) * MG_KT, l * p.planeM + it.x * MG_BM);
                        tc::tma_load_2d(st + A_BYTES, &tmB, &full[s], (it.z + kt) * MG_KT, l * p.planeN + it.y * MG_BN);
                    }
            }
        prod_done:
            // the loads in flight land before the CTA leaves (a dropped stage has none)
            for (uint32_t q = 0; q < (uint32_t)S && q < g; ++q) {
                const uint32_t gg = g - 1 - q;
                if (drop && gg == 0) continue;
                int no_abort = 0;
                tc::mbar_wait(&full[gg % S], (gg / S) & 1, &no_abort, p.err);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t g = 0, c = 0;
            for (int64_t t = blockIdx.x; t < p.nitems && !*abort_flag; t += gridDim.x) {
                const int nk = p.items[t].w & 0xfffff;
                for (int l = 0; l < MG_N; ++l, ++c) {
                    const uint32_t b = c & 1;
                    if (!tc::mbar_wait(&tempty[b], ((c >> 1) & 1) ^ 1, abort_flag, p.err)) goto mma_done;
                    tc::fence_after_sync();
                    for (int kt = 0; kt < nk; ++kt, ++g) {
                        const int s = g % S;
                        if (!tc::mbar_wait(&full[s], (g / S) & 1, abort_flag, p.err, p.hooks.wait_ns)) goto mma_done;
                        tc::fence_after_sync();
                        const uint64_t da = tc::sdesc_k128(base_u32 + s * STAGE);
                        const uint64_t db = tc::sdesc_k128(base_u32 + s * STAGE + A_BYTES);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            tc::umma_i8(tmem_base + b * 256, da + 2 * k, db + 2 * k, IDESC, (kt | k) != 0);
                        tc::umma_commit(&empty[s]);
                    }
                    tc::umma_commit(&tfull[b]);
                }
            }
        mma_done:
            tc::umma_commit(drain);
            int no_abort = 0;
            tc::mbar_wait(drain, 0, &no_abort, p.err);
        }
        __syncwarp();
    } else {
        // thread = TMEM lane (row) and a range of 64 columns; the bytes of four
        // columns are a word, a warp's words are consecutive
        const int q = warp & 3, h = (warp - 2) >> 2;
        const int row = q * 32 + lane;
        uint32_t* scr = p.scratch + (int64_t)blockIdx.x * (CTA_SCRATCH / 4) + (tid - 64);
        const uint32_t tl0 = tmem_base + ((uint32_t)(q * 32) << 16) + h * EPI_COLS;
        uint32_t c = 0;
        bool ok = true;
        for (int64_t t = blockIdx.x; t < p.nitems && ok; t += gridDim.x) {
            const int4 it = p.items[t];
            for (int l = 0; l < MG_N; ++l, ++c) {
                const uint32_t b = c & 1;
                if (!tc::mbar_wait(&tfull[b], (c >> 1) & 1, abort_flag, p.err)) {
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const int mm = c_mod.m[l], pp = c_mod.p[l];
                // 16 columns at a time, the next ones on their way meanwhile
                float v[2][16];
                tc::tmem_ld16(tl0 + b * 256, v[0]);
                tc::tmem_wait_ld();
#pragma unroll
                for (int cg = 0; cg < EPI_COLS / 16; ++cg) {
                    if (cg + 1 < EPI_COLS / 16) tc::tmem_ld16(tl0 + b * 256 + (cg + 1) * 16, v[(cg + 1) & 1]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t r[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int x = __float_as_int(v[cg & 1][4 * j + u]);
                            r[u] = (uint32_t)(x - (__mulhi(x, mm) >> 6) * pp);
                        }
                        __stcg(scr + (l * (EPI_COLS / 4) + 4 * cg + j) * EPI_THREADS,
                               __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410));
                    }
                    if (cg + 1 < EPI_COLS / 16) tc::tmem_wait_ld();
                }
                tc::fence_before_sync();
                tc::mbar_arrive(&tempty[b]);
            }
            if (!ok) break;
            const int m = it.x * MG_BM + row;
            const bool vm = m < p.M;
            const double sr = vm ? p.o.alpha * c_crt.p64 * p.sm[m] : 0.0;
            const int n00 = it.y * MG_BN + h * EPI_COLS, left = p.N - n00;
            double* o = p.o.out + (int64_t)(it.w >> 20) * p.o.split_stride + (int64_t)n00 * p.o.ld + m;
            const int ng = left >= EPI_COLS ? EPI_COLS / 4 : left > 0 ? (left + 3) / 4 : 0;
            uint32_t w[MG_N];
            if (ng > 0) {
#pragma unroll
                for (int l = 0; l < MG_N; ++l) w[l] = __ldcg(scr + l * (EPI_COLS / 4) * EPI_THREADS);
            }
#pragma unroll 1
            for (int cg = 0; cg < ng; ++cg) {
                uint32_t x[MG_N];
                const int nx = cg + 1 < ng ? cg + 1 : cg;
#pragma unroll
                for (int l = 0; l < MG_N; ++l) {
                    x[l] = w[l];
                    w[l] = __ldcg(scr + (l * (EPI_COLS / 4) + nx) * EPI_THREADS);
                }
                double old[4], sc[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool vn = vm && cg * 4 + j < left;
                    old[j] = p.o.accumulate && vn ? o[(int64_t)(cg * 4 + j) * p.o.ld] : 0.0;
                    sc[j] = vn ? sr * p.sn[n00 + cg * 4 + j] : 0.0;
                }
                // byte j of four moduli's words -> the words of element j
                uint32_t e[4][NG];
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    const uint32_t a0 = x[4 * g], a1 = x[4 * g + 1], a2 = x[4 * g + 2], a3 = x[4 * g + 3];
                    const uint32_t t0 = __byte_perm(a0, a1, 0x5140), t1 = __byte_perm(a0, a1, 0x7362);
                    const uint32_t u0 = __byte_perm(a2, a3, 0x5140), u1 = __byte_perm(a2, a3, 0x7362);
                    e[0][g] = __byte_perm(t0, u0, 0x5410);
                    e[1][g] = __byte_perm(t0, u0, 0x7632);
                    e[2][g] = __byte_perm(t1, u1, 0x5410);
                    e[3][g] = __byte_perm(t1, u1, 0x7632);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (vm && cg * 4 + j < left) o[(int64_t)(cg * 4 + j) * p.o.ld] = __fma_rn(crt_element(e[j]), sc[j], old[j]);
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 1) {
        __syncwarp();
        tc::tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace

MgMat mg_mat(const double* p, int64_t ld, int64_t R, int64_t C, double* stat) {
    MgMat x;
    x.p = p;
    x.ld = ld;
    x.n[0] = R;
    x.n[1] = C;
    x.sum[0] = (double2*)stat;
    x.sum[1] = x.sum[0] + R;
    x.scale[0] = stat + 2 * (R + C);
    x.scale[1] = x.scale[0] + R;
    x.f2 = x.scale[1] + C;
    return x;
}

fc_status mg_stats(const MgMat& x, double* part, const int* bad, cudaStream_t st) {
    const int64_t R = x.n[0], C = x.n[1], tc = (C + 127) / 128, tr = (R + 127) / 128;
    double2 *rowp = (double2*)part, *colp = rowp + R * tc;
    mg_stats_kernel<<<dim3((unsigned)tc, (unsigned)tr), 256, 0, st>>>(x.p, x.ld, R, C, rowp, colp, bad);
    const int64_t pr = 256 / fold_lanes(tc), pc = 256 / fold_lanes(tr);
    const dim3 g((unsigned)std::max((R + pr - 1) / pr, (C + pc - 1) / pc), 2);
    mg_stats_fold_kernel<<<g, 256, 0, st>>>(rowp, colp, x, bad);
    return check_launch("residue sums");
}

// One pass over x: residues (r) and, with y, the guard's sums and their check.
static fc_status mg_pass(const MgMat& x, int axis, int8_t* r, const MgMat* y, int py, double* part, int* bad,
                         cudaStream_t st) {
    const int64_t R = x.n[axis], K = x.n[1 - axis], kp = mg_kp(K);
    const double2* ys = y ? y->sum[1 - py] : nullptr;
    double2* gp = (double2*)part;
    const int64_t tiles = axis ? kp / 128 : (kp + 511) / 512;
    const dim3 g((unsigned)(axis ? (R + 31) / 32 : (R + 7) / 8), (unsigned)tiles);
    if (axis) {
        if (r && y) mg_cols_kernel<true, true><<<g, 256, 0, st>>>(x, kp, ys, gp, r, bad);
        else if (r) mg_cols_kernel<true, false><<<g, 256, 0, st>>>(x, kp, ys, gp, r, bad);
        else mg_cols_kernel<false, true><<<g, 256, 0, st>>>(x, kp, ys, gp, r, bad);
    } else {
        if (r && y) mg_rows_kernel<true, true><<<g, 256, 0, st>>>(x, kp, ys, gp, r, bad);
        else if (r) mg_rows_kernel<true, false><<<g, 256, 0, st>>>(x, kp, ys, gp, r, bad);
        else mg_rows_kernel<false, true><<<g, 256, 0, st>>>(x, kp, ys, gp, r, bad);
    }
    const int64_t per = 256 / fold_lanes(tiles);
    if (y) mg_guard_fold_kernel<<<(unsigned)((R + per - 1) / per), 256, 0, st>>>(gp, tiles, x, axis, *y, py, bad);
    return check_launch("residue conversion");
}

fc_status mg_convert(const MgMat& x, int axis, int8_t* r, const MgMat* y, int py, double* part, int* bad,
                     cudaStream_t st, MgOperand* o) {
    const int64_t R = x.n[axis], K = x.n[1 - axis];
    *o = MgOperand{r, x.scale[axis], R, K, mg_kp(K), R};
    return mg_pass(x, axis, r, y, py, part, bad, st);
}

fc_status mg_guard(const MgMat& x, int axis, const MgMat& y, int py, double* part, int* bad, cudaStream_t st) {
    return mg_pass(x, axis, nullptr, &y, py, part, bad, st);
}

// Tile c of the product in launch order: split-major, then groups of GM m-tiles,
// n-major within a group (16 x 9 tiles in flight: 2048 x 2304 of the product,
// whose operands the CTAs share in L2).
struct TileGrid {
    static constexpr int GM = 16;
    int ntm, ntn, nks, kps, upper;
    __host__ __device__ int64_t count() const { return (int64_t)ntm * ntn * ((nks + kps - 1) / kps); }
    __host__ __device__ bool at(int64_t c, int4* it) const {
        const int s = (int)(c / ((int64_t)ntm * ntn));
        const int64_t r = c % ((int64_t)ntm * ntn);
        const int g = (int)(r / ((int64_t)GM * ntn)), q = (int)(r % ((int64_t)GM * ntn));
        const int gm = ntm - g * GM < GM ? ntm - g * GM : GM;
        const int tm = g * GM + q % gm, tn = q / gm;
        const int nk = nks - s * kps < kps ? nks - s * kps : kps;
        *it = make_int4(tm, tn, s * kps, nk | (s << 20));
        return !upper || (int64_t)tm * MG_BM + MG_BM - 1 >= (int64_t)tn * MG_BN;
    }
};

static TileGrid tile_grid(int64_t M, int64_t N, int64_t K, bool upper, int splits) {
    const int nks = (int)(mg_kp(K) / MG_KT);
    return {(int)((M + MG_BM - 1) / MG_BM), (int)((N + MG_BN - 1) / MG_BN), nks, (nks + splits - 1) / splits, upper};
}

int64_t mg_tiles(int64_t M, int64_t N, int64_t K, bool upper, int splits, std::vector<int4>* items) {
    const TileGrid g = tile_grid(M, N, K, upper, splits);
    if (!items && !upper) return g.count();
    int64_t n = 0;
    int4 it;
    for (int64_t c = 0; c < g.count(); ++c)
        if (g.at(c, &it)) {
            if (items) items->push_back(it);
            ++n;
        }
    return n;
}

// The same list written on the device: calls that return before their work is
// done copy nothing from the host.
__global__ void __launch_bounds__(1024) mg_tiles_kernel(TileGrid g, int4* __restrict__ items) {
    __shared__ int cnt[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t base = 0;
    for (int64_t c0 = 0; c0 < g.count(); c0 += 1024) {
        int4 it;
        const bool in = c0 + threadIdx.x < g.count() && g.at(c0 + threadIdx.x, &it);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) cnt[warp] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            before += w < warp ? cnt[w] : 0;
            all += cnt[w];
        }
        if (in) items[base + before + __popc(m & ((1u << lane) - 1))] = it;
        base += all;
        __syncthreads();
    }
}

size_t mg_scratch_bytes() { return CTA_SCRATCH * (size_t)ctx().sm_count; }

fc_status mg_gemm(const MgOperand& A, const MgOperand& B, const MgOut& out, const int4* items, int64_t nitems,
                  void* scratch, int* flags, cudaStream_t st) {
    static std::atomic<uint64_t> done{0};
    uint64_t bit = 0;
    if (attrs_needed(done, &bit)) {
        FC_CUDA(cudaFuncSetAttribute(mg_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        done.fetch_or(bit);
    }
    if (A.kp != B.kp || MG_N * std::max(A.plane, B.plane) + MG_BN > INT32_MAX) return fail(FC_ERR_LAYOUT, "residue GEMM: K differs or is too large");
    CUtensorMap ta, tb;
    FC_TRY(make_tmap_i8_2d(&ta, A.r, A.kp, (uint64_t)(MG_N - 1) * A.plane + A.rows, A.kp, MG_KT, MG_BM));
    FC_TRY(make_tmap_i8_2d(&tb, B.r, B.kp, (uint64_t)(MG_N - 1) * B.plane + B.rows, B.kp, MG_KT, MG_BN));
    const MgArgs a{items,   nitems,  (int)A.rows, (int)B.rows, (int)A.plane, (int)B.plane,
                   A.scale, B.scale, out, (uint32_t*)scratch, flags, flags + 1, wait_hooks()};
    const int grid = (int)std::min<int64_t>(nitems, ctx().sm_count);
    if (grid > 0)
        mg_gemm_kernel<<<grid, THREADS, SMEM, st>>>(ta, tb, a);
    return check_launch("mg_gemm_kernel");
}

__global__ void mg_fold_kernel(const double* __restrict__ part, int splits, int64_t M, int64_t N, double alpha,
                               double* __restrict__ out, int64_t ld) {
    const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (e >= M * N) return;
    double s = 0.0;
    for (int k = 0; k < splits; ++k) s += part[(int64_t)k * M * N + e];
    out[e / M * ld + e % M] = alpha * s;
}

fc_status mg_fold(const double* part, int splits, int64_t M, int64_t N, double alpha, double* out, int64_t ld,
                  cudaStream_t st) {
    mg_fold_kernel<<<(unsigned)((M * N + 255) / 256), 256, 0, st>>>(part, splits, M, N, alpha, out, ld);
    return check_launch("mg_fold_kernel");
}

fc_status mg_outcome(const int* flags, const char* what, cudaStream_t st, bool* stands) {
    int hf[2];
    FC_CUDA(cudaMemcpyAsync(hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, st));
    FC_CUDA(cudaStreamSynchronize(st));
    if (hf[1]) return fail(FC_ERR_TIMEOUT, std::string(what) + ": a pipeline wait ran out");
    *stands = !hf[0];
    return FC_OK;
}

int mg_splits(int64_t M, int64_t N, int64_t K, bool upper) {
    const int64_t tiles = std::max<int64_t>(1, mg_tiles(M, N, 1, upper, 1, nullptr)), nks = mg_kp(K) / MG_KT;
    int64_t s = std::max<int64_t>(1, std::min(ctx().sm_count / tiles, nks / 4));
    // the ranges' sums stay exact: at most MG_KMAX elements each
    const int64_t kps = std::min((nks + s - 1) / s, MG_KMAX / MG_KT);
    return (int)((nks + kps - 1) / kps);
}

fc_status mg_multiply(const MgSrc& a, const MgSrc& b, int64_t K, MgOut out, bool upper, int splits, int* flags,
                      cudaStream_t st, bool* room, double** part_out) {
    *room = false;
    const bool same = a.p == b.p && a.ld == b.ld && a.rows == b.rows && a.cols == b.cols;
    const int64_t rmax = std::max(a.rows, b.rows);
    const TileGrid g = tile_grid(a.rows, b.rows, K, upper, splits);
    // the sums over a range of K stay exact, an item's word holds its split, the launches' grids their tiles
    const int64_t gmax = 65535 * 128;
    if (std::min<int64_t>(K, (int64_t)g.kps * MG_KT) > MG_KMAX || splits > 2047 || rmax > gmax || K > gmax)
        return FC_OK;
    const int64_t items = mg_tiles(a.rows, b.rows, K, upper, splits, nullptr);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    const size_t osa = take(mg_stat_doubles(a.rows, K) * 8), osb = take(same ? 0 : mg_stat_doubles(b.rows, K) * 8);
    const size_t opart = take(mg_part_doubles(rmax, K) * 8), oitems = take(items * sizeof(int4));
    void* mg[WS_MG_SLOTS];
    const size_t results = out.out ? 0 : (splits > 1 ? splits * out.split_stride : out.ld * b.rows) * 8;
    if (!ws_get_mg({mg_bytes(a.rows, K), same ? 0 : mg_bytes(b.rows, K), 0, results, mg_scratch_bytes(), off}, mg))
        return FC_OK;
    *room = true;
    if (!out.out) *part_out = out.out = (double*)mg[3];
    char* m = (char*)mg[5];
    double* part = (double*)(m + opart);
    int4* list = (int4*)(m + oitems);
    mg_tiles_kernel<<<1, 1024, 0, st>>>(g, list);
    auto mat = [&](const MgSrc& s, size_t o) {
        return mg_mat(s.p, s.ld, s.cols ? K : s.rows, s.cols ? s.rows : K, (double*)(m + o));
    };
    const MgMat A = mat(a, osa), B = same ? A : mat(b, osb);
    FC_TRY(mg_stats(A, part, flags, st));
    if (!same) FC_TRY(mg_stats(B, part, flags, st));
    MgOperand oa, ob;
    FC_TRY(mg_convert(A, a.cols, (int8_t*)mg[0], &B, b.cols, part, flags, st, &oa));
    if (same) ob = oa;
    else FC_TRY(mg_convert(B, b.cols, (int8_t*)mg[1], &A, a.cols, part, flags, st, &ob));
    return mg_gemm(oa, ob, out, list, items, mg[4], flags, st);
}

}  // namespace fc
