// Residue conversion kernels and the tcgen05 GEMM of mgemm.cuh.
#include <algorithm>
#include <cmath>

#include "mgemm.cuh"
#include "tc.cuh"
#include "tmap.cuh"

namespace fc {

namespace {

// 15 pairwise coprime integers up to 256 (the largest ones but for the last,
// which makes their product P = 2^117.75 an FP64 number within 2^-56.7).
constexpr int MOD[MG_N] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 193};

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
constexpr int OFF_EXP = 60;        // integers are shifted by 2^60 to be positive

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
// F_l = inv_l / p_l rounded to 72 bits: the sum's error, 2^-64 on average, is a
// sixteenth of the operands' rounding.  Byte b of four F_l is a word, so four
// terms of the sum's byte b are one dp4a, and the sum is nine 20-bit integers.
// (In FP64, on pairs of moduli, the same took 30 FP64 instructions per element,
// which share their pipe with the tensor core: at K = 700 as long as a third of
// its products.)
constexpr int FB = 9;                      // bytes of F_l
constexpr int NG = (MG_N + 3) / 4;         // groups of four moduli
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
static_assert(make_crt().p64 > 0.83 * 18014398509481984.0 && make_crt().p64 < 0.85 * 18014398509481984.0,
              "P = 0.84 2^118: |x| <= 2^116.7 < P / 2");
__constant__ Crt c_crt = make_crt();

// The element whose residues (unsigned bytes, any representatives) are the
// bytes of r[0..NG-1], as x / P * 2^64.
__device__ __forceinline__ double crt_element(const uint32_t (&r)[NG]) {
    uint32_t a[FB];
#pragma unroll
    for (int b = 0; b < FB; ++b) {
        a[b] = 0;
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
        const long long v = __double2ll_rn(x(i) * inv_scale) + (1ll << OFF_EXP);
        lo[i] = (uint32_t)v;
        hi[i] = (uint32_t)((unsigned long long)v >> 32);
    }
    store_residues<0>(lo, hi, dst, plane);
}

// Scale of a row with squared norm n2: the power of two s with
// n2 / s^2 in (2^114.7, 2^116.7].
__device__ __forceinline__ double mg_scale(double n2, int* bad) {
    if (n2 == 0.0) return 1.0;
    if (!(n2 >= 1e-200 && n2 <= 1e200)) {  // also NaN
        *bad = 1;
        return 1.0;
    }
    int k;
    const double f = frexp(n2, &k);  // n2 = f 2^k, f in [0.5, 1)
    int e = (116 - k) >> 1;          // n2 4^e < 2^116
    const int up = k + 2 * (e + 1);  // n2 4^(e+1) = f 2^up, up = 117 or 118
    if (up == 117 && f <= 0.8122) ++e;  // 0.8122 2^117 < 2^116.7
    return ldexp(1.0, -e);
}

// Scales of the rows from their 2-norms, summed in a fixed order: one warp per
// row, or with WIDE a CTA of eight (few long rows: 700 x 5577 took 26 us with a
// warp each, 88 CTAs of dependent loads).
template <bool WIDE>
__global__ void __launch_bounds__(256) mg_row_scale_kernel(const double* __restrict__ x, int64_t ld, int64_t R,
                                                           int64_t K, double* __restrict__ scale, int* bad) {
    __shared__ double red[32];
    constexpr int T = WIDE ? 256 : 32;  // threads per row
    const int64_t r = WIDE ? blockIdx.x : (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= R) return;
    const int t = threadIdx.x % T;
    const double* row = x + r * ld;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int64_t k = t;
    for (; k + 3 * T < K; k += 4 * T) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = row[k + T * u];
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] += v[u] * v[u];
    }
    for (; k < K; k += T) s[0] += row[k] * row[k];
    double n2 = (s[0] + s[1]) + (s[2] + s[3]);
    if constexpr (WIDE) n2 = block_sum(n2, red);
    else n2 = warp_sum(n2);
    if (t == 0) scale[r] = mg_scale(n2, bad);
}

// Partial squared norms of the columns over 256 rows each.
__global__ void __launch_bounds__(256) mg_col_part_kernel(const double* __restrict__ x, int64_t ld, int64_t R,
                                                          int64_t K, double* __restrict__ part) {
    const int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= R) return;
    const int64_t k0 = (int64_t)blockIdx.y * 256, k1 = k0 + 256 < K ? k0 + 256 : K;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int64_t k = k0;
    for (; k + 3 < k1; k += 4) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = x[(k + u) * ld + c];
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] += v[u] * v[u];
    }
    for (; k < k1; ++k) s[0] += x[k * ld + c] * x[k * ld + c];
    part[(int64_t)blockIdx.y * R + c] = (s[0] + s[1]) + (s[2] + s[3]);
}

__global__ void __launch_bounds__(256) mg_col_scale_kernel(const double* __restrict__ part, int64_t R, int64_t nch,
                                                           double* __restrict__ scale, int* bad) {
    const int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= R) return;
    double s = 0.0;
    for (int64_t y = 0; y < nch; ++y) s += part[y * R + c];
    scale[c] = mg_scale(s, bad);
}

// Rows of x -> residues.  A warp takes 512 k of one row: coalesced loads into
// its shared-memory strip (one double of padding per 16, so the 16 k a lane
// then reads lie in other banks than its neighbours'), 16 bytes of each plane
// per lane.  Bound by the integer pipes: about 100 instructions per element.
__global__ void __launch_bounds__(256, 4) mg_rows_kernel(const double* __restrict__ x, int64_t ld, int64_t R, int64_t K,
                                                      int64_t kp, const double* __restrict__ scale,
                                                      int8_t* __restrict__ out) {
    __shared__ double sm[8][512 + 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t segs = (kp + 511) / 512;
    const int64_t id = (int64_t)blockIdx.x * 8 + warp;
    if (id >= R * segs) return;
    const int64_t r = id / segs, k0 = (id % segs) * 512;
    const double* row = x + r * ld;
    double* s = sm[warp];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int k = i * 32 + lane;
        s[k + (k >> 4)] = k0 + k < K ? row[k0 + k] : 0.0;
    }
    __syncwarp();
    const int64_t kk = k0 + lane * 16;
    if (kk >= kp) return;
    const double* mine = s + lane * 17;
    convert16([&](int i) { return mine[i]; }, 1.0 / scale[r], out + r * kp + kk, R * kp);
}

// Columns of x (K x R) -> residues: a CTA takes 32 columns by 128 k through
// shared memory (columns rotated by 4 per 16 k against bank conflicts).
__global__ void __launch_bounds__(256, 4) mg_cols_kernel(const double* __restrict__ x, int64_t ld, int64_t R, int64_t K,
                                                      int64_t kp, const double* __restrict__ scale,
                                                      int8_t* __restrict__ out) {
    __shared__ double sm[128 * 32];
    const int64_t c0 = (int64_t)blockIdx.x * 32, k0 = (int64_t)blockIdx.y * 128;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int idx = i * 256 + threadIdx.x, k = idx >> 5, c = idx & 31;
        sm[k * 32 + ((c + 4 * (k >> 4)) & 31)] = k0 + k < K && c0 + c < R ? x[(k0 + k) * ld + c0 + c] : 0.0;
    }
    __syncthreads();
    const int c = threadIdx.x >> 3, kg = threadIdx.x & 7;
    if (c0 + c >= R) return;
    const double* mine = sm + kg * 16 * 32 + ((c + 4 * kg) & 31);
    convert16([&](int i) { return mine[i * 32]; }, 1.0 / scale[c0 + c], out + (c0 + c) * kp + k0 + kg * 16, R * kp);
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
    int* err;
};

// Persistent: a CTA takes tiles of 128 x 256; per tile it runs the 15 moduli
// one after another, each over all of K, into one of two 256-column TMEM
// accumulators, so the reduction of one modulus overlaps the products of the
// next.  Sixteen warps reduce the int32 sums modulo p and park the residue
// bytes of the tile (480 KiB per CTA: 71 MB in all, which L2 holds; twice that,
// to form a tile's results under the next one's reductions, cost 23% at K =
// 4800) until the last modulus is done; then each thread reads its own bytes
// back and forms the FP64 results.  Lanes are consecutive m, so stores to
// out[n * ld + m] are coalesced.
// Bound by the int8 products at large K (16611^2 x 4800: 15.8 ms, 168 TFLOP/s
// FP64-equivalent) and by the epilogue below K ~ 1000.  Sixteen epilogue warps
// with the dp4a remainder theorem instead of eight with the FP64 one: 5577^2 x
// 700 0.54 -> 0.48 ms, 16384^2 x 2150 8.0 -> 7.55.
__global__ void __launch_bounds__(THREADS, 1)
    mg_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const MgArgs p) {
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
            for (int64_t t = blockIdx.x; t < p.nitems && !*abort_flag; t += gridDim.x) {
                const int4 it = p.items[t];
                const int nk = it.w & 0xfffff;
                for (int l = 0; l < MG_N; ++l)
                    for (int kt = 0; kt < nk; ++kt, ++g) {
                        const int s = g % S;
                        if (!tc::mbar_wait(&empty[s], ((g / S) & 1) ^ 1, abort_flag, p.err)) goto prod_done;
                        tc::mbar_arrive_expect_tx(&full[s], STAGE);
                        uint8_t* st = base + s * STAGE;
                        tc::tma_load_2d(st, &tmA, &full[s], (it.z + kt) * MG_KT, l * p.planeM + it.x * MG_BM);
                        tc::tma_load_2d(st + A_BYTES, &tmB, &full[s], (it.z + kt) * MG_KT, l * p.planeN + it.y * MG_BN);
                    }
            }
        prod_done:
            // the loads in flight land before the CTA leaves
            for (uint32_t q = 0; q < (uint32_t)S && q < g; ++q) {
                const uint32_t gg = g - 1 - q;
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
                        if (!tc::mbar_wait(&full[s], (g / S) & 1, abort_flag, p.err)) goto mma_done;
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
                    const uint32_t a0 = x[4 * g], a1 = 4 * g + 1 < MG_N ? x[4 * g + 1] : 0u;
                    const uint32_t a2 = 4 * g + 2 < MG_N ? x[4 * g + 2] : 0u, a3 = 4 * g + 3 < MG_N ? x[4 * g + 3] : 0u;
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

fc_status mg_convert_rows(const double* src, int64_t ld, int64_t R, int64_t K, MgOperand* o, int* bad,
                          cudaStream_t st) {
    o->rows = o->plane = R;
    o->K = K;
    o->kp = mg_kp(K);
    // one warp per row where that alone fills the chip's 64 warps per SM
    if (R < 64 * ctx().sm_count && K >= 1024)
        mg_row_scale_kernel<true><<<(unsigned)R, 256, 0, st>>>(src, ld, R, K, o->scale, bad);
    else
        mg_row_scale_kernel<false><<<(unsigned)((R + 7) / 8), 256, 0, st>>>(src, ld, R, K, o->scale, bad);
    const int64_t work = R * ((o->kp + 511) / 512);
    mg_rows_kernel<<<(unsigned)((work + 7) / 8), 256, 0, st>>>(src, ld, R, K, o->kp, o->scale, o->r);
    return check_launch("residue conversion (rows)");
}

fc_status mg_convert_cols(const double* src, int64_t ld, int64_t R, int64_t K, MgOperand* o, double* part, int* bad,
                          cudaStream_t st) {
    o->rows = o->plane = R;
    o->K = K;
    o->kp = mg_kp(K);
    const int64_t nch = mg_colchunks(K);
    mg_col_part_kernel<<<dim3((unsigned)((R + 255) / 256), (unsigned)nch), 256, 0, st>>>(src, ld, R, K, part);
    mg_col_scale_kernel<<<(unsigned)((R + 255) / 256), 256, 0, st>>>(part, R, nch, o->scale, bad);
    mg_cols_kernel<<<dim3((unsigned)((R + 31) / 32), (unsigned)(o->kp / 128)), 256, 0, st>>>(src, ld, R, K, o->kp,
                                                                                            o->scale, o->r);
    return check_launch("residue conversion (columns)");
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
                  void* scratch, int* err, cudaStream_t st) {
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
                   A.scale, B.scale, out, (uint32_t*)scratch, err};
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

int mg_splits(int64_t M, int64_t N, int64_t K, bool upper) {
    const int64_t tiles = std::max<int64_t>(1, mg_tiles(M, N, 1, upper, 1, nullptr)), nks = mg_kp(K) / MG_KT;
    int64_t s = std::max<int64_t>(1, std::min(ctx().sm_count / tiles, nks / 4));
    s = std::max(s, (K + MG_KMAX - 1) / MG_KMAX);  // the ranges' sums stay exact
    const int64_t kps = (nks + s - 1) / s;
    return (int)((nks + kps - 1) / kps);
}

fc_status mg_multiply(const MgSrc& a, const MgSrc& b, int64_t K, const MgOut& out, bool upper, int splits, int* flags,
                      cudaStream_t st, bool* room) {
    *room = false;
    const bool same = a.p == b.p && a.ld == b.ld && a.rows == b.rows && a.cols == b.cols;
    const int64_t seg = splits > 1 ? K : std::min<int64_t>(K, MG_KMAX / MG_KT * MG_KT);
    const int64_t rmax = std::max(a.rows, b.rows);
    if (MG_N * rmax + MG_BN > INT32_MAX || K > INT32_MAX) return FC_OK;
    const TileGrid gf = tile_grid(a.rows, b.rows, seg, upper, splits);
    const TileGrid gl = tile_grid(a.rows, b.rows, K % seg ? K % seg : seg, upper, splits);
    const int64_t nfull = mg_tiles(a.rows, b.rows, seg, upper, splits, nullptr);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    const size_t osa = take(a.rows * 8), osb = take(b.rows * 8);
    const size_t opart = take((a.cols || b.cols) ? mg_colpart(rmax, seg) * 8 : 0);
    const size_t ofull = take(nfull * sizeof(int4)), olast = take(nfull * sizeof(int4));
    void* mg[WS_MG_SLOTS];
    if (!ws_get_mg({mg_bytes(a.rows, seg), same ? 0 : mg_bytes(b.rows, seg), 0, mg_scratch_bytes(), off}, mg))
        return FC_OK;
    *room = true;
    char* m = (char*)mg[4];
    mg_tiles_kernel<<<1, 1024, 0, st>>>(gf, (int4*)(m + ofull));
    if (K % seg) mg_tiles_kernel<<<1, 1024, 0, st>>>(gl, (int4*)(m + olast));
    auto convert = [&](const MgSrc& s, void* r, size_t os, int64_t k0, int64_t k, MgOperand* o) {
        *o = MgOperand{(int8_t*)r, (double*)(m + os)};
        return s.cols ? mg_convert_cols(s.p + k0 * s.ld, s.ld, s.rows, k, o, (double*)(m + opart), flags, st)
                      : mg_convert_rows(s.p + k0, s.ld, s.rows, k, o, flags, st);
    };
    for (int64_t k0 = 0; k0 < K; k0 += seg) {
        const int64_t k = std::min(seg, K - k0);
        MgOperand A, B;
        FC_TRY(convert(a, mg[0], osa, k0, k, &A));
        if (same) B = A;
        else FC_TRY(convert(b, mg[1], osb, k0, k, &B));
        MgOut o = out;
        if (k0) o.accumulate = 1;
        const bool part = k != seg;
        FC_TRY(mg_gemm(A, B, o, (const int4*)(m + (part ? olast : ofull)), nfull, mg[3], flags + 1, st));
    }
    return FC_OK;
}

}  // namespace fc
