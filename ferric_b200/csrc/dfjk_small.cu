// DF-J and DF-K of a small molecule in one launch each (FP64).
//
// The general path runs four or five kernels per matrix whose work is a
// microsecond or two each at n = 24, naux = 139; the launches and the serial
// chain between them are the time.  Here one cluster of eight CTAs does the
// whole build: each takes an eighth of the aux rows, forms their contribution
// in shared memory, and the eight partial matrices are added up in rank order
// through distributed shared memory.
//
//   J   d_P = Bp_P . w (packed density weights, ferric-scf/src/df_j.rs:1134-1245),
//       J = sum_P Bp_P d_P
//   K   W = B_Q C for the CTA's rows, Q in groups that fit shared memory,
//       K = sum_Q W_Q W_Q^T, and optionally J's d_Q = sum_mu W_Q[mu] . C[mu]
//       followed by J as above (fc_dfjk_build_occ)
#include <cooperative_groups.h>

#include <algorithm>

#include "dfjk.cuh"
#include "dmma.cuh"

namespace cg = cooperative_groups;

namespace fc {

namespace {

constexpr int NC = 8;        // CTAs of the cluster
constexpr int T = 512;       // threads of a CTA
constexpr int NMAX = 64;     // AO functions
constexpr int OMAX = 16;     // occupied orbitals
constexpr int SMEM_MAX = 227 * 1024;

struct SmallArgs {
    const double* sq;   // (naux, n, n)
    const double* pk;   // (naux, pair)
    const double* d;    // J: density (n x n)
    const double* c;    // K: (n x nocc)
    double* j;
    double* k;
    int naux, n, pair, nocc;
};

// out[r][c] = sum over the CTAs (in rank order) of their packed partials
__device__ __forceinline__ void store_packed(cg::cluster_group& cl, double* jp, const SmallArgs& p) {
    cl.sync();
    const int rank = (int)cl.block_rank();
    for (int e = rank * T + threadIdx.x; e < p.pair; e += NC * T) {
        double s = 0.0;
#pragma unroll
        for (int r = 0; r < NC; ++r) s += cl.map_shared_rank(jp, r)[e];
        int mu = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
        while ((mu + 1) * (mu + 2) / 2 <= e) ++mu;
        while (mu * (mu + 1) / 2 > e) --mu;
        const int nu = e - mu * (mu + 1) / 2;
        p.j[mu * p.n + nu] = s;
        p.j[nu * p.n + mu] = s;
    }
    cl.sync();  // the partials stay until every CTA has read them
}

// jp[k] = sum over the CTA's rows of Bp[P, k] dq[P - q0]
__device__ __forceinline__ void j_pass2(const SmallArgs& p, int q0, int q1, const double* dq, double* jp) {
    for (int k = threadIdx.x; k < p.pair; k += T) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        int q = q0;
        for (; q + 8 <= q1; q += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = p.pk[(int64_t)(q + u) * p.pair + k];
#pragma unroll
            for (int u = 0; u < 8; ++u) s[u & 3] += v[u] * dq[q + u - q0];
        }
        for (; q < q1; ++q) s[0] += p.pk[(int64_t)q * p.pair + k] * dq[q - q0];
        jp[k] = (s[0] + s[1]) + (s[2] + s[3]);
    }
}

__global__ void __cluster_dims__(NC, 1, 1) __launch_bounds__(T) dfj_small_kernel(const SmallArgs p) {
    extern __shared__ double sm[];
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), per = (p.naux + NC - 1) / NC;
    const int q0 = min(rank * per, p.naux), q1 = min(q0 + per, p.naux);
    double* w = sm;            // [pair]
    double* jp = w + p.pair;   // [pair]
    double* dq = jp + p.pair;  // [per]
    for (int e = threadIdx.x; e < p.n * p.n; e += T) {
        const int mu = e / p.n, nu = e % p.n;
        if (nu <= mu) w[mu * (mu + 1) / 2 + nu] = nu == mu ? p.d[e] : p.d[e] + p.d[nu * p.n + mu];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int q = q0 + (threadIdx.x >> 5); q < q1; q += T / 32) {
        const double* row = p.pk + (int64_t)q * p.pair;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        int k = lane;
        for (; k + 224 < p.pair; k += 256) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = row[k + 32 * u];
#pragma unroll
            for (int u = 0; u < 8; ++u) s[u & 3] += v[u] * w[k + 32 * u];
        }
        for (; k < p.pair; k += 32) s[0] += row[k] * w[k];
        const double v = warp_sum((s[0] + s[1]) + (s[2] + s[3]));
        if (lane == 0) dq[q - q0] = v;
    }
    __syncthreads();
    j_pass2(p, q0, q1, dq, jp);
    store_packed(cl, jp, p);
}

// Shared memory of the K kernel, in doubles.  Pitches are 4 modulo 8, so the
// DMMA fragments (row g = lane / 4, k + lane % 4) are read without conflicts.
struct SmallK {
    int n, nocc, per, group;  // group: aux rows held at a time
    __host__ __device__ static int pitch(int x) { return (x + 3) / 8 * 8 + 4; }
    __host__ __device__ int op() const { return (nocc + 7) / 8 * 8; }
    __host__ __device__ int ldb() const { return pitch(n); }                  // B rows, C^T rows
    __host__ __device__ int ldw() const { return pitch(group * nocc); }       // W rows
    __host__ __device__ int pair() const { return n * (n + 1) / 2; }
    __host__ __device__ int ct() const { return 0; }                          // [op][ldb] C^T, zero padded
    __host__ __device__ int kp() const { return ct() + op() * ldb(); }        // [n][n] partial K
    __host__ __device__ int jp() const { return kp() + n * n; }               // [pair] partial J
    __host__ __device__ int dq() const { return jp() + pair(); }              // [per]
    __host__ __device__ int w() const { return dq() + per + 8; }              // [n rounded to 8][ldw] W[mu, (Q, i)]
    __host__ __device__ int b() const { return w() + (n + 7) / 8 * 8 * ldw(); }  // [group n + 7][ldb]
    __host__ __device__ int total() const { return b() + (group * n + 7) * ldb(); }
};

// K = sum_Q W_Q W_Q^T with W_Q = B_Q C.  Both products on the DMMA path: one
// warp takes eight rows (Q, mu) of the first and up to MAXT tiles 8 x 8 of K's
// upper triangle in the second (in the FMA pipe the second was bound by shared
// memory: n 64, naux 250, nocc 16 took 800 us).  The next group's B is copied
// while this one's W is multiplied.
constexpr int MAXT = 3;  // 36 tiles at n = 64 over 16 warps
__global__ void __cluster_dims__(NC, 1, 1) __launch_bounds__(T) dfk_small_kernel(const SmallArgs p, const SmallK z) {
    extern __shared__ double sm[];
    cg::cluster_group cl = cg::this_cluster();
    const int n = p.n, nocc = p.nocc, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tq = lane & 3;
    const int rank = (int)cl.block_rank();
    const int q0 = min(rank * z.per, p.naux), q1 = min(q0 + z.per, p.naux);
    const int ldb = z.ldb(), ldw = z.ldw(), kn = (n + 3) / 4 * 4;
    double *ct = sm + z.ct(), *kp = sm + z.kp(), *jp = sm + z.jp(), *dq = sm + z.dq(), *W = sm + z.w(), *B = sm + z.b();

    auto copy = [&](int qg) {  // B of the group that starts at qg
        const int nr = qg < q1 ? min(z.group, q1 - qg) * n : 0;
        const double* src = p.sq + (int64_t)qg * n * n;
        for (int r = warp; r < nr; r += T / 32)
            for (int c = lane; c < n; c += 32) cp_async8(B + r * ldb + c, src + r * n + c, true);
        cp_async_commit();
    };
    copy(q0);
    for (int e = t; e < z.op() * ldb; e += T) {
        const int i = e / ldb, nu = e % ldb;
        ct[e] = i < nocc && nu < n ? p.c[nu * nocc + i] : 0.0;
    }
    for (int r = t; r < z.group * n; r += T)
        for (int c = n; c < kn; ++c) B[r * ldb + c] = 0.0;
    // this warp's tiles of K: numbers warp, warp + 16, ... of the upper triangle
    const int nt = (n + 7) / 8;
    int tm[MAXT], tn[MAXT];
#pragma unroll
    for (int x = 0; x < MAXT; ++x) {
        int k = warp + x * (T / 32), r = 0;
        while (r < nt && k >= nt - r) k -= nt - r++;
        tm[x] = r < nt ? r : -1;
        tn[x] = r + k;
    }
    double acc[MAXT][2] = {};
    for (int qg = q0; qg < q1; qg += z.group) {
        const int nq = min(z.group, q1 - qg), nr = nq * n, L = nq * nocc, L4 = (L + 3) / 4 * 4;
        cp_async_wait<0>();
        __syncthreads();  // B, C^T, and the last group's W has been read
        for (int r0 = warp * 8; r0 < nr; r0 += T / 32 * 8) {
            double v[OMAX / 8][2] = {};
            const double* a = B + (r0 + g) * ldb + tq;
            const double* b = ct + g * ldb + tq;
            for (int k = 0; k < kn; k += 4) {
                const double af = a[k];
                dmma_8x8x4(v[0], af, b[k]);
                if (nocc > 8) dmma_8x8x4(v[1], af, b[8 * ldb + k]);
            }
            const int r = r0 + g, q = r / n, mu = r % n;
            if (r < nr) {
#pragma unroll
                for (int y = 0; y < OMAX / 8; ++y)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i = 8 * y + 2 * tq + h;
                        if (i < nocc) W[mu * ldw + q * nocc + i] = v[y][h];
                    }
            }
        }
        for (int mu = t; mu < n; mu += T)
            for (int k = L; k < L4; ++k) W[mu * ldw + k] = 0.0;
        __syncthreads();
        copy(qg + z.group);
        if (p.j) {
            for (int q = warp; q < nq; q += T / 32) {
                double s = 0.0;
                for (int mu = lane; mu < n; mu += 32)
                    for (int i = 0; i < nocc; ++i) s += W[mu * ldw + q * nocc + i] * ct[i * ldb + mu];
                s = warp_sum(s);
                if (lane == 0) dq[qg - q0 + q] = s;
            }
        }
        for (int k = 0; k < L4; k += 4) {
#pragma unroll
            for (int x = 0; x < MAXT; ++x)
                if (tm[x] >= 0)
                    dmma_8x8x4(acc[x], W[(tm[x] * 8 + g) * ldw + k + tq], W[(tn[x] * 8 + g) * ldw + k + tq]);
        }
    }
#pragma unroll
    for (int x = 0; x < MAXT; ++x)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = tm[x] * 8 + g, c = tn[x] * 8 + 2 * tq + h;
            if (tm[x] >= 0 && r < n && c < n) kp[r * n + c] = acc[x][h];
        }
    cl.sync();
    // the upper element gives both: K is exactly symmetric
    for (int e = rank * T + t; e < n * n; e += NC * T) {
        const int r = e / n, c = e % n;
        const int u = r < c ? r * n + c : c * n + r;
        double s = 0.0;
#pragma unroll
        for (int x = 0; x < NC; ++x) s += cl.map_shared_rank(kp, x)[u];
        p.k[e] = s;
    }
    if (p.j) {
        j_pass2(p, q0, q1, dq, jp);
        store_packed(cl, jp, p);
    } else {
        cl.sync();  // the partials stay until every CTA has read them
    }
}

fc_status small_attrs() {
    static std::atomic<uint64_t> done{0};
    uint64_t bit = 0;
    if (!attrs_needed(done, &bit)) return FC_OK;
    FC_CUDA(cudaFuncSetAttribute(dfj_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    FC_CUDA(cudaFuncSetAttribute(dfk_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    done.fetch_or(bit);
    return FC_OK;
}

}  // namespace

// Where one cluster beats the general path's launches (J and K, host to host):
// K at naux n^2 of 0.64 MB (n 24, naux 139) 79 -> 68.5 us, 1.4 MB 84 -> 70, 2.6 MB
// 86 -> 84.5, 3.8 MB (n 56, naux 150) 88 -> 95; J up to 4.2 MB of packed rows
// (n 64, naux 250) 23 -> 12.  The aux rows' own vector stays within shared
// memory up to 4096 of them.
bool dfj_small_fits(const fc_dfjk* h) {
    return !h->l_chol && h->n <= NMAX && h->naux <= 4096 && h->naux * h->pair * 8 <= 4 << 20;
}
bool dfk_small_fits(const fc_dfjk* h, int64_t nocc) {
    return h->b_sq && h->n <= NMAX && nocc >= 1 && nocc <= OMAX && h->naux <= 4096 &&
           h->naux * h->n * h->n * 8 <= 2 << 20;
}

fc_status dfj_small(const fc_dfjk* h, const double* d, double* j, cudaStream_t st) {
    FC_TRY(small_attrs());
    const SmallArgs a{nullptr, h->b_pk, d, nullptr, j, nullptr, (int)h->naux, (int)h->n, (int)h->pair, 0};
    const size_t smem = (2 * h->pair + (h->naux + NC - 1) / NC) * 8;
    dfj_small_kernel<<<NC, T, smem, st>>>(a);
    return check_launch("dfj_small_kernel");
}

fc_status dfk_small(const fc_dfjk* h, const double* c_occ, int64_t nocc, double* k, double* j, cudaStream_t st) {
    FC_TRY(small_attrs());
    const SmallArgs a{h->b_sq, h->b_pk, nullptr, c_occ, j, k, (int)h->naux, (int)h->n, (int)h->pair, (int)nocc};
    SmallK z{(int)h->n, (int)nocc, (int)((h->naux + NC - 1) / NC), 1};
    while (z.group < z.per) {  // as many aux rows as fit
        ++z.group;
        if (z.total() * 8 > SMEM_MAX) {
            --z.group;
            break;
        }
    }
    dfk_small_kernel<<<NC, T, (size_t)z.total() * 8, st>>>(a, z);
    return check_launch("dfk_small_kernel");
}

}  // namespace fc
