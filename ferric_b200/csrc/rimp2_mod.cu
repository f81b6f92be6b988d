// FP64 RI-MP2 with its contractions on the int8 tensor cores (mgemm.cuh).
//
// Per occupied chunk pair (I, J), I <= J:
//     G = B_I^T B_J             residue GEMM, only its upper part when I == J
//     Tt = (2 G - G^x) / D      amp_kernel, in place, with the energy and
//                               dE/deps partials (G^x: virtuals exchanged)
//     Gamma_I += 4 B_J Tt^T     residue GEMMs over the chunk's columns, and
//     Gamma_J += 4 B_I Tt       over its rows when I != J
// Every unordered pair is formed once and both of its amplitude blocks come
// from it, so the products are 2 naux nvir^2 P + 2 naux nov^2, P the number of
// unordered pairs.  The DMMA kernels of rimp2_f64.cu keep the integrals on
// chip but run at 37 TFLOP/s at most; here a GEMM runs at 142-165 TFLOP/s
// (FP64 products, adjoints at naux = 2150 and 4800) and the passes over G and Tt
// (about 10 bytes per element beside 4 naux flops) are a tenth of the time.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fc_internal.cuh"
#include "mgemm.cuh"
#include "rimp2.cuh"

namespace fc {

namespace {

constexpr int AT = 32;               // virtuals per side of an amplitude tile
constexpr int AN = 128;              // threads of its CTA
constexpr int AP = AT + 1;           // pitch in shared memory
constexpr int AE = AT * AT / AN;      // elements per thread
constexpr int AMP_SMEM = 3 * AT * AP * 8;
enum AmpMode { AMP_ENERGY, AMP_GRAD, AMP_CROSS };

struct AmpArgs {
    double* g;           // rows (i - i0, a), columns (j - j0, b), pitch ld
    int64_t ld;
    const int2* pairs;   // of this launch
    const int2* tiles;   // (ta, tb), ta <= tb (cross: all)
    int ntiles, i0, j0, nvir, nvir2;
    const double *eo, *ev, *eo2, *ev2;
    int same;            // I == J: pairs i <= j, only columns >= rows of g are given
    int has_kappa;
    double kappa;
    const int* bad;      // up: g is not used
    double* part;        // [item][3]: E_os, E_ss, sum of t Tt
    double* vir;         // [item][2 AT]: sums of t Tt by virtual of ta and of tb
};

// One (pair, tile pair) per CTA: the tiles (a in ta, b in tb) and (b, a) of
// the pair's block, so each element meets its exchange partner.  Gradient
// mode writes Tt over G (and its transpose when I == J, whose lower part the
// GEMM leaves out).  Bound by its reads and writes of g, given enough CTAs in
// flight: tiles of 64 x 64 (two CTAs per SM) ran at 1.7 TB/s.
template <int MODE>
__global__ void __launch_bounds__(AN) amp_kernel(const AmpArgs p) {
    if (*p.bad) return;
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[32];
    double* X = sm;              // X[a][b] = (ia|jb), then Tt_ij[a, b]
    double* Y = sm + AT * AP;    // Y[b][a] = (ib|ja), then Tt_ij[b, a]
    double* C = Y + AT * AP;     // t Tt of both orderings
    const int tid = threadIdx.x;
    const int64_t item = (int64_t)blockIdx.y * p.ntiles + blockIdx.x;
    const int2 ij = p.pairs[blockIdx.y], tt = p.tiles[blockIdx.x];
    const int i = ij.x, j = ij.y, A0 = tt.x * AT, B0 = tt.y * AT;
    const int nva = p.nvir, nvb = MODE == AMP_CROSS ? p.nvir2 : p.nvir;
    const int na = min(AT, nva - A0), nb = min(AT, nvb - B0);
    const bool off = A0 != B0, dia = MODE != AMP_CROSS && p.same && i == j;
    double* gx = p.g + ((int64_t)(i - p.i0) * nva + A0) * p.ld + (int64_t)(j - p.j0) * nvb + B0;
    double* gy = p.g + ((int64_t)(i - p.i0) * nva + B0) * p.ld + (int64_t)(j - p.j0) * nvb + A0;
    // each thread keeps its columns' loads together
#pragma unroll 4
    for (int e = tid; e < AT * AT; e += AN) {
        const int r = e / AT, c = e % AT;
        if (r < na && c < nb) X[r * AP + c] = gx[(int64_t)r * p.ld + c];
        if (MODE != AMP_CROSS && off && !dia && r < nb && c < na) Y[r * AP + c] = gy[(int64_t)r * p.ld + c];
    }
    __syncthreads();

    const double eij = p.eo[i] + (MODE == AMP_CROSS ? p.eo2[j] : p.eo[j]);
    const double w = MODE == AMP_CROSS ? 1.0 : i == j ? 1.0 : 2.0;
    KSum os, ss, oc;
    const int b = tid % AT;
    const bool vb = b < nb;
    const double eb = vb ? (MODE == AMP_CROSS ? p.ev2 : p.ev)[B0 + b] : 0.0;
    double t1[AE], t2[AE];
#pragma unroll
    for (int k = 0; k < AE; ++k) {
        const int a = tid / AT + (AN / AT) * k;
        t1[k] = t2[k] = 0.0;
        double s = 0.0;
        if (vb && a < na) {
            const double D = eij - p.ev[A0 + a] - eb;
            double f = 1.0 / D;
            if (MODE == AMP_ENERGY && p.has_kappa) {
                const double d1 = 1.0 - exp(p.kappa * D);
                f *= d1 * d1;
            }
            if (MODE == AMP_CROSS) {
                const double x = X[a * AP + b];
                os.add(x * x * f);
            } else {
                // the lower part of a diagonal block is the upper one's mirror
                const double x = dia && !off && a > b ? X[b * AP + a] : X[a * AP + b];
                const double y = dia ? x : off ? Y[b * AP + a] : X[b * AP + a];
                if (off) {  // the elements (a, b) and (b, a)
                    os.add((x * x + y * y) * f);
                    ss.add((x - y) * (x - y) * f);
                } else {
                    os.add(x * x * f);
                    ss.add(x * (x - y) * f);
                }
                if (MODE == AMP_GRAD) {
                    t1[k] = (2.0 * x - y) * f;
                    t2[k] = (2.0 * y - x) * f;
                    const double c1 = x * f * t1[k], c2 = y * f * t2[k];
                    oc.add(off ? c1 + c2 : c1);
                    s = i == j ? c1 : c1 + c2;  // ordering (j, i) swaps the virtuals
                }
            }
        }
        if (MODE == AMP_GRAD) C[a * AP + b] = s;
    }
    const double vos = block_sum(os.value(), red), vss = block_sum(ss.value(), red);
    const double voc = MODE == AMP_GRAD ? block_sum(oc.value(), red) : 0.0;  // (block_sum synchronises)
    if (tid == 0) {
        p.part[3 * item] = w * vos;
        p.part[3 * item + 1] = w * vss;
        p.part[3 * item + 2] = voc;
    }
    if constexpr (MODE == AMP_GRAD) {
#pragma unroll
        for (int k = 0; k < AE; ++k) {
            const int a = tid / AT + (AN / AT) * k;
            X[a * AP + b] = t1[k];
            if (off) Y[b * AP + a] = t2[k];
        }
        __syncthreads();
        if (tid < 2 * AT) {
            const int r = tid % AT;
            double s = 0.0;
            if (tid < AT) {
                for (int c = 0; c < AT; ++c) s += C[r * AP + c];
            } else if (off) {
                for (int c = 0; c < AT; ++c) s += C[c * AP + r];
            }
            p.vir[item * (2 * AT) + tid] = s;
        }
        // the mirrored blocks of a diagonal chunk pair: Tt_ji[b, a] = Tt_ij[a, b]
        double* mx = p.g + ((int64_t)(j - p.j0) * nva + B0) * p.ld + (int64_t)(i - p.i0) * nva + A0;
        double* my = p.g + ((int64_t)(j - p.j0) * nva + A0) * p.ld + (int64_t)(i - p.i0) * nva + B0;
        const bool mir = p.same && i != j;
#pragma unroll 4
        for (int e = tid; e < AT * AT; e += AN) {
            const int r = e / AT, c = e % AT;
            if (r < na && c < nb) {
                gx[(int64_t)r * p.ld + c] = X[r * AP + c];
                if (mir && off) my[(int64_t)r * p.ld + c] = Y[c * AP + r];
            }
            if (off && r < nb && c < na) gy[(int64_t)r * p.ld + c] = Y[r * AP + c];
            if (mir && r < nb && c < na) mx[(int64_t)r * p.ld + c] = X[c * AP + r];
        }
    }
}

// Sums of a pair's items, one warp per pair: psum[pair][3].
__global__ void __launch_bounds__(256) amp_pair_sum_kernel(const double* __restrict__ part, int64_t npairs, int ntiles,
                                                           double* __restrict__ psum) {
    const int64_t x = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (x >= npairs) return;
    KSum s[3];
    for (int t = threadIdx.x & 31; t < ntiles; t += 32)
#pragma unroll
        for (int k = 0; k < 3; ++k) s[k].add(part[3 * (x * ntiles + t) + k]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double v = warp_sum(s[k].value());
        if ((threadIdx.x & 31) == 0) psum[3 * x + k] = v;
    }
}

// Block 0: acc[0..1] += E_os, E_ss of all pairs; block 1 + k: acc_occ[o] += the
// t Tt sums of the pairs that hold orbital o, the k-th of chunks I and J.
__global__ void __launch_bounds__(256) amp_fold_kernel(const double* __restrict__ psum, const int2* __restrict__ pairs,
                                                       int64_t npairs, int i0, int ni, int j0, double* acc,
                                                       double* acc_occ) {
    __shared__ double red[32];
    KSum a, b;
    if (blockIdx.x == 0) {
        for (int64_t k = threadIdx.x; k < npairs; k += 256) {
            a.add(psum[3 * k]);
            b.add(psum[3 * k + 1]);
        }
        const double va = block_sum(a.value(), red), vb = block_sum(b.value(), red);
        if (threadIdx.x == 0) {
            acc[0] += va;
            acc[1] += vb;
        }
        return;
    }
    const int k0 = (int)blockIdx.x - 1, o = k0 < ni ? i0 + k0 : j0 + (k0 - ni);
    for (int64_t k = threadIdx.x; k < npairs; k += 256) {
        const int2 pr = pairs[k];
        if (pr.x == o || pr.y == o) a.add(psum[3 * k + 2]);
    }
    const double v = block_sum(a.value(), red);
    if (threadIdx.x == 0) acc_occ[o] += v;
}

// Sums of the items' virtual rows over VP pairs: out[chunk][ntile AT].
constexpr int VP = 32;
__global__ void __launch_bounds__(256) amp_vir_part_kernel(const double* __restrict__ vir, int64_t npairs, int ntile,
                                                           double* __restrict__ out) {
    constexpr int G = 256 / AT;
    __shared__ double sh[G][AT];
    const int t = blockIdx.x, r = threadIdx.x % AT, g = threadIdx.x / AT;
    const int ntiles = ntile * (ntile + 1) / 2;
    const int64_t x0 = (int64_t)blockIdx.y * VP, x1 = min(x0 + VP, npairs);
    KSum s;
    for (int64_t x = x0 + g; x < x1; x += G)
        for (int u = 0; u < ntile; ++u) {
            // tile (min, max) in the row-major list of ta <= tb
            const int lo = min(t, u), hi = max(t, u);
            const int64_t item = x * ntiles + (int64_t)lo * ntile - (int64_t)lo * (lo - 1) / 2 + (hi - lo);
            s.add(vir[item * (2 * AT) + (t <= u ? 0 : AT) + r]);
        }
    sh[g][r] = s.value();
    __syncthreads();
    if (g == 0) {
        double v = 0.0;
        for (int k = 0; k < G; ++k) v += sh[k][r];
        out[((int64_t)blockIdx.y * ntile + t) * AT + r] = v;
    }
}

// de_dvir[a] += 2 sum over the chunks, one warp per 32 virtuals and eight
// ranges of chunks.
__global__ void __launch_bounds__(256) amp_vir_fold_kernel(const double* __restrict__ part, int64_t nch, int nvir,
                                                           int pitch, double* __restrict__ de_dvir) {
    __shared__ double sh[8][32];
    const int a = blockIdx.x * 32 + (threadIdx.x & 31), g = threadIdx.x >> 5;
    KSum s;
    if (a < nvir)
        for (int64_t c = g; c < nch; c += 8) s.add(part[c * pitch + a]);
    sh[g][threadIdx.x & 31] = s.value();
    __syncthreads();
    if (g == 0 && a < nvir) {
        double v = 0.0;
        for (int k = 0; k < 8; ++k) v += sh[k][threadIdx.x & 31];
        de_dvir[a] += 2.0 * v;
    }
}

__global__ void scale_to_kernel(const double* __restrict__ x, int64_t n, double s, double* __restrict__ y) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) y[k] = s * x[k];
}

fc_status amp_attrs() {
    static std::atomic<uint64_t> done{0};
    uint64_t bit = 0;
    if (!attrs_needed(done, &bit)) return FC_OK;
    FC_CUDA(cudaFuncSetAttribute(amp_kernel<AMP_ENERGY>, cudaFuncAttributeMaxDynamicSharedMemorySize, AMP_SMEM));
    FC_CUDA(cudaFuncSetAttribute(amp_kernel<AMP_GRAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, AMP_SMEM));
    FC_CUDA(cudaFuncSetAttribute(amp_kernel<AMP_CROSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, AMP_SMEM));
    done.fetch_or(bit);
    return FC_OK;
}

// Aligned pieces of one workspace slot.
struct Carver {
    char* base = nullptr;
    size_t off = 0;
    template <class T>
    T* take(size_t n) {
        T* p = reinterpret_cast<T*>(base + off);
        off += (n * sizeof(T) + 255) & ~size_t(255);
        return p;
    }
};

int64_t balanced(int64_t n, int64_t cap) {  // chunk size of the fewest equal chunks of at most cap
    cap = std::max<int64_t>(1, std::min(cap, n));
    const int64_t k = (n + cap - 1) / cap;
    return (n + k - 1) / k;
}

struct ChunkPair {
    int64_t i0, ni, j0, nj, p0, np, t0[3], nt[3];  // first pair, pairs; tiles of G, Gamma_I, Gamma_J
    bool same() const { return i0 == j0; }
};

}  // namespace

// Where the residue form pays: the conversions (about 110 instructions per
// element), the passes over G and the launches are spread over enough
// products.  Gradient at 2 naux (nocc nvir)^2 = 1.67e9 (naux 364, nocc 17, nvir
// 89): 348 us here, 378 DMMA; at 4.7e9 435 and 570; the forms cross near 1.3e9
// (340, 16, 85: 333 and 326).
bool mod_grad_pays(int64_t naux, int64_t nocc, int64_t nvir) {
    return naux <= MG_KMAX && 2.0 * naux * (double)(nocc * nvir) * (double)(nocc * nvir) >= 1.5e9;
}

// Returns FC_OK with *ran = false where the caller has to take the DMMA form
// (no room for the residues, operand rows out of range, or a product's guard).
fc_status rimp2_grad_mod(const Rimp2Dev& d, cudaStream_t st, double* e_os, double* e_ss, double* gamma,
                         double* de_docc, double* de_dvir, fc_stats* stats, const GammaSink* sink,
                         const DensOut* dens, bool* ran) {
    *ran = false;
    FC_TRY(amp_attrs());
    const int64_t nocc = d.nocc, nvir = d.nvir, naux = d.naux, nov = nocc * nvir;
    // Tt in FP64 and the residues of its rows fit the chunk budget
    int64_t cc = 1;
    while (cc < nocc && (8 + MG_N) * (cc + 1) * nvir * (cc + 1) * nvir <= d.chunk_bytes &&
           (cc + 1) * nvir <= MG_KMAX)
        ++cc;
    if (cc * nvir > MG_KMAX) return FC_OK;
    cc = balanced(nocc, cc);
    const int64_t nch = (nocc + cc - 1) / cc, cv = cc * nvir;
    // the densities contract whole rows of t and Tt: one chunk, both kept
    if (dens && (nch > 1 || dens_chunk_f64(nocc, nvir, nocc, 4 * d.chunk_bytes) < nocc)) return FC_OK;
    const int ntile = (int)((nvir + AT - 1) / AT), ntiles = ntile * (ntile + 1) / 2;

    std::vector<ChunkPair> cps;
    std::vector<int2> hp;
    std::vector<int4> ht;
    int64_t np_max = 0;
    for (int64_t I = 0; I < nch; ++I)
        for (int64_t J = I; J < nch; ++J) {
            ChunkPair x{};
            x.i0 = I * cc;
            x.ni = std::min(cc, nocc - x.i0);
            x.j0 = J * cc;
            x.nj = std::min(cc, nocc - x.j0);
            x.p0 = (int64_t)hp.size();
            for (int64_t i = x.i0; i < x.i0 + x.ni; ++i)
                for (int64_t j = I == J ? i : x.j0; j < x.j0 + x.nj; ++j) hp.push_back(make_int2((int)i, (int)j));
            x.np = (int64_t)hp.size() - x.p0;
            np_max = std::max(np_max, x.np);
            x.t0[0] = (int64_t)ht.size();
            x.nt[0] = mg_tiles(x.nj * nvir, x.ni * nvir, naux, I == J, 1, &ht);
            x.t0[1] = (int64_t)ht.size();
            x.nt[1] = mg_tiles(x.ni * nvir, naux, x.nj * nvir, false, 1, &ht);
            x.t0[2] = (int64_t)ht.size();
            x.nt[2] = I == J ? 0 : mg_tiles(x.nj * nvir, naux, x.ni * nvir, false, 1, &ht);
            cps.push_back(x);
        }
    const int64_t npairs = (int64_t)hp.size();
    for (int ta = 0; ta < ntile; ++ta)
        for (int tb = ta; tb < ntile; ++tb) hp.push_back(make_int2(ta, tb));
    if (np_max > 65535) return FC_OK;  // the amplitude kernel's grid

    // chunk J's columns of b_ov as rows: [MG_N][naux][kp(J)]
    std::vector<MgOperand> bq((size_t)nch);
    size_t bq_bytes = 0;
    for (int64_t J = 0; J < nch; ++J) bq_bytes += mg_bytes(naux, std::min(cc, nocc - J * cc) * nvir);
    const int64_t nvch = (np_max + VP - 1) / VP;
    const size_t np_items = (size_t)np_max * ntiles;
    double *bstat, *tstat, *mpart, *part, *acc;
    std::vector<double*> qstat((size_t)nch, nullptr);  // sums of b_ov's column chunks
    int2* pairs;
    int4* items;
    const size_t out_bytes = (size_t)(nocc + 2) * 8 + 64;
    auto misc = [&](Carver& c) {
        pairs = c.take<int2>(hp.size());
        part = c.take<double>(np_items * (3 + 2 * AT) + (size_t)np_max * 3 + (size_t)nvch * ntile * AT);
        acc = c.take<double>(out_bytes / 8);
        bstat = c.take<double>(mg_stat_doubles(naux, nov));
        for (int64_t J = 0; nch > 1 && J < nch; ++J) qstat[(size_t)J] = c.take<double>(mg_stat_doubles(naux, cv));
        tstat = c.take<double>(mg_stat_doubles(cv, cv));
        mpart = c.take<double>(std::max(mg_part_doubles(naux, nov), mg_part_doubles(cv, cv)));
        items = c.take<int4>(ht.size());
    };
    // All scratch is spare memory but the densities' slabs, which the DMMA form
    // takes too (of the same size: it has one chunk where this form has one).
    DensF64 dx{};
    if (dens) FC_TRY(dens_f64_alloc(nocc, nvir, nocc, st, &dx));
    Carver cm;
    misc(cm);
    void* mg[WS_MG_SLOTS];
    if (!ws_get_mg({mg_bytes(nov, naux), bq_bytes, mg_bytes(cv, cv), dens ? 0 : (size_t)cv * cv * 8,
                    mg_scratch_bytes(), cm.off},
                   mg, dens != nullptr))
        return FC_OK;
    cm = Carver{(char*)mg[5], 0};
    misc(cm);

    double* T = dens ? dx.ts : (double*)mg[3];
    double* virp = part + 3 * np_items;
    double* psum = virp + np_items * 2 * AT;
    double* vch = psum + 3 * np_max;
    double* acc_occ = acc + 2;            // [nocc], behind E_os and E_ss
    int* flags = (int*)(acc_occ + nocc);  // out-of-range rows, wait timeout
    const int2* dpairs = pairs;
    FC_CUDA(cudaMemcpyAsync(pairs, hp.data(), hp.size() * sizeof(int2), cudaMemcpyHostToDevice, st));
    FC_CUDA(cudaMemcpyAsync(items, ht.data(), ht.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
    FC_CUDA(cudaMemsetAsync(acc, 0, out_bytes, st));
    FC_CUDA(cudaMemsetAsync(de_dvir, 0, nvir * 8, st));

    Context& c = ctx();
    const int64_t ncp = (int64_t)cps.size();
    cudaEvent_t *ev = nullptr, *ev2 = nullptr;
    if (stats) {
        FC_TRY(timing_events((int)ncp, &ev));
        FC_TRY(timing_events2((int)(2 * ncp), &ev2));
        FC_CUDA(cudaEventRecord(c.ev0, st));
    }
    const MgMat B = mg_mat(d.b_ov, nov, naux, nov, bstat);
    MgOperand bt;
    FC_TRY(mg_stats(B, mpart, flags, st));
    FC_TRY(mg_convert(B, 1, (int8_t*)mg[0], &B, 1, mpart, flags, st, &bt));
    int64_t nl = 4;
    std::vector<MgMat> bm((size_t)nch);
    int nadj = 0;
    double adj_flops = 0.0, adj_bytes = 0.0;
    size_t bq_off = 0;
    std::vector<char> seen((size_t)nch, 0);
    // Gamma[:, rows of R] (+)= 4 B_ov[:, columns of K] Tt^T, Tt's rows as residues
    auto adjoint = [&](const MgOperand& t, int64_t r0, int64_t k0, const int4* its, int64_t nits) -> fc_status {
        MgOperand& b = bq[(size_t)(k0 / cc)];
        if (stats) FC_CUDA(cudaEventRecord(ev2[2 * nadj], st));
        char& s = seen[(size_t)(r0 / cc)];
        FC_TRY(mg_gemm(t, b, MgOut{gamma + r0 * nvir, nov, 0, 4.0, s}, its, nits, mg[4], flags, st));
        s = 1;
        if (stats) FC_CUDA(cudaEventRecord(ev2[2 * nadj + 1], st));
        ++nadj;
        adj_flops += 2.0 * (double)naux * (double)t.rows * (double)t.K;
        adj_bytes += (double)MG_N * (naux + t.rows) * (double)t.K + 16.0 * (double)naux * (double)t.rows;
        return FC_OK;
    };
    for (int64_t x = 0; x < ncp; ++x) {
        const ChunkPair& cp = cps[(size_t)x];
        const int64_t J = cp.j0 / cc, ri = cp.ni * nvir, rj = cp.nj * nvir;
        if (stats) FC_CUDA(cudaEventRecord(ev[2 * x], st));
        FC_TRY(mg_gemm(bt.slice(cp.j0 * nvir, rj), bt.slice(cp.i0 * nvir, ri), MgOut{T, rj, 0, 1.0, 0},
                       items + cp.t0[0], cp.nt[0], mg[4], flags, st));
        if (stats) FC_CUDA(cudaEventRecord(ev[2 * x + 1], st));
        AmpArgs a{};
        a.g = T;
        a.ld = rj;
        a.pairs = dpairs + cp.p0;
        a.tiles = dpairs + npairs;
        a.ntiles = ntiles;
        a.i0 = (int)cp.i0;
        a.j0 = (int)cp.j0;
        a.nvir = (int)nvir;
        a.eo = d.eps_occ;
        a.ev = d.eps_vir;
        a.same = cp.same();
        a.bad = flags;
        a.part = part;
        a.vir = virp;
        amp_kernel<AMP_GRAD><<<dim3((unsigned)ntiles, (unsigned)cp.np), AN, AMP_SMEM, st>>>(a);
        amp_pair_sum_kernel<<<(unsigned)((cp.np + 7) / 8), 256, 0, st>>>(part, cp.np, ntiles, psum);
        amp_fold_kernel<<<(unsigned)(1 + cp.ni + (cp.same() ? 0 : cp.nj)), 256, 0, st>>>(
            psum, a.pairs, cp.np, (int)cp.i0, (int)cp.ni, (int)cp.j0, acc, acc_occ);
        const int64_t vc = (cp.np + VP - 1) / VP;
        amp_vir_part_kernel<<<dim3((unsigned)ntile, (unsigned)vc), 256, 0, st>>>(virp, cp.np, ntile, vch);
        amp_vir_fold_kernel<<<(unsigned)((nvir + 31) / 32), 256, 0, st>>>(vch, vc, (int)nvir, ntile * AT, de_dvir);
        FC_TRY(check_launch("residue gradient: amplitudes"));
        nl += 6;
        const MgMat tm = mg_mat(T, rj, ri, rj, tstat);
        FC_TRY(mg_stats(tm, mpart, flags, st));
        MgMat& bj = bm[(size_t)J];
        if (!bj.p) {  // first use of chunk J's columns: converted under its product's guard
            bj = nch == 1 ? B : mg_mat(d.b_ov + cp.j0 * nvir, nov, naux, rj, qstat[(size_t)J]);
            if (nch > 1) FC_TRY(mg_stats(bj, mpart, flags, st));
            FC_TRY(mg_convert(bj, 0, (int8_t*)mg[1] + bq_off, &tm, 0, mpart, flags, st, &bq[(size_t)J]));
            bq_off += mg_bytes(naux, rj);
            nl += nch > 1 ? 2 : 0;
        } else {
            FC_TRY(mg_guard(bj, 0, tm, 0, mpart, flags, st));
        }
        MgOperand t;
        FC_TRY(mg_convert(tm, 0, (int8_t*)mg[2], &bj, 0, mpart, flags, st, &t));
        FC_TRY(adjoint(t, cp.i0, cp.j0, items + cp.t0[1], cp.nt[1]));
        nl += 6;
        if (!cp.same()) {
            const MgMat& bi = bm[(size_t)(cp.i0 / cc)];
            FC_TRY(mg_guard(bi, 0, tm, 1, mpart, flags, st));
            FC_TRY(mg_convert(tm, 1, (int8_t*)mg[2], &bi, 0, mpart, flags, st, &t));
            FC_TRY(adjoint(t, cp.j0, cp.i0, items + cp.t0[2], cp.nt[2]));
            nl += 4;
        }
        // row I of the chunk pairs is done: Gamma's columns of chunk I are final
        if (sink && cp.j0 + cp.nj == nocc) FC_TRY(gamma_sink_block(sink, gamma, naux, nov, nvir, cp.i0, cp.ni, st));
    }
    if (dens) {
        FC_TRY(dens_f64_block(dx, 0, nocc, nocc, st, &nl));
        FC_TRY(dens_f64_slab(dx, nocc, st, &nl));
        FC_TRY(dens_f64_finish(dx, *dens, st, &nl));
    }
    scale_to_kernel<<<(unsigned)((nocc + 255) / 256), 256, 0, st>>>(acc_occ, nocc, -2.0, de_docc);
    FC_TRY(check_launch("scale_to_kernel"));
    if (stats) FC_CUDA(cudaEventRecord(c.ev1, st));
    double h[2];
    int hf[2];
    FC_CUDA(cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, st));
    FC_CUDA(cudaMemcpyAsync(hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, st));
    FC_CUDA(cudaStreamSynchronize(st));
    if (hf[1]) return fail(FC_ERR_TIMEOUT, "RI-MP2 gradient: a pipeline wait ran out");
    if (hf[0]) {
        // the DMMA form writes Gamma again: the copies of this one come first
        if (sink) FC_CUDA(cudaStreamSynchronize(sink->stream));
        return FC_OK;
    }
    *ran = true;
    *e_os = h[0];
    *e_ss = h[1];
    if (stats) {
        float ms = 0.f;
        FC_CUDA(cudaEventElapsedTime(&ms, c.ev0, c.ev1));
        const double P = (double)nocc * (nocc + 1) / 2.0;
        stats->kernel_ms = ms;
        stats->flops = 2.0 * naux * (double)nvir * nvir * P + 2.0 * naux * (double)nov * nov;
        stats->precision = FC_PREC_F64;
        stats->launches += (int)(nl + nadj + 1);
        stats->tile_m = MG_BM;
        stats->tile_n = MG_BN;
        stats->k_panel = 0;
        stats->d2h_bytes += sizeof(h) + sizeof(hf);
        stats->h2d_bytes += hp.size() * sizeof(int2) + ht.size() * sizeof(int4);
        stats->main_launches = (int)ncp;
        FC_TRY(timing_sum((int)ncp, &stats->main_ms));
        stats->main_flops = 2.0 * naux * (double)nvir * nvir * P;
        stats->main_bytes = (double)MG_N * naux * (double)nov * (double)(nch + 1) + 8.0 * P * (double)nvir * nvir;
        stats->aux_launches = nadj;
        FC_TRY(timing_sum2(nadj, &stats->aux_ms));
        stats->aux_flops = adj_flops;
        stats->aux_bytes = adj_bytes;
    }
    return FC_OK;
}

// ------------------------------------------------------------- energies --

// At 2 naux rows cols = 1.65e9 (naux 420, nocc 18, nvir 110; cols: half of the
// row's columns on average) 153 us here, 190 DMMA.  Below, DMMA's last wave
// decides: 153 and 160 at 1.0e9 (700, 10, 120), 150 and 143 at 1.24e9 (400, 16,
// 110), 136 and 99 at 5e8.  The two spins' energies, three passes each: 329 and
// 386 at 2.7e9, 326 and 318 at 1.9e9.
bool mod_energy_pays(int64_t naux, int64_t rows, int64_t cols, int nspin) {
    return naux <= MG_KMAX && 2.0 * naux * (double)rows * (double)cols >= (nspin > 1 ? 2.2e9 : 1.1e9);
}

namespace {

// One pair sum: the pairs i <= j of one spin (b == a), or all (i, J) of two.
struct EnergyPass {
    int a, b;
    AmpMode mode;
    int64_t c0 = 0, nc = 0;      // its row chunks
    int ntiles = 0;
    int64_t tiles0 = 0;          // its virtual tiles in the pair table
};
struct EnergyChunk {
    int64_t i0, ni, j0, nj, p0, np, t0, nt;
};

// e[2 k], e[2 k + 1]: E_os and E_ss of pass k (cross: E_ab, 0) of the spins'
// b_ov, converted once each.  G of a chunk of rows is formed by the residue
// GEMM and read once by amp_kernel; chunks of at most 2 GiB.
fc_status energy_passes(const UmpSpin* spin, int nspin, std::vector<EnergyPass>& passes, int64_t naux, int has_kappa,
                        double kappa, int64_t budget, cudaStream_t st, double* e, fc_stats* stats, bool* ran) {
    *ran = false;
    FC_TRY(amp_attrs());
    budget = std::min(budget, int64_t(2) << 30);
    std::vector<EnergyChunk> ch;
    std::vector<int2> hp;
    std::vector<int4> ht;
    size_t g_max = 0, items_max = 0;
    int64_t np_max = 0;
    for (EnergyPass& ps : passes) {
        const UmpSpin &A = spin[ps.a], &B = spin[ps.b];
        const int nta = (int)((A.nvir + AT - 1) / AT), ntb = (int)((B.nvir + AT - 1) / AT);
        const int64_t row = A.nvir * B.nocc * B.nvir * 8;  // bytes of G per orbital of the rows
        const int64_t ci = balanced(A.nocc, std::min(budget / row, (int64_t)65535 / B.nocc));
        if (row > budget || B.nocc > 65535) return FC_OK;  // (the amplitude kernel's grid)
        ps.ntiles = ps.mode == AMP_CROSS ? nta * ntb : nta * (nta + 1) / 2;
        ps.c0 = (int64_t)ch.size();
        for (int64_t i0 = 0; i0 < A.nocc; i0 += ci) {
            EnergyChunk x{};
            x.i0 = i0;
            x.ni = std::min(ci, A.nocc - i0);
            x.j0 = ps.mode == AMP_CROSS ? 0 : i0;
            x.nj = B.nocc - x.j0;
            x.p0 = (int64_t)hp.size();
            for (int64_t i = i0; i < i0 + x.ni; ++i)
                for (int64_t j = ps.mode == AMP_CROSS ? 0 : i; j < B.nocc; ++j)
                    hp.push_back(make_int2((int)i, (int)j));
            x.np = (int64_t)hp.size() - x.p0;
            x.t0 = (int64_t)ht.size();
            x.nt = mg_tiles(x.nj * B.nvir, x.ni * A.nvir, naux, ps.mode != AMP_CROSS, 1, &ht);
            g_max = std::max(g_max, (size_t)(x.ni * A.nvir * x.nj * B.nvir));
            items_max = std::max(items_max, (size_t)x.np * ps.ntiles);
            np_max = std::max(np_max, x.np);
            ch.push_back(x);
        }
        ps.nc = (int64_t)ch.size() - ps.c0;
        ps.tiles0 = (int64_t)hp.size();
        for (int ta = 0; ta < nta; ++ta)
            for (int tb = ps.mode == AMP_CROSS ? 0 : ta; tb < ntb; ++tb) hp.push_back(make_int2(ta, tb));
    }
    int64_t rows[2] = {0, 0}, rmax = 0;
    for (int s = 0; s < nspin; ++s) {
        rows[s] = spin[s].nocc * spin[s].nvir;
        rmax = std::max(rmax, rows[s]);
    }
    const int64_t npass = (int64_t)passes.size();
    // all scratch is spare memory: the DMMA form needs next to none
    double *stat[2], *mpart, *part, *acc;
    int2* pairs;
    int4* items;
    auto misc = [&](Carver& c) {
        pairs = c.take<int2>(hp.size());
        part = c.take<double>(items_max * 3 + (size_t)np_max * 3);
        acc = c.take<double>(32);
        for (int s = 0; s < nspin; ++s) stat[s] = c.take<double>(mg_stat_doubles(naux, rows[s]));
        mpart = c.take<double>(mg_part_doubles(naux, rmax));
        items = c.take<int4>(ht.size());
    };
    Carver cm;
    misc(cm);
    void* mg[WS_MG_SLOTS];
    if (!ws_get_mg({mg_bytes(rows[0], naux), nspin > 1 ? mg_bytes(rows[1], naux) : 0, 0, g_max * 8,
                    mg_scratch_bytes(), cm.off},
                   mg))
        return FC_OK;
    cm = Carver{(char*)mg[5], 0};
    misc(cm);
    double* G = (double*)mg[3];
    double* psum = part + 3 * items_max;
    int* flags = (int*)(acc + 2 * npass);
    FC_CUDA(cudaMemcpyAsync(pairs, hp.data(), hp.size() * sizeof(int2), cudaMemcpyHostToDevice, st));
    FC_CUDA(cudaMemcpyAsync(items, ht.data(), ht.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
    FC_CUDA(cudaMemsetAsync(acc, 0, 256, st));
    Context& c = ctx();
    if (stats) FC_CUDA(cudaEventRecord(c.ev0, st));
    MgMat B[2];
    MgOperand op[2];
    for (int s = 0; s < nspin; ++s) {
        B[s] = mg_mat(spin[s].b_ov, rows[s], naux, rows[s], stat[s]);
        FC_TRY(mg_stats(B[s], mpart, flags, st));
        FC_TRY(mg_convert(B[s], 1, (int8_t*)mg[s], &B[s], 1, mpart, flags, st, &op[s]));
    }
    int nl = 4 * nspin;
    if (nspin > 1) {  // the product of the two spins
        for (int s = 0; s < 2; ++s) FC_TRY(mg_guard(B[s], 1, B[1 - s], 1, mpart, flags, st));
        nl += 4;
    }
    double flops = 0.0;
    for (int64_t k = 0; k < npass; ++k) {
        const EnergyPass& ps = passes[(size_t)k];
        const UmpSpin &A = spin[ps.a], &B = spin[ps.b];
        for (int64_t q = ps.c0; q < ps.c0 + ps.nc; ++q) {
            const EnergyChunk& x = ch[(size_t)q];
            const int64_t ld = x.nj * B.nvir;
            FC_TRY(mg_gemm(op[ps.b].slice(x.j0 * B.nvir, ld), op[ps.a].slice(x.i0 * A.nvir, x.ni * A.nvir),
                           MgOut{G, ld, 0, 1.0, 0}, items + x.t0, x.nt, mg[4], flags, st));
            AmpArgs a{};
            a.g = G;
            a.ld = ld;
            a.pairs = pairs + x.p0;
            a.tiles = pairs + ps.tiles0;
            a.ntiles = ps.ntiles;
            a.i0 = (int)x.i0;
            a.j0 = (int)x.j0;
            a.nvir = (int)A.nvir;
            a.nvir2 = (int)B.nvir;
            a.eo = A.eps_occ;
            a.ev = A.eps_vir;
            a.eo2 = B.eps_occ;
            a.ev2 = B.eps_vir;
            a.same = ps.mode != AMP_CROSS;
            a.has_kappa = has_kappa;
            a.kappa = kappa;
            a.bad = flags;
            a.part = part;
            const dim3 grid((unsigned)ps.ntiles, (unsigned)x.np);
            if (ps.mode == AMP_CROSS) amp_kernel<AMP_CROSS><<<grid, AN, AMP_SMEM, st>>>(a);
            else amp_kernel<AMP_ENERGY><<<grid, AN, AMP_SMEM, st>>>(a);
            amp_pair_sum_kernel<<<(unsigned)((x.np + 7) / 8), 256, 0, st>>>(part, x.np, ps.ntiles, psum);
            amp_fold_kernel<<<1, 256, 0, st>>>(psum, a.pairs, x.np, 0, 0, 0, acc + 2 * k, nullptr);
            FC_TRY(check_launch("residue energy"));
            nl += 4;
        }
        const double P = ps.mode == AMP_CROSS ? (double)A.nocc * B.nocc : (double)A.nocc * (A.nocc + 1) / 2.0;
        flops += 2.0 * naux * (double)A.nvir * B.nvir * P;
    }
    if (stats) FC_CUDA(cudaEventRecord(c.ev1, st));
    double h[8];  // the sums, then the flags
    FC_CUDA(cudaMemcpyAsync(h, acc, (2 * npass + 1) * 8, cudaMemcpyDeviceToHost, st));
    FC_CUDA(cudaStreamSynchronize(st));
    int hf[2];
    std::memcpy(hf, h + 2 * npass, sizeof(hf));
    if (hf[1]) return fail(FC_ERR_TIMEOUT, "RI-MP2 energy: a pipeline wait ran out");
    if (hf[0]) return FC_OK;
    *ran = true;
    for (int64_t k = 0; k < 2 * npass; ++k) e[k] = h[k];
    if (stats) {
        float ms = 0.f;
        FC_CUDA(cudaEventElapsedTime(&ms, c.ev0, c.ev1));
        stats->kernel_ms = ms;
        stats->flops = flops;
        stats->precision = FC_PREC_F64;
        stats->launches += nl;
        stats->tile_m = MG_BM;
        stats->tile_n = MG_BN;
        stats->k_panel = 0;
        stats->d2h_bytes += (2 * npass + 1) * 8;
        stats->h2d_bytes += hp.size() * sizeof(int2) + ht.size() * sizeof(int4);
        stats->main_launches = (int)ch.size();
        stats->main_ms = ms;
        stats->main_flops = flops;
        stats->main_bytes = (double)MG_N * naux * (rows[0] + rows[1]);
    }
    return FC_OK;
}

}  // namespace

fc_status rimp2_energy_mod(const Rimp2Dev& d, cudaStream_t st, double* e_os, double* e_ss, fc_stats* stats,
                           bool* ran) {
    const UmpSpin s{d.b_ov, d.eps_occ, d.eps_vir, d.nocc, d.nvir};
    std::vector<EnergyPass> ps{{0, 0, AMP_ENERGY}};
    double e[2] = {0.0, 0.0};
    FC_TRY(energy_passes(&s, 1, ps, d.naux, d.has_kappa, d.kappa, d.chunk_bytes, st, e, stats, ran));
    if (*ran) {
        *e_os = e[0];
        *e_ss = e[1];
    }
    return FC_OK;
}

fc_status ump2_energy_mod(const UmpSpin& a, const UmpSpin& b, int64_t naux, int64_t budget, cudaStream_t st,
                          double* e_aa, double* e_bb, double* e_ab, fc_stats* stats, bool* ran) {
    const UmpSpin s[2] = {a, b};
    std::vector<EnergyPass> ps{{0, 0, AMP_ENERGY}, {1, 1, AMP_ENERGY}, {0, 1, AMP_CROSS}};
    double e[6] = {};
    FC_TRY(energy_passes(s, 2, ps, naux, 0, 0.0, budget, st, e, stats, ran));
    if (*ran) {
        // one spin's E_ss = 2 E_sigma-sigma (no pair where it has one orbital)
        *e_aa = a.nocc < 2 ? 0.0 : 0.5 * e[1];
        *e_bb = b.nocc < 2 ? 0.0 : 0.5 * e[3];
        *e_ab = e[4];
    }
    return FC_OK;
}

}  // namespace fc
