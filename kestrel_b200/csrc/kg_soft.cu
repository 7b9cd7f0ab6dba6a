// kg_soft.cu — the GL/PL estimator on soft genotype likelihoods
// (src/wrapper.rs:89-330 with src/mixture.rs:9-140 and src/coefficients.rs:
// 40-141): per-site allele frequencies by the HWE SQP on the samples'
// likelihoods, then for every pair the Jacquard SQP on the rows L_s = sum over
// (gx, gy) of GLx(gx) GLy(gy) m(gx, gy) of its sites.
//
// Layout: biallelic likelihoods double [sample][site][3] (0/0, 0/1, 1/1;
// linear scale; a NaN marks a missing sample) as loaded; the kept sites'
// likelihoods are also packed as FP32, two sites a record [sample][site pair]
// {l0a, l0b, l1a, l1b}, {l2a, l2b, 0, 0} (NaN where a sample is missing and
// past the last site), beside {pa, pb, qa, qb} of the kept frequencies.  Tri-
// and tetra-allelic sites: double [sample][site][6] and [sample][site][10] in the
// VCF genotype order.
//
// Lanes take the kept sites; the SQP itself is FP64.  FP32C pairs without tri-
// and tetra-allelic sites run in waves: the evaluations in soft_pass_kernel, four
// warps a pair, the solver between them in soft_advance_kernel, a thread per
// pair (kg_advance.cuh).  In one kernel the solver's 1,300 straight instructions an
// iteration pushed the site loop out of the instruction caches (its warps waited
// for instructions twice as long as they issued) and took 145,000 cycles a QP.
// The other pairs run in soft_pairs_kernel, a warp per pair from a counter.  The
// evaluations (f, g and H at a point) of the biallelic sites have one of two forms:
//   * FP32 (the default, KG_PREC_FP32C): from the FP32 likelihoods, which stay
//     L2-resident for cohorts of a few hundred samples, each site's row L is
//     formed from the pair's nine likelihood products in closed form, two sites
//     an instruction (packed FP32); d = eps + L.x with the FP32 hi parts of x,
//     the sums in FP32 promoted to FP64 (per site parity: gradient and
//     objective every 8 sites, Hessian every 32 into the lane's shared memory),
//     and the lo parts of x restored to first order in FP64;
//     near convergence the objective change is summed as log(d / d_old), as
//     on the hard-call path.  A pair whose FP32 condition estimate exceeds
//     COND_RECHECK, or whose KKT residual stalls below 1e-6 three times, is
//     re-evaluated in FP64 and stays FP64 (the hard-call path's rule).
//   * FP64 (KG_PREC_FP64, and escalated pairs): from the FP64 likelihoods,
//     each row the sum over the nine genotype pairs of GLx GLy m(gx, gy).
// Tri- and tetra-allelic sites keep the genotypes of the alleles left after
// the frequency cut (src/wrapper.rs:349-409); their rows (G' x G' x 9 terms
// each) are built once per pair in FP64 into the warp's scratch, as the
// reference builds its pair buffer once, and every evaluation adds their FP64
// sums to the biallelic ones.  The shared-memory sums of a warp are 45 rows of
// 33 doubles: the 32 lanes' partials and the warp's total.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cstdlib>
#include <string>
#include <vector>

#include "kestrel_gpu.h"
#include "kg_advance.cuh"
#include "kg_allele.cuh"
#include "kg_alleleN.cuh"
#include "kg_bulk.cuh"
#include "kg_engine.h"
#include "kg_pair.cuh"
#include "kg_qp1.cuh"
#include "kg_solver.cuh"

namespace kg {

#define KG_SOFT_TRY(expr)                                                       \
    do {                                                                        \
        cudaError_t e_ = (expr);                                                \
        if (e_ != cudaSuccess) {                                                \
            err = std::string(#expr) + ": " + cudaGetErrorString(e_);           \
            return e_ == cudaErrorMemoryAllocation ? KG_ENOMEM : KG_ECUDA;      \
        }                                                                       \
    } while (0)

// Thread per site: frequencies (REF, ALT) and the keep flag (both non-zero
// after the maf cut).  Adjacent threads read adjacent sites of a sample.
__device__ __forceinline__ double warp_allsum(double v) {
    // butterfly: every lane adds the same two partials at every level, so all
    // lanes end with the same bits
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Warp per site: the HWE SQP of the site's frequencies with the samples over
// the lanes (the sums of src/mixture.rs's objective and derivatives reduced
// across the warp; every lane then runs the same solver steps on the same
// values).
__global__ void soft_freq_kernel(const double* __restrict__ gl, int64_t n_samples, int64_t n_sites, double maf,
                                 uint64_t iterations, double* __restrict__ pf, double* __restrict__ qf,
                                 uint8_t* __restrict__ keep) {
    const int lane = threadIdx.x & 31;
    const int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (v >= n_sites) return;
    const double eps = make_tune(iterations).epsilon;
    auto rowp = [&](int64_t s) { return gl + (s * n_sites + v) * 3; };
    double called = 0.0;
    for (int64_t s = lane; s < n_samples; s += 32) {
        const double* r = rowp(s);
        called += !(isnan(r[0]) || isnan(r[1]) || isnan(r[2]));
    }
    called = warp_allsum(called);
    double p = 0.0, q = 0.0;
    if (called > 0.0) {
        auto obj = [&](double x0, double x1) {
            double acc = 0.0;
            const double w0 = x0 * x0, w1 = 2.0 * x0 * x1, w2 = x1 * x1;
            for (int64_t s = lane; s < n_samples; s += 32) {
                const double* r = rowp(s);
                const double l0 = r[0], l1 = r[1], l2 = r[2];
                if (isnan(l0) || isnan(l1) || isnan(l2)) continue;
                acc += log(fma(w2, l2, fma(w1, l1, fma(w0, l0, eps))));
            }
            return -warp_allsum(acc) / called;
        };
        auto gh = [&](double x0, double x1, double& g0, double& g1, double& h00, double& h01, double& h11) {
            double zg0 = 0.0, zg1 = 0.0, z00 = 0.0, z01 = 0.0, z11 = 0.0;
            for (int64_t s = lane; s < n_samples; s += 32) {
                const double* r = rowp(s);
                const double l0 = r[0], l1 = r[1], l2 = r[2];
                if (isnan(l0) || isnan(l1) || isnan(l2)) continue;
                const double lx0 = fma(l1, x1, fma(l0, x0, 0.0));
                const double lx1 = fma(l2, x1, fma(l1, x0, 0.0));
                const double d = fma(x1, lx1, fma(x0, lx0, eps));
                const double inv = 1.0 / d;
                const double a0 = lx0 * inv, a1 = lx1 * inv;
                zg0 += a0;
                zg1 += a1;
                z00 += 2.0 * a0 * a0 - l0 * inv;
                z01 += 2.0 * a0 * a1 - l1 * inv;
                z11 += 2.0 * a1 * a1 - l2 * inv;
            }
            g0 = -2.0 * warp_allsum(zg0) / called;
            g1 = -2.0 * warp_allsum(zg1) / called;
            h00 = 2.0 * warp_allsum(z00) / called;
            h01 = 2.0 * warp_allsum(z01) / called;
            h11 = 2.0 * warp_allsum(z11) / called;
        };
        allele2_fit(obj, gh, iterations, maf, p, q);
    }
    if (lane == 0) {
        pf[v] = p;
        qf[v] = q;
        keep[v] = (p > 0.0 && q > 0.0) ? 1 : 0;
    }
}

constexpr int SOFT_WARPS = 4;
constexpr int HS = 33;   // shared-memory stride of the Hessian sums: 32 lane partials, then the warp total
// A warp's shared memory: the Hessian sums (45 rows of HS doubles, padded to
// 16 bytes), then per lane SOFT_STAGES slots of 80 bytes for the FP32 form's
// prefetched sites (the two samples' records of a site pair and its
// frequencies).
constexpr int SOFT_STAGES = 2;
constexpr int SOFT_SLOT = 5;   // float4 of a slot
constexpr int SOFT_SUMS_BYTES = (45 * HS * 8 + 15) / 16 * 16;
constexpr int SOFT_WARP_SMEM = SOFT_SUMS_BYTES + 32 * SOFT_STAGES * SOFT_SLOT * 16;
constexpr int SOFT_SMEM = SOFT_WARPS * SOFT_WARP_SMEM;

// ---------------------------------------------------------- tri / tetra
// A loaded tri- or tetra-allelic site after its frequency fit: G' genotypes of
// the remaining alleles (0: discarded), the original genotype index of each,
// and the site's G' x G' rows m[g'x][g'y] (stride ML_SOFT_ROWS rows).
constexpr int SOFT_MULTI_ROWS = 100;

struct SoftMultiDev {
    const double* gl[2];      // [sample][site][G0] of the tri- and of the tetra-allelic sites
    int64_t n[2];             // their site counts
    int64_t total;            // n[0] + n[1]: tri-allelic sites first
    const int32_t* gk;        // per site: G' (0 = discarded)
    const uint8_t* gidx;      // per site: [10] original genotype of reduced genotype g'
    const double* rows;       // per site: SOFT_MULTI_ROWS x 9
    double* scratch;          // per warp: total x 9, the current pair's rows (NaN first entry: no row)
};

// Per-sample likelihood rows of one multi-allelic site (a row with a NaN is a
// missing sample), weight 1: the row source of allele_fit.
struct SoftRows {
    const double* gl;
    int64_t n_samples, n_sites, v;
    int a, g0;
    __device__ int alleles() const { return a; }
    __device__ int rows() const { return (int)n_samples; }
    __device__ double weight(int) const { return 1.0; }
    __device__ bool row(int k, double* l) const {
        const double* r = gl + ((int64_t)k * n_sites + v) * g0;
        bool ok = true;
        for (int g = 0; g < MAXG; g++) {
            l[g] = g < g0 ? r[g] : 0.0;
            ok = ok && !(g < g0 && isnan(l[g]));
        }
        return ok;
    }
};

// Thread per tri-/tetra-allelic site: the frequency fit on the samples'
// likelihoods with the maf cut, the alleles left (in order), each reduced
// genotype's original index and the site's rows; used[0..2] counts the sites
// left with 2, 3, 4 alleles.
__global__ void soft_multi_site_kernel(SoftMultiDev M, int64_t n_samples, double maf, uint64_t iterations,
                                       int32_t* __restrict__ gk, uint8_t* __restrict__ gidx,
                                       double* __restrict__ rows, unsigned long long* __restrict__ used) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= M.total) return;
    const int c = t < M.n[0] ? 0 : 1;
    const int64_t v = c == 0 ? t : t - M.n[0];
    SoftRows src;
    src.gl = M.gl[c];
    src.n_samples = n_samples;
    src.n_sites = M.n[c];
    src.v = v;
    src.a = c == 0 ? 3 : 4;
    src.g0 = c == 0 ? 6 : 10;
    double f[MAXA];
    allele_fit(src, iterations, maf, f);
    int keep[MAXA], na = 0;
    double fk[MAXA] = {0.0, 0.0, 0.0, 0.0};
    for (int a = 0; a < src.a; a++)
        if (f[a] > 0.0) {
            keep[na] = a;
            fk[na] = f[a];
            na++;
        }
    if (na < 2) {
        gk[t] = 0;
        return;
    }
    const int g = na * (na + 1) / 2;
    gk[t] = g;
    int k = 0;
    for (int j = 0; j < na; j++)
        for (int i = 0; i <= j; i++) gidx[MAXG * t + k++] = (uint8_t)(keep[j] * (keep[j] + 1) / 2 + keep[i]);
    double* R = rows + (int64_t)SOFT_MULTI_ROWS * 9 * t;
    for (int gx = 0; gx < g; gx++) {
        int i, j;
        genotype_alleles(gx, i, j);
        for (int gy = 0; gy < g; gy++) {
            int a, b;
            genotype_alleles(gy, a, b);
            iis_row(i, j, a, b, fk[0], fk[1], fk[2], fk[3], R + 9 * (gx * g + gy));
        }
    }
    atomicAdd(&used[na - 2], 1ull);
}

// The pair's rows at the multi-allelic sites, in FP64, into the warp's
// scratch: sum over the remaining genotypes of GLx(gx) GLy(gy) m[gx][gy]
// (gx outer, gy inner, as src/mixture.rs:9-60 accumulates); NaN first entry
// when a sample is missing or the site was discarded.  Returns the warp's count
// of rows.
__device__ __noinline__ int64_t soft_multi_build(const SoftMultiDev M, int64_t x, int64_t y, int lane, double* R) {
    int64_t m = 0;
    for (int64_t t = lane; t < M.total; t += 32) {
        double* o = R + 9 * t;
        const int g = M.gk[t];
        bool ok = g > 0;
        double L[9];
#pragma unroll
        for (int k = 0; k < 9; k++) L[k] = 0.0;
        if (ok) {
            const int c = t < M.n[0] ? 0 : 1;
            const int64_t v = c == 0 ? t : t - M.n[0];
            const int g0 = c == 0 ? 6 : 10;
            const double* lx = M.gl[c] + (x * M.n[c] + v) * g0;
            const double* ly = M.gl[c] + (y * M.n[c] + v) * g0;
            const uint8_t* gi = M.gidx + MAXG * t;
            const double* mm = M.rows + (int64_t)SOFT_MULTI_ROWS * 9 * t;
            for (int gx = 0; gx < g && ok; gx++) {
                const double ax = lx[gi[gx]];
                for (int gy = 0; gy < g; gy++) {
                    const double gg = ax * ly[gi[gy]];
#pragma unroll
                    for (int k = 0; k < 9; k++) L[k] = fma(gg, mm[9 * (gx * g + gy) + k], L[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < 9; k++) ok = ok && !isnan(L[k]);
        }
        if (ok) {
#pragma unroll
            for (int k = 0; k < 9; k++) o[k] = L[k];
            m++;
        } else {
            o[0] = CUDART_NAN;
        }
    }
    for (int off = 16; off > 0; off >>= 1) m += __shfl_xor_sync(0xffffffffu, m, off);
    __syncwarp();   // the rows are read by every lane's evaluations
    return m;
}

// Adds the pair's multi-allelic rows at xt to the warp's totals, in FP64:
// G (warp-uniform), the 45 Hessian totals at hs[a * HS + 32], F (sum log d, or
// sum log(d / d_old) with d_old at xc, d - d_old from step (difference_step), in a
// difference pass) and n.
__device__ __noinline__ void soft_multi_add(const double* R, int64_t total, const double* xt, const double* step,
                                            const double* xc, bool diff, double eps, int lane, double* hs, double* G, double& F,
                                            int64_t& n) {
    double g[9], f = 0.0;
#pragma unroll
    for (int i = 0; i < 9; i++) g[i] = 0.0;
    int64_t m = 0;
    for (int a = 0; a < 45; a++) hs[a * HS + lane] = 0.0;
    for (int64_t t = lane; t < total; t += 32) {
        const double* L = R + 9 * t;
        if (isnan(L[0])) continue;
        double d = eps;
#pragma unroll
        for (int i = 0; i < 9; i++) d = fma(xt[i], L[i], d);
        const double r = 1.0 / d;
        double b[9];
#pragma unroll
        for (int i = 0; i < 9; i++) {
            g[i] = fma(L[i], r, g[i]);
            b[i] = L[i] * r;
        }
        int a = 0;
#pragma unroll
        for (int i = 0; i < 9; i++)
#pragma unroll
            for (int j = i; j < 9; j++, a++) hs[a * HS + lane] = fma(b[i], b[j], hs[a * HS + lane]);
        if (!diff) {
            f += log(d);
        } else {
            double dc = eps, dl = 0.0;
#pragma unroll
            for (int i = 0; i < 9; i++) {
                dc = fma(xc[i], L[i], dc);
                dl = fma(step[i], L[i], dl);
            }
            f += log1p(dl / dc);
        }
        m++;
    }
    for (int off = 16; off > 0; off >>= 1) {
        f += __shfl_xor_sync(0xffffffffu, f, off);
        m += __shfl_xor_sync(0xffffffffu, m, off);
#pragma unroll
        for (int i = 0; i < 9; i++) g[i] += __shfl_xor_sync(0xffffffffu, g[i], off);
    }
    __syncwarp();
    for (int a = 0; a < 45; a++) {
        double h = hs[a * HS + lane];
        for (int off = 16; off > 0; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
        if (lane == 0) hs[a * HS + 32] += h;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 9; i++) G[i] += g[i];
    F += f;
    n += m;
}

// The Hessian total (i, j) of the upper triangle, row-major.
__device__ __forceinline__ double htotal(const double* hs, int i, int j) {
    const int i0 = i < j ? i : j, j0 = i < j ? j : i;
    return hs[(i0 * 9 - i0 * (i0 - 1) / 2 + (j0 - i0)) * HS + 32];
}

// The warp's 45 Hessian totals from the lanes' partials: hs[a * HS + 32].
__device__ __forceinline__ void hessian_totals(double* hs, int lane) {
    __syncwarp();
    for (int a = 0; a < 45; a++) {
        double h = hs[a * HS + lane];
        for (int off = 16; off > 0; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
        if (lane == 0) hs[a * HS + 32] = h;
    }
    __syncwarp();
}

// The FP64 site loop over every parts-th group of 32 kept sites from part on:
// this lane's sums of log d, L r and (in shared memory) L L' r^2, r = 1/(eps +
// L.x), and its rows without a NaN.
__device__ __forceinline__ void soft_sites64(const double* __restrict__ gl, int64_t n_sites,
                                             const int32_t* __restrict__ kept, const double* __restrict__ kp,
                                             const double* __restrict__ kq, int64_t nk, int64_t x, int64_t y,
                                             const double* xv, double eps, int lane, int part, int parts, double* hs,
                                             double (&g)[9], double& f, int64_t& n) {
    f = 0.0;
#pragma unroll
    for (int i = 0; i < 9; i++) g[i] = 0.0;
    for (int a = 0; a < 45; a++) hs[a * HS + lane] = 0.0;
    n = 0;
    for (int64_t k = lane + 32 * part; k < nk; k += 32 * parts) {
        const int64_t v = kept[k];
        const double* lx = gl + (x * n_sites + v) * 3;
        const double* ly = gl + (y * n_sites + v) * 3;
        const double ax[3] = {lx[0], lx[1], lx[2]}, ay[3] = {ly[0], ly[1], ly[2]};
        if (isnan(ax[0] + ax[1] + ax[2] + ay[0] + ay[1] + ay[2])) continue;
        const double p = kp[k], q = kq[k];
        double L[9];
#pragma unroll
        for (int i = 0; i < 9; i++) L[i] = 0.0;
#pragma unroll
        for (int gx = 0; gx < 3; gx++)
#pragma unroll
            for (int gy = 0; gy < 3; gy++) {
                const double w = ax[gx] * ay[gy];
                double m[9];
                cls_row(gx, gy, p, q, m);
#pragma unroll
                for (int i = 0; i < 9; i++) L[i] = fma(w, m[i], L[i]);
            }
        double d = eps;
#pragma unroll
        for (int i = 0; i < 9; i++) d = fma(xv[i], L[i], d);
        f += log(d);
        const double r = 1.0 / d;
        double b[9];
#pragma unroll
        for (int i = 0; i < 9; i++) {
            g[i] = fma(L[i], r, g[i]);
            b[i] = L[i] * r;
        }
        int a = 0;
#pragma unroll
        for (int i = 0; i < 9; i++)
#pragma unroll
            for (int j = i; j < 9; j++, a++) hs[a * HS + lane] = fma(b[i], b[j], hs[a * HS + lane]);
        n++;
    }
}

// f, g and this lane's Hessian row at x over the pair's rows (-(1/n) sum log(eps
// + L.x), -(1/n) sum L r, (1/n) sum L L' r^2, r = 1/(eps + L.x)); n = rows
// without a NaN.  hs: the warp's Hessian sums in shared memory; R, nm: the
// pair's multi-allelic rows.
__device__ __noinline__ int64_t soft_evaluate(const double* __restrict__ gl, int64_t n_sites,
                                              const int32_t* __restrict__ kept, const double* __restrict__ kp,
                                              const double* __restrict__ kq, int64_t nk, int64_t x, int64_t y,
                                              const double* xv, double eps, int lane, double* hs, const double* R,
                                              int64_t nm, PairEval& ev) {
    double f, g[9];
    int64_t n;
    soft_sites64(gl, n_sites, kept, kp, kq, nk, x, y, xv, eps, lane, 0, 1, hs, g, f, n);
    // warp sums (fixed butterfly order)
    for (int off = 16; off > 0; off >>= 1) {
        f += __shfl_xor_sync(0xffffffffu, f, off);
        n += __shfl_xor_sync(0xffffffffu, n, off);
#pragma unroll
        for (int i = 0; i < 9; i++) g[i] += __shfl_xor_sync(0xffffffffu, g[i], off);
    }
    hessian_totals(hs, lane);
    if (nm > 0) soft_multi_add(R, nm, xv, xv, xv, false, eps, lane, hs, g, f, n);
    const double dn = (double)n;
    ev.f = -f / dn;
#pragma unroll
    for (int i = 0; i < 9; i++) ev.g[i] = -g[i] / dn;
    // lane i < 9 takes row i of H
#pragma unroll
    for (int j = 0; j < 9; j++) ev.Hr[j] = lane < 9 ? htotal(hs, lane, j) / dn : 0.0;
    __syncwarp();
    return n;
}

// Packs the kept sites' likelihoods and frequencies as FP32, two sites a record
// (see the file comment).
__global__ void soft_pack32_kernel(const double* __restrict__ gl, int64_t n_samples, int64_t n_sites,
                                   const int32_t* __restrict__ kept, const double* __restrict__ kp,
                                   const double* __restrict__ kq, int64_t nk, float4* __restrict__ g32,
                                   float4* __restrict__ pq32) {
    const int64_t np = (nk + 1) / 2, total = n_samples * np;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = t / np, j = t - s * np;
        float l[2][3];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int64_t k = 2 * j + h;
            const double* r = gl + (s * n_sites + (k < nk ? kept[k] : 0)) * 3;
            const bool miss = k >= nk || isnan(r[0]) || isnan(r[1]) || isnan(r[2]);
#pragma unroll
            for (int g = 0; g < 3; g++) l[h][g] = miss ? CUDART_NAN_F : (float)r[g];
        }
        g32[2 * t] = make_float4(l[0][0], l[1][0], l[0][1], l[1][1]);
        g32[2 * t + 1] = make_float4(l[0][2], l[1][2], 0.f, 0.f);
        if (s == 0) {
            const int64_t k1 = 2 * j + 1 < nk ? 2 * j + 1 : 2 * j;
            pq32[j] = make_float4((float)kp[2 * j], (float)kp[k1], (float)kq[2 * j], (float)kq[k1]);
        }
    }
}

// The FP32 site loop (see the file comment) over every parts-th group of 32
// site pairs from part on, at xt: this lane's FP64 sums G of L r and F of log2 d
// or (DIFF: step = xt - xc less its part along xc, difference_step) of log(d /
// d_old), in shared memory of L L' r^2, and its sites.
template <bool DIFF>
__device__ __forceinline__ void soft_sites32(const float4* __restrict__ g32, const float4* __restrict__ pq32, int64_t nk,
                                             int64_t x, int64_t y, const double* xt, const double* step, double eps,
                                             int lane, int part, int parts, double* hs, float4* slots, double (&G)[9],
                                             double& F, int64_t& n) {
    const bool diff = DIFF;
    float xh[9], sd[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
        xh[i] = (float)xt[i];
        sd[i] = DIFF ? (float)step[i] : 0.f;
    }
    F = 0.0;
    float2 g[9], h[45], o = dup2(0.f);
#pragma unroll
    for (int i = 0; i < 9; i++) { G[i] = 0.0; g[i] = dup2(0.f); }
#pragma unroll
    for (int a = 0; a < 45; a++) h[a] = dup2(0.f);
    for (int a = 0; a < 45; a++) hs[a * HS + lane] = 0.0;
    const int np = (int)((nk + 1) >> 1);   // site pairs
    const float4* lx = g32 + x * 2 * (int64_t)np;
    const float4* ly = g32 + y * 2 * (int64_t)np;
    const float2 e32 = dup2((float)eps);
    n = 0;
    // Warp-uniform iterations over site pairs (a lane past the end has NaN
    // records), so that the FP64 flushes below run once per warp.  The pair of
    // the next iteration is copied by cp.async into the lane's slots: the
    // prefetch holds no registers.  Two sites an instruction, because the loop is
    // bound by fetching and issuing it: with one site the warps waited for
    // instructions twice as long as they issued (277 a site, three warps a
    // scheduler at different places of the kernel).
    float4* my = slots + lane * (SOFT_SLOT * SOFT_STAGES);
    const uint32_t my0 = smem_u32(my);
    auto issue = [&](int it2) {
        const int k2 = lane + 32 * (it2 * parts + part);
        if (k2 < np) {
            const uint32_t d = my0 + 16u * SOFT_SLOT * (uint32_t)(it2 & 1);
            cp_async16(d, lx + 2 * k2);
            cp_async16(d + 16u, lx + 2 * k2 + 1);
            cp_async16(d + 32u, ly + 2 * k2);
            cp_async16(d + 48u, ly + 2 * k2 + 1);
            cp_async16(d + 64u, pq32 + k2);
        }
        cp_async_commit();
    };
    const int iters = max(0, (((np + 31) >> 5) - part + parts - 1) / parts);
    issue(0);
    for (int it = 0; it < iters; it++) {
        issue(it + 1);
        cp_async_wait<1>();   // this iteration's pair has landed
        const float4* st = my + SOFT_SLOT * (it & 1);
        const bool in = lane + 32 * (it * parts + part) < np;
        float2 X0 = dup2(CUDART_NAN_F), X1 = X0, X2 = X0, Y0 = X0, Y1 = X0, Y2 = X0, p = dup2(0.f), q = p;
        if (in) {
            const float4 a0 = st[0], c0 = st[2], f0 = st[4];
            X0 = make_float2(a0.x, a0.y);
            X1 = make_float2(a0.z, a0.w);
            X2 = *reinterpret_cast<const float2*>(st + 1);
            Y0 = make_float2(c0.x, c0.y);
            Y1 = make_float2(c0.z, c0.w);
            Y2 = *reinterpret_cast<const float2*>(st + 3);
            p = make_float2(f0.x, f0.y);
            q = make_float2(f0.z, f0.w);
        }
        // L = sum over (gx, gy) of GLx(gx) GLy(gy) m(gx, gy), the nine rows of
        // the biallelic conditional table (cls_row) gathered by entry
        const float2 A = mul2(X0, Y0), B = mul2(X2, Y2), C = mul2(X0, Y2), D = mul2(X2, Y0);
        const float2 E = mul2(X0, Y1), Fx = mul2(X2, Y1), Gx = mul2(X1, Y0), Hx = mul2(X1, Y2), I = mul2(X1, Y1);
        // a missing sample's record is NaN (the product is one too where a
        // likelihood is beyond FP32: such a pair's sums become NaN and it goes on in FP64)
        const bool v0 = !(isnan(X0.x) || isnan(Y0.x)), v1 = !(isnan(X0.y) || isnan(Y0.y));
        const float2 two = dup2(2.0f);
        const float2 p2 = mul2(p, p), q2 = mul2(q, q), pq = mul2(p, q), p2q = mul2(p2, q), pq2 = mul2(p, q2);
        const float2 S2 = fma2(A, p2, mul2(B, q2)), S3 = fma2(A, mul2(p2, p), mul2(B, mul2(q2, q)));
        float2 L[9];
        L[0] = fma2(A, p, mul2(B, q));
        L[1] = fma2(add2(C, D), pq, S2);
        L[2] = fma2(add2(E, Fx), pq, S2);
        L[3] = fma2(mul2(two, E), p2q, fma2(mul2(two, Fx), pq2, fma2(C, pq2, fma2(D, p2q, S3))));
        L[4] = fma2(add2(Gx, Hx), pq, S2);
        L[5] = fma2(mul2(two, Gx), p2q, fma2(mul2(two, Hx), pq2, fma2(C, p2q, fma2(D, pq2, S3))));
        L[6] = fma2(mul2(two, I), pq, S2);
        const float2 FH = add2(Fx, Hx), EG = add2(E, Gx);
        L[7] = fma2(I, add2(p2q, pq2), fma2(FH, pq2, fma2(EG, p2q, S3)));
        const float2 p2q2 = mul2(p2, q2);
        L[8] = fma2(mul2(dup2(4.0f), I), p2q2,
                    fma2(mul2(two, FH), mul2(pq2, q),
                         fma2(mul2(two, EG), mul2(p2q, p),
                              fma2(add2(C, D), p2q2, fma2(A, mul2(p2, p2), mul2(B, mul2(q2, q2)))))));
        // d = eps + L.x in three chains (dot9_eps)
        const float2 da = fma2(L[0], dup2(xh[0]), fma2(L[3], dup2(xh[3]), fma2(L[6], dup2(xh[6]), e32)));
        const float2 db = fma2(L[1], dup2(xh[1]), fma2(L[4], dup2(xh[4]), mul2(L[7], dup2(xh[7]))));
        const float2 dc = fma2(L[2], dup2(xh[2]), fma2(L[5], dup2(xh[5]), mul2(L[8], dup2(xh[8]))));
        const float2 d = add2(da, add2(db, dc));
        const float2 r = make_float2(v0 ? rcp_approx(d.x) : 0.f, v1 ? rcp_approx(d.y) : 0.f);
        if (!v0 || !v1) {
#pragma unroll
            for (int i = 0; i < 9; i++) L[i] = make_float2(v0 ? L[i].x : 0.f, v1 ? L[i].y : 0.f);
        }
        if (!diff) {
            o = add2(o, make_float2(v0 ? lg2_approx(d.x) : 0.f, v1 ? lg2_approx(d.y) : 0.f));
        } else {
            float2 dl = mul2(L[0], dup2(sd[0]));
#pragma unroll
            for (int i = 1; i < 9; i++) dl = fma2(L[i], dup2(sd[i]), dl);
            dl = mul2(dl, r);
            o = add2(o, make_float2(neg_log1m(dl.x), neg_log1m(dl.y)));
        }
#pragma unroll
        for (int i = 0; i < 9; i++) {
            g[i] = fma2(L[i], r, g[i]);
            L[i] = mul2(L[i], r);
        }
        {
            int a = 0;
#pragma unroll
            for (int i = 0; i < 9; i++)
#pragma unroll
                for (int j = i; j < 9; j++, a++) h[a] = fma2(L[i], L[j], h[a]);
        }
        n += (v0 ? 1 : 0) + (v1 ? 1 : 0);
        if ((it & 7) == 7) {
#pragma unroll
            for (int i = 0; i < 9; i++) {
                G[i] += (double)g[i].x;
                G[i] += (double)g[i].y;
                g[i] = dup2(0.f);
            }
            F += (double)o.x;
            F += (double)o.y;
            o = dup2(0.f);
        }
        if ((it & 15) == 15) {
#pragma unroll
            for (int a2 = 0; a2 < 45; a2++) {
                hs[a2 * HS + lane] += (double)(h[a2].x + h[a2].y);
                h[a2] = dup2(0.f);
                asm volatile("" ::: "memory");   // one read-modify-write at a time: no register peak
            }
        }
    }
    cp_async_wait<0>();   // no copy outstanding into the slots (they are past the last site)
#pragma unroll
    for (int i = 0; i < 9; i++) {
        G[i] += (double)g[i].x;
        G[i] += (double)g[i].y;
    }
    F += (double)o.x;
    F += (double)o.y;
#pragma unroll
    for (int a = 0; a < 45; a++) hs[a * HS + lane] += (double)(h[a].x + h[a].y);
}

// The FP32 evaluation (see the file comment) at xt; in a difference pass
// (DIFF) the objective is f_old - (1/n) sum log(d / d_old) with d_old at xc,
// step = xt - xc less its part along xc (difference_step).  hs: the warp's FP64
// Hessian sums in shared memory; R, nm: the pair's multi-allelic rows, added in
// FP64 after the lo correction of the biallelic sums.  Returns n.  Not inlined:
// the site loop gets the registers the pair's SQP state would hold.
template <bool DIFF>
__device__ __noinline__ int64_t soft_evaluate32(const float4* __restrict__ g32, const float4* __restrict__ pq32,
                                                int64_t nk, int64_t x, int64_t y,
                                                const double* xt, const double* step, const double* xc, double f_old,
                                                double eps, int lane, double* hs, float4* slots, const double* R,
                                                int64_t nm, PairEval& ev) {
    const bool diff = DIFF;
    float xh[9];
#pragma unroll
    for (int i = 0; i < 9; i++) xh[i] = (float)xt[i];
    double G[9], F;
    int64_t n;
    soft_sites32<DIFF>(g32, pq32, nk, x, y, xt, step, eps, lane, 0, 1, hs, slots, G, F, n);
    // warp sums (fixed butterfly order)
    for (int off = 16; off > 0; off >>= 1) {
        F += __shfl_xor_sync(0xffffffffu, F, off);
        n += __shfl_xor_sync(0xffffffffu, n, off);
#pragma unroll
        for (int i = 0; i < 9; i++) G[i] += __shfl_xor_sync(0xffffffffu, G[i], off);
    }
    hessian_totals(hs, lane);
    // the lo parts of x to first order: sum log d gains sum_j lo_j G_j, and
    // G_i loses sum_j H_ij lo_j (a difference pass uses the step's FP32 values)
    double lo[9];
#pragma unroll
    for (int j = 0; j < 9; j++) lo[j] = xt[j] - (double)xh[j];
    double corr = 0.0;
#pragma unroll
    for (int j = 0; j < 9; j++) corr = fma(lo[j], G[j], corr);
    double Gc[9];
#pragma unroll
    for (int i = 0; i < 9; i++) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < 9; j++) s = fma(htotal(hs, i, j), lo[j], s);
        Gc[i] = G[i] - s;
    }
    // objective so far in natural-log units (direct: F counted log2 d)
    double fsum = diff ? F : F * 0.69314718055994530942 + corr;
    if (nm > 0) soft_multi_add(R, nm, xt, step, xc, diff, eps, lane, hs, Gc, fsum, n);
    const double dn = (double)n;
    ev.df = -fsum / dn;   // in a difference pass the objective's change
    ev.f = diff ? f_old + ev.df : ev.df;
#pragma unroll
    for (int i = 0; i < 9; i++) ev.g[i] = -Gc[i] / dn;
#pragma unroll
    for (int j = 0; j < 9; j++) ev.Hr[j] = lane < 9 ? htotal(hs, lane, j) / dn : 0.0;
    __syncwarp();
    return n;
}

// The QP and the condition estimate of the warp's pair, by every lane alike
// (kg_qp1.cuh) from its shared memory: in holds H's upper triangle and, for the
// QP, c.  One thread's straight chain takes a fifth of the row-parallel form's
// 145,000 cycles of shuffles and divisions.
__device__ __noinline__ void soft_qp(const double* in, const Tune& tu, double* y) {
    double v[9];
#pragma unroll
    for (int i = 0; i < 9; i++) v[i] = y[i];
    qp_simplex_thread<true>([in](int k) { return in[k]; }, tu, v);
#pragma unroll
    for (int i = 0; i < 9; i++) y[i] = v[i];
}
__device__ __noinline__ double soft_condition(const double* in, const double* x, const double* g, double tol) {
    double xv[9], gv[9];
#pragma unroll
    for (int i = 0; i < 9; i++) { xv[i] = x[i]; gv[i] = g[i]; }
    return condition_thread([in](int k) { return in[k]; }, xv, gv, tol);
}
// Lane i < 9's row of H to the upper triangle in shared memory.
__device__ __forceinline__ void soft_share_hessian(const double* Hr, int lane, double* in) {
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 9; j++)
        if (lane < 9 && j >= lane) in[lane * 9 - lane * (lane - 1) / 2 + (j - lane)] = Hr[j];
    __syncwarp();
}

// Warp per output row of the first ns samples (x-major, y >= x), taken from a
// counter; the Jacquard SQP of src/sqp.rs:49-93 in FP64 on FP32 evaluations
// (prec64 = 0) or FP64 ones.  stats: [0] grad-Hessian evaluations, [1] of them
// in FP64, [2] pairs escalated to FP64, [3] pair-sites evaluated (summed over
// evaluations), [4] of them in FP64.
__global__ void __launch_bounds__(SOFT_WARPS * 32, 2) soft_pairs_kernel(
    const double* __restrict__ gl, int64_t n_sites, const int32_t* __restrict__ kept, const double* __restrict__ kp,
    const double* __restrict__ kq, const float4* __restrict__ g32, const float4* __restrict__ pq32, int prec64, int64_t nk, int64_t ns, int64_t n_rows, uint64_t iterations,
    kg_output* out, unsigned long long* next, int* no_rows, unsigned long long* stats, SoftMultiDev M) {
    extern __shared__ __align__(16) unsigned char soft_smem[];   // SOFT_WARP_SMEM per warp
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double* hs = reinterpret_cast<double*>(soft_smem + w * SOFT_WARP_SMEM);
    float4* slots = reinterpret_cast<float4*>(soft_smem + w * SOFT_WARP_SMEM + SOFT_SUMS_BYTES);
    // the warp's scratch for its pair's multi-allelic rows
    double* R = M.total > 0 ? M.scratch + ((int64_t)blockIdx.x * SOFT_WARPS + w) * M.total * 9 : nullptr;
    const Tune tu = make_tune(iterations);
    unsigned long long c_gh = 0, c_f64 = 0, c_esc = 0, c_sites = 0, c_sites64 = 0;
    for (;;) {
        unsigned long long r = 0;
        if (lane == 0) r = atomicAdd(next, 1ull);
        r = __shfl_sync(0xffffffffu, r, 0);
        if ((int64_t)r >= n_rows) break;
        int64_t lo = 0, hi = ns - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) / 2;
            if (mid * ns - mid * (mid - 1) / 2 <= (int64_t)r) lo = mid;
            else hi = mid - 1;
        }
        const int64_t x = lo, y = x + ((int64_t)r - (x * ns - x * (x - 1) / 2));
        double xv[9];
#pragma unroll
        for (int i = 0; i < 9; i++) xv[i] = x == y ? 0.0 : 1.0 / 9.0;
        if (x == y) { xv[0] = 0.5; xv[6] = 0.5; }
        normalise9(xv);
        bool fp64 = prec64 != 0;
        if (M.total > 0) soft_multi_build(M, x, y, lane, R);
        // one evaluation at xt: FP64, or FP32 (a difference pass relative to xc
        // and the objective f_old there when diff)
        PairEval ev;
        auto eval = [&](const double* xt, const double* xc, bool diff, double f_old) -> int64_t {
            c_gh++;
            int64_t m;
            if (fp64) {
                c_f64++;
                m = soft_evaluate(gl, n_sites, kept, kp, kq, nk, x, y, xt, tu.epsilon, lane, hs, R, M.total, ev);
                c_sites64 += (unsigned long long)m;
            } else {
                double step[9];
                difference_step(xt, xc, step);
                m = diff ? soft_evaluate32<true>(g32, pq32, nk, x, y, xt, step, xc, f_old, tu.epsilon, lane, hs, slots,
                                                 R, M.total, ev)
                         : soft_evaluate32<false>(g32, pq32, nk, x, y, xt, step, xc, f_old, tu.epsilon, lane, hs, slots,
                                                  R, M.total, ev);
            }
            c_sites += (unsigned long long)m;
            return m;
        };
        const int64_t n = eval(xv, xv, false, 0.0);
        kg_output* o = out + r;
        if (n == 0) {
            if (lane == 0) {
                o->x = (uint64_t)x;
                o->y = (uint64_t)y;
                for (int i = 0; i < 9; i++) o->jacquard[i] = 0.0;
                o->obj = CUDART_NAN;
                o->iters = 0;
                o->cond = CUDART_NAN;
                atomicOr(no_rows, 1);
            }
            continue;
        }
        double f = ev.f, g[9], Hr[9];
#pragma unroll
        for (int i = 0; i < 9; i++) { g[i] = ev.g[i]; Hr[i] = ev.Hr[i]; }
        uint64_t iters = tu.sqp_max_iter;
        double cond = CUDART_NAN;
        int near_count = 0;
        for (uint64_t it = 0; it < tu.sqp_max_iter; it++) {
            double resid;
            bool conv = kkt_ok(xv, g, tu.sqp_conv_tol, &resid);
            if (!fp64 && (conv || resid < 1e-6)) {
                if (!conv) near_count++;
                soft_share_hessian(Hr, lane, hs);
                const double c32 = conv ? soft_condition(hs, xv, g, tu.sqp_conv_tol) : 0.0;
                if (conv ? !(c32 <= COND_RECHECK) : (near_count >= 3)) {
                    // FP64 re-evaluation at the same point; the pair stays FP64
                    fp64 = true;
                    c_esc++;
                    eval(xv, xv, false, 0.0);
                    f = ev.f;
#pragma unroll
                    for (int i = 0; i < 9; i++) { g[i] = ev.g[i]; Hr[i] = ev.Hr[i]; }
                    conv = kkt_ok(xv, g, tu.sqp_conv_tol, &resid);
                } else if (conv) {
                    iters = it;
                    cond = c32;
                    break;
                }
            }
            if (conv) {
                iters = it;
                soft_share_hessian(Hr, lane, hs);
                cond = soft_condition(hs, xv, g, tu.sqp_conv_tol);
                break;
            }
            double cr = 0.0;
            if (lane < 9) cr = pick9(g, lane) - dot_fma(9, Hr, xv);
            double yv[9], p[9];
            soft_share_hessian(Hr, lane, hs);
            if (lane < 9) hs[QP_Q + lane] = cr;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 9; i++) yv[i] = xv[i];
            soft_qp(hs, tu, yv);
            __syncwarp();   // every lane has read hs before the next sums
#pragma unroll
            for (int i = 0; i < 9; i++) p[i] = yv[i] - xv[i];
            const double gp = dot_fma(9, g, p);
            const double tt = tu.bls_sufficient_decrease * gp;
            double alpha = 1.0, xn[9];
            for (int bls = 0;;) {
#pragma unroll
                for (int i = 0; i < 9; i++) xn[i] = xv[i] + alpha * p[i];
                normalise9(xn);
                const bool change = fabs(alpha * gp) < DIFF_BELOW;
                eval(xn, xv, change, f);
                // the change itself resolves the test far below an ulp of f
                const bool accept = change && !fp64 ? ev.df <= alpha * tt : ev.f <= f + alpha * tt;
                bls++;
                if (accept || bls == tu.bls_max_iter) break;
                alpha *= tu.bls_step_size_reduce;
            }
#pragma unroll
            for (int i = 0; i < 9; i++) { xv[i] = xn[i]; g[i] = ev.g[i]; Hr[i] = ev.Hr[i]; }
            f = ev.f;
        }
        if (lane == 0) {
            o->x = (uint64_t)x;
            o->y = (uint64_t)y;
            for (int i = 0; i < 9; i++) o->jacquard[i] = xv[i];
            o->obj = f;
            o->iters = iters;
            o->cond = cond;
        }
    }
    if (lane == 0) {
        atomicAdd(&stats[0], c_gh);
        atomicAdd(&stats[1], c_f64);
        atomicAdd(&stats[2], c_esc);
        atomicAdd(&stats[3], c_sites);
        atomicAdd(&stats[4], c_sites64);
    }
}

// ------------------------------------------------------------------- waves

// what changes from call to call, in device memory (the launches are a graph)
struct SoftCall {
    const double* gl;
    const int32_t* kept;
    const double *kp, *kq;
    const float4 *g32, *pq32;
    int64_t n_sites, nk;
};

__global__ void soft_init_kernel(SlotArgs A, int n, unsigned long long max_waves) { init_slot(A, 1, n, max_waves); }

// A pass's sums of a slot: sum L L' r^2 (45, upper triangle), sum L r (9), the
// objective sum, the sites.
constexpr int SOFT_PART = 56;

// A block per slot of the pass list, its warps every fourth group of 32 sites
// (or site pairs): a wave over few slots lasts a quarter of a warp's site loop.
// The warps' sums are added in a fixed order; two blocks per SM (255 registers,
// no spills: with three, 168 registers, 200 samples x 15,000 sites took 20.2
// against 15.0 ms).
__global__ void __launch_bounds__(SOFT_WARPS * 32, 2) soft_pass_kernel(SlotArgs A, const SoftCall* call,
                                                                      double* partial) {
    extern __shared__ __align__(16) unsigned char soft_smem[];   // SOFT_WARP_SMEM per warp
    __shared__ double part_sum[SOFT_WARPS][11];
    __shared__ double total[45];
    if (A.clk->stop) return;   // a device loop past its last wave
    if (threadIdx.x == 0) atomicMin(&A.clk->start[1], global_ns());
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const PhaseEnd pe{&A.clk->end[1], lane == 0};
    double* hs = reinterpret_cast<double*>(soft_smem + w * SOFT_WARP_SMEM);
    float4* slots = reinterpret_cast<float4*>(soft_smem + w * SOFT_WARP_SMEM + SOFT_SUMS_BYTES);
    const SoftCall C = *call;
    const int n_list = A.ctl->n[A.par];
    const PairSeg sg = A.seg[0];
    for (int i = blockIdx.x; i < n_list; i += gridDim.x) {
        const int s = A.list_cur[i];
        const int kind = A.count[s].w & 7;
        int64_t x, y;
        pair_of(sg.idx0 + (s - sg.slot0), x, y);
        const double* st = A.state + slot_at(s, NS_VALS);
        double xt[9], step[9], G[9], F;
        int64_t n;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            xt[k] = st[(NS_XT + k) * NS_LANES];
            step[k] = kind == NP_DIFF ? st[(NS_STEP + k) * NS_LANES] : 0.0;
        }
        if (kind >= NP_FP64)
            soft_sites64(C.gl, C.n_sites, C.kept, C.kp, C.kq, C.nk, x, y, xt, A.tune.epsilon, lane, w, SOFT_WARPS, hs, G,
                         F, n);
        else if (kind == NP_DIFF)
            soft_sites32<true>(C.g32, C.pq32, C.nk, x, y, xt, step, A.tune.epsilon, lane, w, SOFT_WARPS, hs, slots, G, F, n);
        else
            soft_sites32<false>(C.g32, C.pq32, C.nk, x, y, xt, step, A.tune.epsilon, lane, w, SOFT_WARPS, hs, slots, G, F,
                                n);
        // warp sums (fixed butterfly order), then the block's
        for (int off = 16; off > 0; off >>= 1) {
            F += __shfl_xor_sync(0xffffffffu, F, off);
            n += __shfl_xor_sync(0xffffffffu, n, off);
#pragma unroll
            for (int k = 0; k < 9; k++) G[k] += __shfl_xor_sync(0xffffffffu, G[k], off);
        }
        if (lane < 9) part_sum[w][lane] = pick9(G, lane);
        if (lane == 9) part_sum[w][9] = F;
        if (lane == 10) part_sum[w][10] = (double)n;
        __syncthreads();
        double* P = partial + slot_at(s, SOFT_PART);
        for (int a = w; a < 45; a += SOFT_WARPS) {
            double h = 0.0;
#pragma unroll
            for (int v = 0; v < SOFT_WARPS; v++)
                h += reinterpret_cast<const double*>(soft_smem + v * SOFT_WARP_SMEM)[a * HS + lane];
            for (int off = 16; off > 0; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
            if (lane == 0) {
                total[a] = h;
                P[a * NS_LANES] = h;
            }
        }
        __syncthreads();
        if (w == 0 && lane < 11) {
            double v = 0.0;
#pragma unroll
            for (int u = 0; u < SOFT_WARPS; u++) v += part_sum[u][lane];
            if (kind < NP_FP64) {
                // the lo parts of x to first order: sum log d gains sum_j lo_j
                // G_j, and G_i loses sum_j H_ij lo_j (a difference pass's
                // objective uses the step's FP32 values)
                double corr = 0.0;
#pragma unroll
                for (int j = 0; j < 9; j++) {
                    const double lo = xt[j] - (double)(float)xt[j], gj = __shfl_sync(0x7FFu, v, j);
                    const int r = min(lane, 8);
                    corr = fma(lane < 9 ? total[r <= j ? upper_at(r, j) : upper_at(j, r)] : gj, lo, corr);
                }
                if (lane < 9) v -= corr;
                else if (lane == 9 && kind != NP_DIFF) v = v * 0.69314718055994530942 + corr;
            }
            P[(45 + lane) * NS_LANES] = v;
        }
        __syncthreads();   // the sums are read before the next slot's
    }
}

struct SoftSums {
    static constexpr bool FP32 = true, COEF = false;
    const double* partial;
    static __device__ double none() { return 0.0; }
    __device__ __forceinline__ void load(int s, int, double*, double& obj, double (&g)[9], double (&T)[QP_Q],
                                         double& nsites) const {
        const double* P = partial + slot_at(s, SOFT_PART);
#pragma unroll
        for (int k = 0; k < QP_Q; k++) T[k] = P[k * NS_LANES];
#pragma unroll
        for (int k = 0; k < 9; k++) g[k] = P[(45 + k) * NS_LANES];
        obj = P[54 * NS_LANES];
        nsites = P[55 * NS_LANES];
    }
    // (soft_relatedness reads them back: FP64 passes and their sites)
    __device__ __forceinline__ void count(int, int, int, int f64p, double nsites, bool, unsigned long long* sum) const {
        atomicAdd(&sum[7], (unsigned long long)f64p);
        atomicAdd(&sum[6], (unsigned long long)nsites * (unsigned long long)f64p);
    }
};

__global__ void __launch_bounds__(NA_THREADS) soft_advance_kernel(SlotArgs A, const double* partial, int in_loop,
                                                                  cudaGraphConditionalHandle loop) {
    advance_wave(A, SoftSums{partial}, in_loop, loop);
}

// Pairs in flight at most (0.26 GB of slots): far more than the SMs hold, and a
// chunk's tail of waves over few pairs is short beside its first ones.
constexpr int64_t SOFT_SLOTS = (int64_t)1 << 18;

// The waves' graph and buffers, kept between calls.
struct SoftWaves {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    DevBuf slots, words;
    PinBuf host;
    int64_t cap = 0;
    uint64_t iterations = 0;
    int dev = -1;
    cudaStream_t st = nullptr;
    SlotArgs args[2]{};
    double* partial = nullptr;
    int pass_blocks = 0, advance_blocks = 0;
    void drop() {
        if (x) cudaGraphExecDestroy(x);
        if (g) cudaGraphDestroy(g);
        x = nullptr;
        g = nullptr;
        cap = 0;
    }
    ~SoftWaves() { drop(); }
};

// What a call's waves read and write beside the slots, one buffer on the device
// and its copy on the host.
struct SoftWords {
    CohortDev co;
    PairSeg seg;
    SoftCall call;
    SlotCtl ctl;
    WaveClock clk;
    RunCounters run;
};

static void launch_soft_wave(const SoftWaves& E, const SoftWords* D, int par, int in_loop, cudaGraphConditionalHandle h,
                             cudaStream_t st) {
    soft_pass_kernel<<<E.pass_blocks, SOFT_WARPS * 32, SOFT_SMEM, st>>>(E.args[par], &D->call, E.partial);
    soft_advance_kernel<<<E.advance_blocks, NA_THREADS, 0, st>>>(E.args[par], E.partial, in_loop, h);
}

static int run_soft_waves(SoftWork& w, const SoftCall& call, int64_t ns, uint64_t iterations, kg_output* d_out,
                          cudaStream_t st, std::string& err, uint64_t* counters) {
    if (!w.waves) w.waves = std::make_shared<SoftWaves>();
    SoftWaves& E = *w.waves;
    int dev = 0, sms = 148;
    KG_SOFT_TRY(cudaGetDevice(&dev));
    KG_SOFT_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t total = ns * (ns + 1) / 2;
    const size_t per_slot = sizeof(double) * (NS_VALS + SOFT_PART) + sizeof(int4) + 2 * sizeof(int);
    const int64_t cap = (std::min<int64_t>(total, SOFT_SLOTS) + 31) / 32 * 32;
    if (E.cap < cap || E.iterations != iterations || E.dev != dev || E.st != st) {
        int64_t keep = E.dev == dev ? std::max<int64_t>(E.cap, cap) : cap;
        E.drop();
        // fewer pairs in flight where the memory is short
        cudaError_t e;
        while ((e = (cudaError_t)E.slots.reserve(per_slot * (size_t)keep)) == cudaErrorMemoryAllocation && keep > 4096) {
            cudaGetLastError();
            keep = keep / 64 * 32;
        }
        KG_SOFT_TRY(e);
        KG_SOFT_TRY((cudaError_t)E.words.reserve(sizeof(SoftWords)));
        KG_SOFT_TRY((cudaError_t)E.host.reserve(sizeof(SoftWords)));
        SoftWords* D = E.words.as<SoftWords>();
        SlotArgs A{};
        A.cohorts = &D->co;
        A.seg = &D->seg;
        A.state = E.slots.as<double>();
        E.partial = A.state + (size_t)NS_VALS * keep;
        A.count = reinterpret_cast<int4*>(E.partial + (size_t)SOFT_PART * keep);
        int* lists = reinterpret_cast<int*>(A.count + keep);
        A.ctl = &D->ctl;
        A.clk = &D->clk;
        A.counters = &D->run;
        A.tune = make_tune(iterations);
        for (int par = 0; par < 2; par++) {
            E.args[par] = A;
            E.args[par].par = par;
            E.args[par].list_cur = lists + (par ? keep : 0);
            E.args[par].list_next = lists + (par ? 0 : keep);
        }
        int occ = 0;
        KG_SOFT_TRY(cudaFuncSetAttribute(soft_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SOFT_SMEM));
        KG_SOFT_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, soft_pass_kernel, SOFT_WARPS * 32, SOFT_SMEM));
        E.pass_blocks = sms * std::max(1, occ);
        KG_SOFT_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, soft_advance_kernel, NA_THREADS, 0));
        E.advance_blocks = sms * std::max(1, occ);
        KG_SOFT_TRY(wave_loop_graph(
            st,
            [&](int par, int in_loop, cudaGraphConditionalHandle h) {
                launch_soft_wave(E, D, par, in_loop, h, st);
            },
            &E.g, &E.x));
        E.cap = keep;
        E.iterations = iterations;
        E.dev = dev;
        E.st = st;
    }
    SoftWords* D = E.words.as<SoftWords>();
    SoftWords* H = E.host.as<SoftWords>();
    *H = SoftWords{};
    H->co.kind = COHORT_TRIANGLE;
    H->co.n_x = ns;
    H->co.n_pairs = total;
    H->co.out = d_out;
    H->co.max_iter = iterations;
    H->call = call;
    const char* hw = std::getenv("KESTREL_HOST_WAVES");
    const bool host_waves = hw && hw[0] == '1';   // for kernel profilers, as in run_nodes
    uint64_t launches = 0;
    const unsigned long long bound = wave_bound(iterations, 2);
    for (int64_t at = 0; at < total; at += E.cap) {
        const int n = (int)std::min<int64_t>(E.cap, total - at);
        H->seg = PairSeg{at, 0, n, 0, 0};
        // the counters go on from chunk to chunk
        KG_SOFT_TRY(cudaMemcpyAsync(D, H, sizeof(SoftWords), cudaMemcpyHostToDevice, st));
        soft_init_kernel<<<(n + 127) / 128, 128, 0, st>>>(E.args[0], n, bound);
        KG_SOFT_TRY(cudaGetLastError());
        if (host_waves) {
            for (int par = 0;; par ^= 1) {
                launch_soft_wave(E, D, par, 0, cudaGraphConditionalHandle{}, st);
                launches += 2;
                KG_SOFT_TRY(cudaMemcpyAsync(H, D, sizeof(SoftWords), cudaMemcpyDeviceToHost, st));
                KG_SOFT_TRY(cudaStreamSynchronize(st));
                if (H->clk.stop) break;
            }
        } else {
            KG_SOFT_TRY(cudaGraphLaunch(E.x, st));
        }
        KG_SOFT_TRY(cudaMemcpyAsync(H, D, sizeof(SoftWords), cudaMemcpyDeviceToHost, st));
        KG_SOFT_TRY(cudaStreamSynchronize(st));
        if (H->clk.limit_hit) {
            err = "the wave loop reached its wave limit";
            return KG_ETIMEOUT;
        }
        launches += 1 + (host_waves ? 0 : 4 * H->clk.iters);
    }
    if (counters) {
        counters[0] = H->run.gh_passes;
        counters[1] = H->run.shape_sites[0];   // SoftSums::count
        counters[2] = H->run.fp64_pairs;
        counters[3] = H->run.work_units;
        counters[4] = H->run.flops_fp64;
        counters[5] = launches;
    }
    if (H->run.nosite_pairs) {
        err = "a pair shares no called segregating site";
        return KG_ENOSITES;
    }
    return KG_OK;
}

int soft_relatedness(SoftWork& w, const DevBuf& gl, int64_t n_samples, int64_t n_sites, int64_t ns,
                     uint64_t iterations, double maf, kg_output* d_out, cudaStream_t st, std::string& err,
                     int64_t* n_kept, int precision,
                     uint64_t* counters, const SoftMultiInput* multi, int64_t* multi_used) {
    if (!(maf >= 0.0)) maf = 1.0 / (2.0 * (double)n_samples);
    DevBuf &pf = w.pf, &qf = w.qf, &keep = w.keep, &idx = w.idx, &kp = w.kp, &kq = w.kq, &ctr = w.ctr;
    DevBuf &g32 = w.g32, &pq32 = w.pq32, &mgk = w.mgk, &mgidx = w.mgidx, &mrows = w.mrows, &mused = w.mused;
    DevBuf& mscratch = w.mscratch;
    KG_SOFT_TRY((cudaError_t)pf.reserve(sizeof(double) * n_sites));
    KG_SOFT_TRY((cudaError_t)qf.reserve(sizeof(double) * n_sites));
    KG_SOFT_TRY((cudaError_t)keep.reserve((size_t)n_sites));
    soft_freq_kernel<<<(unsigned)((n_sites + 3) / 4), 128, 0, st>>>(gl.as<double>(), n_samples, n_sites, maf,
                                                                        iterations, pf.as<double>(), qf.as<double>(),
                                                                        keep.as<uint8_t>());
    KG_SOFT_TRY(cudaGetLastError());
    // the kept sites, compacted on the host (one small copy each way)
    std::vector<double> hp((size_t)n_sites), hq((size_t)n_sites);
    std::vector<uint8_t> hk((size_t)n_sites);
    KG_SOFT_TRY(cudaMemcpyAsync(hp.data(), pf.p, sizeof(double) * n_sites, cudaMemcpyDeviceToHost, st));
    KG_SOFT_TRY(cudaMemcpyAsync(hq.data(), qf.p, sizeof(double) * n_sites, cudaMemcpyDeviceToHost, st));
    KG_SOFT_TRY(cudaMemcpyAsync(hk.data(), keep.p, (size_t)n_sites, cudaMemcpyDeviceToHost, st));
    KG_SOFT_TRY(cudaStreamSynchronize(st));
    std::vector<int32_t> ki;
    std::vector<double> kpv, kqv;
    for (int64_t v = 0; v < n_sites; v++)
        if (hk[(size_t)v]) {
            ki.push_back((int32_t)v);
            kpv.push_back(hp[(size_t)v]);
            kqv.push_back(hq[(size_t)v]);
        }
    const int64_t nk = (int64_t)ki.size();
    if (n_kept) *n_kept = nk;
    // tri- and tetra-allelic sites: frequencies, remaining alleles, rows
    SoftMultiDev M{};
    M.n[0] = multi ? multi->n3 : 0;
    M.n[1] = multi ? multi->n4 : 0;
    M.gl[0] = multi ? multi->gl3 : nullptr;
    M.gl[1] = multi ? multi->gl4 : nullptr;
    M.total = M.n[0] + M.n[1];
    unsigned long long mu[3] = {0, 0, 0};
    if (M.total > 0) {
        KG_SOFT_TRY((cudaError_t)mgk.reserve(sizeof(int32_t) * M.total));
        KG_SOFT_TRY((cudaError_t)mgidx.reserve((size_t)MAXG * M.total));
        KG_SOFT_TRY((cudaError_t)mrows.reserve(sizeof(double) * 9 * SOFT_MULTI_ROWS * (size_t)M.total));
        KG_SOFT_TRY((cudaError_t)mused.reserve(sizeof(unsigned long long) * 3));
        KG_SOFT_TRY(cudaMemsetAsync(mused.p, 0, sizeof(unsigned long long) * 3, st));
        M.gk = mgk.as<int32_t>();
        M.gidx = mgidx.as<uint8_t>();
        M.rows = mrows.as<double>();
        soft_multi_site_kernel<<<(unsigned)((M.total + 127) / 128), 128, 0, st>>>(
            M, n_samples, maf, iterations, mgk.as<int32_t>(), mgidx.as<uint8_t>(), mrows.as<double>(),
            mused.as<unsigned long long>());
        KG_SOFT_TRY(cudaGetLastError());
        KG_SOFT_TRY(cudaMemcpyAsync(mu, mused.p, sizeof(mu), cudaMemcpyDeviceToHost, st));
        KG_SOFT_TRY(cudaStreamSynchronize(st));
    }
    if (multi_used)
        for (int k = 0; k < 3; k++) multi_used[k] = (int64_t)mu[k];
    if (nk == 0 && mu[0] + mu[1] + mu[2] == 0) {
        err = "no segregating site left after allele-frequency filtering";
        return KG_ENOSITES;
    }
    const int64_t nk1 = std::max<int64_t>(nk, 1);   // buffers exist even with no biallelic site
    KG_SOFT_TRY((cudaError_t)idx.reserve(sizeof(int32_t) * nk1));
    KG_SOFT_TRY((cudaError_t)kp.reserve(sizeof(double) * nk1));
    KG_SOFT_TRY((cudaError_t)kq.reserve(sizeof(double) * nk1));
    KG_SOFT_TRY((cudaError_t)ctr.reserve(sizeof(unsigned long long) * 6 + sizeof(int)));
    KG_SOFT_TRY(cudaMemcpyAsync(idx.p, ki.data(), sizeof(int32_t) * nk, cudaMemcpyHostToDevice, st));
    KG_SOFT_TRY(cudaMemcpyAsync(kp.p, kpv.data(), sizeof(double) * nk, cudaMemcpyHostToDevice, st));
    KG_SOFT_TRY(cudaMemcpyAsync(kq.p, kqv.data(), sizeof(double) * nk, cudaMemcpyHostToDevice, st));
    KG_SOFT_TRY(cudaMemsetAsync(ctr.p, 0, sizeof(unsigned long long) * 6 + sizeof(int), st));
    unsigned long long* next = ctr.as<unsigned long long>();
    unsigned long long* stats = next + 1;
    int* no_rows = reinterpret_cast<int*>(next + 6);
    const bool fp64 = precision == KG_PREC_FP64;
    if (!fp64) {
        const int64_t pairs = (nk1 + 1) / 2;   // of sites
        KG_SOFT_TRY((cudaError_t)g32.reserve(sizeof(float4) * 2 * (size_t)(n_samples * pairs)));
        KG_SOFT_TRY((cudaError_t)pq32.reserve(sizeof(float4) * pairs));
        const int64_t total = n_samples * ((nk + 1) / 2);
        if (total > 0) {
            const unsigned blocks = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 16);
            soft_pack32_kernel<<<blocks, 256, 0, st>>>(gl.as<double>(), n_samples, n_sites, idx.as<int32_t>(),
                                                       kp.as<double>(), kq.as<double>(), nk, g32.as<float4>(),
                                                       pq32.as<float4>());
        }
    }
    if (!fp64 && M.total == 0) {
        const SoftCall call{gl.as<double>(),    idx.as<int32_t>(),  kp.as<double>(), kq.as<double>(),
                            g32.as<float4>(),   pq32.as<float4>(), n_sites,         nk};
        return run_soft_waves(w, call, ns, iterations, d_out, st, err, counters);
    }
    const int64_t rows = ns * (ns + 1) / 2;
    int dev = 0, sms = 148;
    KG_SOFT_TRY(cudaGetDevice(&dev));
    KG_SOFT_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int occ = 0;
    KG_SOFT_TRY(cudaFuncSetAttribute(soft_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SOFT_SMEM));
    KG_SOFT_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, soft_pairs_kernel, SOFT_WARPS * 32, SOFT_SMEM));
    const int64_t grid = (int64_t)sms * std::max(1, occ);
    if (M.total > 0) {
        KG_SOFT_TRY((cudaError_t)mscratch.reserve(sizeof(double) * 9 * (size_t)(grid * SOFT_WARPS * M.total)));
        M.scratch = mscratch.as<double>();
    }
    soft_pairs_kernel<<<(unsigned)grid, SOFT_WARPS * 32, SOFT_SMEM, st>>>(
        gl.as<double>(), n_sites, idx.as<int32_t>(), kp.as<double>(), kq.as<double>(), g32.as<float4>(),
        pq32.as<float4>(), fp64 ? 1 : 0, nk, ns, rows, iterations, d_out, next, no_rows, stats, M);
    KG_SOFT_TRY(cudaGetLastError());
    int h_no_rows = 0;
    unsigned long long hs[5] = {0, 0, 0, 0, 0};
    KG_SOFT_TRY(cudaMemcpyAsync(&h_no_rows, no_rows, sizeof(int), cudaMemcpyDeviceToHost, st));
    KG_SOFT_TRY(cudaMemcpyAsync(hs, stats, sizeof(hs), cudaMemcpyDeviceToHost, st));
    KG_SOFT_TRY(cudaStreamSynchronize(st));
    if (counters)
        for (int i = 0; i < 5; i++) counters[i] = hs[i];
    if (h_no_rows) {
        err = "a pair shares no called segregating site";
        return KG_ENOSITES;
    }
    return KG_OK;
}

}  // namespace kg
