// kg_node.cu — pairs on frequency nodes (kg_node.h): the cohort's bins and
// digits, the integer matrix product that forms every pair's node weights on
// the tensor cores, the pass over nodes, and the host loop.
//
// Layout of a prepared cohort.  A kept site is folded to its rarer allele: t =
// min(p, 1 - p), genotypes 0 and 2 exchanged where p > 1/2.  Bins are double:
// bin k holds the sites with t in its interval, whose folded genotype pairs
// (0,0), (0,1), ... see the frequency t and whose pairs (2,2), (2,1), ... see
// 1 - t, so the nine genotype pairs of a bin are nine sets of nodes:
//   u     0    1    2    3    4    5    6    7    8
//   gx,gy 0,0  2,2  0,1  2,1  1,0  1,2  0,2  2,0  1,1
//   shape A    A    B1   B1   B2   B2   C    C    D
//   at    t    1-t  t    1-t  t    1-t  t    1-t  t
// Sites are stored bin by bin, each bin padded to NODE_STAGE sites:
//   nd_planes [sample][word] {lo, hi} bit planes of 32 folded sites (3: missing
//             or padding)
//   nd_dig    [column][site] signed digits: column j * L + l (of 32) holds digit
//             l (256^l) of round(2^30 l_j(t)), l_j the Lagrange basis of the
//             bin's nodes.  Within a word of 32 sites
//             byte 4 q + i is site q + 8 i, the order in which four shifted
//             bits of a plane word become four bytes with one AND.
// CLS needs sum t^k, k <= 4, only, for which the same eight nodes are exact on
// one interval [0, 1/2] (five would be): its bins are equal runs of sites (to
// spread a small cohort over the SMs), all on that interval.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "kg_advance.cuh"
#include "kg_bulk.cuh"
#include "kg_engine.h"
#include "kg_log.cuh"
#include "kg_node.h"
#include "kg_pair.cuh"
#include "kg_qp1.cuh"
#include "kg_tmem.cuh"
#include "kg_wave.cuh"

namespace kg {

#define KG_NODE_TRY(expr)                                                       \
    do {                                                                        \
        cudaError_t e_ = (expr);                                                \
        if (e_ != cudaSuccess) {                                                \
            err = std::string(#expr) + ": " + cudaGetErrorString(e_);           \
            return e_ == cudaErrorMemoryAllocation ? KG_ENOMEM : KG_ECUDA;      \
        }                                                                       \
    } while (0)

// ------------------------------------------------------------ preparation

// A double bin: its first site (a multiple of NODE_STAGE), its stages.
struct NodeBin {
    int32_t start, stages;
};

int node_bins(bool cls, int64_t n_kept, int64_t n_samples, double t_min) {
    if (n_kept <= 0 || n_samples <= 0) return 0;
    // places, padding included, are 32-bit
    if (n_kept > (int64_t)INT_MAX - (NODE_MAX_BINS + 1) * NODE_STAGE) return 0;
    if (cls) {
        if (!(t_min >= 0.0)) return 0;
        const int64_t by_work = (n_kept + 1023) / 1024, by_sms = 296 / n_samples + 1;
        return (int)std::max<int64_t>(1, std::min<int64_t>({by_work, by_sms, 16}));
    }
    if (!(t_min > 0.0) || t_min > 0.5) return 0;
    const double need = std::ceil(std::log(0.5 / t_min) / std::log(NODE_RATIO));
    if (!(need <= (double)NODE_MAX_BINS)) return 0;
    return std::max(1, (int)need);
}

constexpr int NODE_PLACE_THREADS = 512;

// What places a folded frequency: bin edges 1/2 * q^k (q < 1), or equal runs.
struct NodeGrid {
    int bins;
    int by_index;      // CLS: bins are runs of sites on [0, 1/2]
    double q;          // ratio of a bin's lower to its upper end
    double inv_log_q;
    int64_t n_kept;
};

__device__ __forceinline__ void bin_interval(const NodeGrid& G, int k, double& lo, double& hi) {
    if (G.by_index) {
        lo = 0.0;
        hi = 0.5;
    } else {
        hi = 0.5 * pow(G.q, (double)k);
        lo = hi * G.q;
    }
}

// (site: its index among the kept ones; p: its REF frequency)
__device__ __forceinline__ int bin_of(const NodeGrid& G, int64_t site, double p) {
    if (G.by_index) return (int)(site * G.bins / G.n_kept);
    const double t = fmin(p, 1.0 - p);
    const int k = (int)floor(log(2.0 * t) * G.inv_log_q);
    return min(max(k, 0), G.bins - 1);
}

__global__ void node_hist_kernel(NodeGrid G, const double* __restrict__ p64, int* __restrict__ hist) {
    __shared__ int h[NODE_MAX_BINS];
    for (int k = threadIdx.x; k < G.bins; k += blockDim.x) h[k] = 0;
    __syncthreads();
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < G.n_kept) atomicAdd(&h[bin_of(G, s, p64[freq_index(s)])], 1);
    __syncthreads();
    for (int k = threadIdx.x; k < G.bins; k += blockDim.x)
        if (h[k]) atomicAdd(&hist[k], h[k]);
}

// One block: the bins' starts and stages from the histogram (which becomes
// the places' cursors) and the node points.
__global__ void node_layout_kernel(NodeGrid G, int* __restrict__ hist, NodeBin* __restrict__ bin,
                                   double* __restrict__ t) {
    constexpr int J = NODE_J;
    if (threadIdx.x == 0) {
        int at = 0;
        for (int k = 0; k < G.bins; k++) {
            const int st = (hist[k] + NODE_STAGE - 1) / NODE_STAGE;
            bin[k] = NodeBin{at, st};
            hist[k] = at;
            at += st * NODE_STAGE;
        }
    }
    for (int e = threadIdx.x; e < G.bins * J; e += blockDim.x) {
        const int k = e / J, j = e - k * J;
        double lo, hi;
        bin_interval(G, k, lo, hi);
        t[e] = 0.5 * (lo + hi) - 0.5 * (hi - lo) * cospi((2 * j + 1) / (2.0 * J));
    }
}

// Kept sites to their places: place[pos] = raw site, bit 31 set where the
// genotypes are exchanged (the order of a bin's blocks does not matter: the sums
// are integers).  A block counts its sites per bin in shared memory and takes
// one run of places per bin; within a warp they follow the site order.
__global__ void __launch_bounds__(NODE_PLACE_THREADS) node_place_kernel(NodeGrid G, const double* __restrict__ p64,
                                                                        const int32_t* __restrict__ site_of,
                                                                        int* __restrict__ cursor,
                                                                        uint32_t* __restrict__ place) {
    __shared__ int count[NODE_MAX_BINS], base[NODE_MAX_BINS];
    for (int k = threadIdx.x; k < G.bins; k += blockDim.x) count[k] = 0;
    __syncthreads();
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = s < G.n_kept;
    const double p = live ? p64[freq_index(s)] : 0.5;
    const int k = live ? bin_of(G, s, p) : -1, lane = threadIdx.x & 31;
    const unsigned same = __match_any_sync(0xffffffffu, k);
    const int first = __ffs(same) - 1;
    int at = 0;
    if (live && lane == first) at = atomicAdd(&count[k], __popc(same));
    at = __shfl_sync(0xffffffffu, at, first) + __popc(same & ((1u << lane) - 1u));
    __syncthreads();
    for (int i = threadIdx.x; i < G.bins; i += blockDim.x)
        if (count[i]) base[i] = atomicAdd(&cursor[i], count[i]);
    __syncthreads();
    if (live) place[base[k] + at] = (uint32_t)site_of[s] | (p > 0.5 ? 0x80000000u : 0u);
}

// The digits of the placed sites' basis values, a thread per place: a warp's 32
// bytes of a column are one sector.  (Written by the sites' threads, in the order
// of the kept sites, every byte was a sector of its own: 2.1 ms for 3,000,000
// sites, the places' atomics included, against 0.13 ms.)  Places without a site:
// zeros.  pf: REF frequencies of the raw sites.
__global__ void __launch_bounds__(256) node_digits_kernel(NodeGrid G, const double* __restrict__ pf,
                                                          const uint32_t* __restrict__ place, int8_t* __restrict__ dig,
                                                          int64_t mp) {
    constexpr int J = NODE_J, L = NODE_L;
    // the first-kind Chebyshev points z_j = -cos((2j+1) pi / 2J) and their
    // barycentric weights
    __shared__ double zc[J], wj[J];
    if (threadIdx.x < J) {
        const int j = threadIdx.x;
        zc[j] = cospi((2 * j + 1) / (2.0 * J));
        wj[j] = ((j & 1) ? -1.0 : 1.0) * sinpi((2 * j + 1) / (2.0 * J));
    }
    __syncthreads();
    const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= mp) return;
    const int64_t byte = (pos & ~(int64_t)31) | ((pos & 7) << 2) | ((pos >> 3) & 3);
    const uint32_t e = place[pos];
    if (e == 0xFFFFFFFFu) {
        for (int c = 0; c < J * L; c++) dig[c * mp + byte] = 0;
        return;
    }
    const double p = pf[e & 0x7FFFFFFFu];
    const double t = fmin(p, 1.0 - p);
    double lo, hi;
    bin_interval(G, G.by_index ? 0 : bin_of(G, 0, p), lo, hi);
    const double z = (t - 0.5 * (lo + hi)) / (0.5 * (hi - lo));
    double b[J], sum = 0.0;
    int hit = -1;
#pragma unroll
    for (int j = 0; j < J; j++) {
        const double dz = z + zc[j];
        if (dz == 0.0) hit = j;
        b[j] = wj[j] / dz;
        sum += b[j];
    }
    // fixed point, the rounding errors' sum taken by the largest: the weights
    // of a site add up to 1 exactly, so sites of one frequency, whose errors
    // are the same, shift no sum by a constant (and a pair's weights count
    // its sites)
    constexpr long long ONE = 1ll << (8 * L - 2);
    long long fx[J], total = 0;
    int top = 0;
#pragma unroll
    for (int j = 0; j < J; j++) {
        const double l = hit >= 0 ? (j == hit ? 1.0 : 0.0) : b[j] / sum;
        fx[j] = __double2ll_rn(l * (double)ONE);
        total += fx[j];
        if (l > 0.5) top = j;
    }
#pragma unroll
    for (int j = 0; j < J; j++) {
        long long v = fx[j] + (j == top ? ONE - total : 0ll);
#pragma unroll
        for (int d = 0; d < L; d++) {
            const int lo8 = (int)((v + 128) & 255) - 128;
            dig[(int64_t)(j * L + d) * mp + byte] = (int8_t)lo8;
            v = (v - lo8) >> 8;
        }
    }
}

// A block per (sample, part): warps build the folded {lo, hi} planes of 32
// placed sites a time; the sample's codes are read through L1.  mask: sites to
// keep (NULL: all).
__global__ void node_pack_kernel(const uint8_t* __restrict__ raw, int64_t stride, const uint8_t* __restrict__ mask,
                                 const uint32_t* __restrict__ place, int64_t words, uint2* __restrict__ planes) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint8_t* row = raw + (int64_t)blockIdx.x * stride;
    uint2* out = planes + (int64_t)blockIdx.x * words;
    for (int64_t k = (int64_t)blockIdx.y * nw + w; k < words; k += (int64_t)gridDim.y * nw) {
        const uint32_t e = place[k * 32 + lane];
        unsigned c = 3u;
        if (e != 0xFFFFFFFFu) {
            c = row[e & 0x7FFFFFFFu];
            if (mask && !mask[e & 0x7FFFFFFFu]) c = 3u;
            if ((e >> 31) && c < 3u) c = 2u - c;
        }
        const unsigned lo = __ballot_sync(0xffffffffu, c & 1u), hi = __ballot_sync(0xffffffffu, (c >> 1) & 1u);
        if (lane == 0) out[k] = make_uint2(lo, hi);
    }
}

static void pack_placed(const uint8_t* codes, int64_t rows, int64_t stride, const uint8_t* mask, const DevBuf& place,
                        int64_t mp, const DevBuf& planes, cudaStream_t st) {
    // enough blocks to fill the SMs, few enough that a sample's row is read by few
    const int64_t words = mp / 32;
    const int parts = (int)std::max<int64_t>(1, std::min<int64_t>((words + 63) / 64, 1184 / rows + 1));
    node_pack_kernel<<<dim3((unsigned)rows, parts), 256, 0, st>>>(codes, stride, mask, place.as<uint32_t>(), words,
                                                                  planes.as<uint2>());
}

int prepare_nodes(Cohort& c, const uint8_t* codes, int64_t stride, int bins, cudaStream_t st, std::string& err) {
    const int64_t mp = ((c.n_kept + NODE_STAGE - 1) / NODE_STAGE + bins) * NODE_STAGE;
    NodeGrid G;
    G.bins = bins;
    G.by_index = c.cls ? 1 : 0;
    // the last bin holds the smallest frequency and reaches below it, by less than a bin
    G.q = c.cls ? 1.0 : 1.0 / NODE_RATIO;
    G.inv_log_q = c.cls ? 0.0 : 1.0 / std::log(G.q);
    G.n_kept = c.n_kept;
    const size_t head = sizeof(int) * NODE_MAX_BINS + sizeof(NodeBin) * NODE_MAX_BINS;
    KG_NODE_TRY((cudaError_t)c.nd_bins.reserve(head));
    KG_NODE_TRY((cudaError_t)c.nd_t.reserve(sizeof(double) * bins * NODE_J));
    KG_NODE_TRY((cudaError_t)c.nd_place.reserve(sizeof(uint32_t) * mp));
    KG_NODE_TRY((cudaError_t)c.nd_dig.reserve((size_t)32 * mp));
    KG_NODE_TRY((cudaError_t)c.nd_planes.reserve(sizeof(uint2) * (mp / 32) * c.n_samples));
    int* hist = c.nd_bins.as<int>();
    NodeBin* bin = reinterpret_cast<NodeBin*>(hist + NODE_MAX_BINS);
    KG_NODE_TRY(cudaMemsetAsync(hist, 0, sizeof(int) * NODE_MAX_BINS, st));
    KG_NODE_TRY(cudaMemsetAsync(c.nd_place.p, 0xFF, sizeof(uint32_t) * mp, st));
    const int grid = (int)((c.n_kept + 255) / 256);
    node_hist_kernel<<<grid, 256, 0, st>>>(G, c.p64.as<double>(), hist);
    node_layout_kernel<<<1, 256, 0, st>>>(G, hist, bin, c.nd_t.as<double>());
    node_place_kernel<<<(int)((c.n_kept + NODE_PLACE_THREADS - 1) / NODE_PLACE_THREADS), NODE_PLACE_THREADS, 0, st>>>(
        G, c.p64.as<double>(), c.site_of.as<int32_t>(), hist, c.nd_place.as<uint32_t>());
    node_digits_kernel<<<(int)((mp + 255) / 256), 256, 0, st>>>(G, c.pfull.as<double>(), c.nd_place.as<uint32_t>(),
                                                               c.nd_dig.as<int8_t>(), mp);
    pack_placed(codes, c.n_samples, stride, nullptr, c.nd_place, mp, c.nd_planes, st);
    KG_NODE_TRY(cudaGetLastError());
    c.nd_n = bins;
    c.nd_mp = mp;
    return KG_OK;
}

int prepare_query_nodes(const Cohort& panel, QueryPlanes& q, const uint8_t* codes, int64_t n_rows, int64_t row_stride,
                        const uint8_t* site_mask, cudaStream_t st, std::string& err) {
    if (n_rows <= 0 || row_stride < panel.n_sites || !codes || panel.nd_n <= 0) {
        err = "query rows must be positive and cover the panel's sites";
        return KG_EINVAL;
    }
    const int64_t ns = panel.n_sites;
    q.n_rows = n_rows;
    KG_NODE_TRY((cudaError_t)q.raw.reserve((size_t)(n_rows * ns)));
    KG_NODE_TRY(cudaMemcpy2DAsync(q.raw.p, (size_t)ns, codes, (size_t)row_stride, (size_t)ns, (size_t)n_rows,
                                  cudaMemcpyHostToDevice, st));
    const uint8_t* dmask = nullptr;
    if (site_mask) {
        KG_NODE_TRY((cudaError_t)q.mask.reserve((size_t)ns));
        KG_NODE_TRY(cudaMemcpyAsync(q.mask.p, site_mask, (size_t)ns, cudaMemcpyHostToDevice, st));
        dmask = q.mask.as<uint8_t>();
    }
    KG_NODE_TRY((cudaError_t)q.planes.reserve(sizeof(uint2) * (panel.nd_mp / 32) * n_rows));
    pack_placed(q.raw.as<uint8_t>(), n_rows, ns, dmask, panel.nd_place, panel.nd_mp, q.planes, st);
    KG_NODE_TRY(cudaGetLastError());
    return KG_OK;
}

// --------------------------------------------------- the node weights W

// For a sample y and a block of 128 samples x, per bin: the nine products
//   D[a][b](x, column) = sum over the bin's sites of [g'x = a] [g'y = b] digit(column)
// on the integer tensor cores (M = 128 samples x, N = 3 x 32 columns, K = the
// bin's sites), then W = sum over digits of 256^l D, exact, as doubles.
//
// Indicators are one bit a site in HBM, 8 bits in the product: the A operand
// ([g'x = a], 128 x K) is expanded from the plane words straight into tensor
// memory, a thread per sample, and the B operand ([g'y = b] digits, 96 x K)
// into shared memory in the 128-byte swizzle.  With A in shared memory its
// 48 KB a stage would be written and read again through the 128 B/clk port,
// which B's 12 KB written and 36 KB read already keep busy half the time.
// Per stage of 128 sites: 12 instructions of 48 cycles.  Expanding A takes a
// warp longer than that (250 instructions, half of them at half rate, and the
// tensor-memory stores behind a wait), so two groups of four warps take half a
// stage each, into four half-stage buffers, and every expansion is in registers
// before its buffer is waited for.  A lone issuing thread was what bound the
// first form (18.2 ms at 1024 samples x 100,000 sites against 7.6 ms of
// instructions): a wait on a barrier that is long complete takes it 270 cycles,
// an instruction 30.  So three warps issue, one a genotype of x (their
// accumulators are apart), all lanes converged (one thread of a diverged warp
// took 25.5 ms), with one wait and one commit a half-stage.
// A sum of NODE_SEG_STAGES stages of digits fits the 32-bit accumulators
// whatever the digits (sites of one frequency have the same ones); a bin that
// may be longer is done in segments, which add up in 64 bits in memory.
constexpr int NW_THREADS = 608;          // 2 x 4 warps expand A, 4 expand B, 4 read out, 3 issue
constexpr int NW_N = 96;                 // B's rows: 3 genotypes of y x 32 columns
constexpr int NW_BSTAGE = NW_N * NODE_STAGE;
constexpr int NW_STAGES = 2;
constexpr int NW_AHEAD = 2;              // stages whose planes and digits a thread has in flight
constexpr uint32_t NW_TM_A = 320;        // tensor-memory column of A's half-stages, 48 each (D: 0 .. 287)
constexpr int NW_SMEM = 120 * 1024;      // more than half an SM's: one block (it owns the tensor memory)

struct NodeProduct {
    const uint2* planes;       // [sample][words] of the A operand's samples
    const uint2* planes_b;     // of the B operand's (a triangle: the same)
    const int8_t* dig;         // [32][mp]
    const NodeBin* bin;
    int64_t words, mp;
    int32_t n_samples;         // rows of planes
    int32_t rect;              // query x panel: A's samples are the panel's (y), B's the query's (x)
    int32_t bins;
    int64_t idx0, idx1;        // the pairs of this chunk: y (y + 1) / 2 + x, x <= y (rect: x n_samples + y)
    int64_t slot0;             // slot of pair idx0 within w's columns
    int64_t first_unit, n_yx;  // the first (y, x block) in the count from y = 0, how many
    int32_t seg, segs;         // stages of a unit at most, units a bin takes at most (1: no segments)
    double* w;                 // see NodeDev
    int64_t group;
    unsigned long long* stalled;
};

// (y, block of 128 samples x) number u, counted from y = 0: y has y / 128 + 1.
__host__ __device__ inline int64_t yx_before(int64_t y) {
    const int64_t q = y >> 7;
    return 64 * q * (q + 1) + (y - (q << 7)) * (q + 1);
}
// A unit: a segment of bin k for a (y, x block) pair; a segment's pairs follow
// one another.
struct NodeUnit {
    int y, xb, k;
    int start, stages;   // its first site and its stages (0: an empty bin)
};
// (B's sample, block of A's samples)
__device__ __forceinline__ void decode_yx(const NodeProduct& P, int64_t u, int& y, int& xb) {
    if (P.rect) {
        const int64_t nb = (P.n_samples + 127) >> 7;
        y = (int)(u / nb);
        xb = (int)(u - y * nb);
        return;
    }
    int64_t q = (int64_t)((sqrt(1.0 + (double)u / 16.0) - 1.0) * 0.5);
    while (q > 0 && 64 * q * (q + 1) > u) q--;
    while (64 * (q + 1) * (q + 2) <= u) q++;
    const int64_t r = u - 64 * q * (q + 1);
    y = (int)((q << 7) + r / (q + 1));
    xb = (int)(r % (q + 1));
}

// SEGS: bins in segments (seg0: each bin's first, then their number), else each
// bin a unit.
template <bool SEGS>
__device__ __forceinline__ NodeUnit node_unit(const NodeProduct& P, const int* seg0, int64_t un) {
    NodeUnit U;
    U.k = (int)(un / P.n_yx);
    decode_yx(P, P.first_unit + (un - U.k * P.n_yx), U.y, U.xb);
    int seg = 0, parts = 1;
    if (SEGS) {
        const int q = U.k;
        int lo = 0, hi = P.bins - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (seg0[mid] <= q) lo = mid;
            else hi = mid - 1;
        }
        U.k = lo;
        seg = q - seg0[lo];
        parts = seg0[lo + 1] - seg0[lo];
    }
    // (a bin's segments are equal to a stage, and none is empty)
    const NodeBin bn = P.bin[U.k];
    const int first = SEGS ? (int)((int64_t)bn.stages * seg / parts) : 0;
    U.stages = SEGS ? (int)((int64_t)bn.stages * (seg + 1) / parts) - first : bn.stages;
    U.start = bn.start + first * NODE_STAGE;
    return U;
}

// Bounded wait: false once the limit or another warp's has run out.
__device__ __forceinline__ bool nw_wait(uint64_t* bar, uint32_t parity, volatile int* gave_up) {
    for (uint32_t i = 0; i < MBAR_WAIT_LIMIT; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63) == 63 && *gave_up) return false;
    }
    *gave_up = 1;
    return false;
}
// The same for a whole warp, one answer for all its lanes.
__device__ __forceinline__ bool nw_wait_warp(uint64_t* bar, uint32_t parity, volatile int* gave_up) {
    return __all_sync(0xffffffffu, nw_wait(bar, parity, gave_up));
}
// A wait ran out: instructions that were issued may still read the operands and
// write the accumulators (else the last read-out has waited for all).  All warps
// call it; out of line: in the kernel it took 0.8% of it (512 x 100,000 CLS, 3.62
// against 3.59 ms).
__device__ __noinline__ void nw_drain(uint64_t* drained, int warp) {
    if (warp >= 16) {
        if (elect_one()) mma_commit(smem_u32(drained));
        __syncwarp();
        mbar_wait(drained, 0u);
    }
    __syncthreads();
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <bool SEGS>
__global__ void __launch_bounds__(NW_THREADS, 1) node_weights_kernel(NodeProduct P) {
    constexpr int J = NODE_J, L = NODE_L;
    extern __shared__ __align__(1024) unsigned char nw_smem[];
    // buffer 2 stage + half; B's stage arrives with its first half and is free
    // with its second
    __shared__ __align__(8) uint64_t full[2 * NW_STAGES], empty[2 * NW_STAGES], acc_full, acc_empty;
    __shared__ __align__(8) uint64_t drained;
    __shared__ uint32_t tm_slot;
    __shared__ int gave_up;
    __shared__ int seg0[SEGS ? NODE_MAX_BINS + 1 : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t b0 = (smem_u32(nw_smem) + 1023u) & ~1023u;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * NW_STAGES; i++) {
            mbar_init(&full[i], (i & 1) ? 4 : 8);   // four warps of A's, with the first half four of B's
            mbar_init(&empty[i], 3);                // the issuing warps
        }
        mbar_init(&acc_full, 3);
        mbar_init(&acc_empty, 4);
        mbar_init(&drained, 3);
        gave_up = 0;
        fence_mbar_init();
        if (SEGS) {
            int at = 0;
            for (int k = 0; k < P.bins; k++) {
                seg0[k] = at;
                at += (P.bin[k].stages + P.seg - 1) / P.seg;
            }
            seg0[P.bins] = at;
        }
    }
    if (warp == 16) tmem_alloc<512>(smem_u32(&tm_slot));
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tm = tm_slot;
    const int64_t n_units = P.n_yx * (SEGS ? seg0[P.bins] : P.bins);
    uint32_t seq = 0;    // stages so far
    bool ok = true;
    if (warp < 8) {
        // ---- A: a thread per sample x; group warp / 4 expands that half of
        // every stage, into buffers (2 stage + half) % 4
        const uint32_t half = warp >> 2;
        const uint32_t my = tm + ((uint32_t)((warp & 3) * 32) << 16) + NW_TM_A + half * 48;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const NodeUnit U = node_unit<SEGS>(P, seg0, un);
            const int x = U.xb * 128 + (warp & 3) * 32 + lane;
            const uint32_t live = x < P.n_samples ? ~0u : 0u;
            const uint4* src =
                reinterpret_cast<const uint4*>(P.planes + (int64_t)(live ? x : 0) * P.words + (U.start >> 5)) + half;
            uint4 v[NW_AHEAD];
#pragma unroll
            for (int j = 0; j < NW_AHEAD; j++)
                if (j < U.stages) v[j] = src[2 * j];
            for (int i0 = 0; ok && i0 < U.stages; i0 += NW_AHEAD) {
#pragma unroll
                for (int j = 0; j < NW_AHEAD; j++) {
                    const int i = i0 + j;
                    if (i >= U.stages) break;
                    const uint32_t lo[2] = {v[j].x, v[j].z}, hi[2] = {v[j].y, v[j].w};
                    if (i + NW_AHEAD < U.stages) v[j] = src[2 * (i + NW_AHEAD)];
                    uint32_t r[48];
#pragma unroll
                    for (int a = 0; a < 3; a++)
#pragma unroll
                        for (int w = 0; w < 2; w++) {
                            const uint32_t m =
                                (a == 0 ? ~(lo[w] | hi[w]) : a == 1 ? lo[w] & ~hi[w] : hi[w] & ~lo[w]) & live;
#pragma unroll
                            for (int q = 0; q < 8; q++) r[16 * a + 8 * w + q] = (m >> q) & 0x01010101u;
                        }
                    const uint32_t st = seq % NW_STAGES;
                    if (!nw_wait_warp(&empty[2 * st + half], ((seq / NW_STAGES) & 1u) ^ 1u, &gave_up)) { ok = false; break; }
                    tmem_fence_after();
#pragma unroll
                    for (int a = 0; a < 3; a++) tmem_store16(my + st * 96 + a * 16, r + 16 * a);
                    tmem_store_wait();
                    tmem_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[2 * st + half]);
                    seq++;
                }
            }
        }
    } else if (warp < 12) {
        // ---- B: thread (row, 16-site piece); rows row and row + 16 of the
        // 32 columns, for the three genotypes of y
        const int tid = threadIdx.x - 256, c = tid & 7, row = tid >> 3;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const NodeUnit U = node_unit<SEGS>(P, seg0, un);
            const int8_t* d0 = P.dig + (int64_t)row * P.mp + U.start + 16 * c;
            const uint2* py = P.planes_b + (int64_t)U.y * P.words + (U.start >> 5) + (c >> 1);
            uint4 va[NW_AHEAD], vb[NW_AHEAD];
            uint2 pl[NW_AHEAD];
            auto fetch = [&](int i, uint4& a4, uint4& b4, uint2& p2) {
                a4 = *reinterpret_cast<const uint4*>(d0 + (int64_t)i * NODE_STAGE);
                b4 = *reinterpret_cast<const uint4*>(d0 + 16 * P.mp + (int64_t)i * NODE_STAGE);
                p2 = py[4 * i];
            };
#pragma unroll
            for (int j = 0; j < NW_AHEAD; j++)
                if (j < U.stages) fetch(j, va[j], vb[j], pl[j]);
            for (int i0 = 0; ok && i0 < U.stages; i0 += NW_AHEAD) {
#pragma unroll
                for (int j = 0; j < NW_AHEAD; j++) {
                    const int i = i0 + j;
                    if (i >= U.stages) break;
                    const uint32_t lo = pl[j].x, hi = pl[j].y;
                    uint4 va3[3], vb3[3];
#pragma unroll
                    for (int b = 0; b < 3; b++) {
                        const uint32_t m = (b == 0 ? ~(lo | hi) : b == 1 ? lo & ~hi : hi & ~lo) >> (4 * (c & 1));
                        uint32_t f[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) f[q] = ((m >> q) & 0x01010101u) * 255u;
                        va3[b] = make_uint4(va[j].x & f[0], va[j].y & f[1], va[j].z & f[2], va[j].w & f[3]);
                        vb3[b] = make_uint4(vb[j].x & f[0], vb[j].y & f[1], vb[j].z & f[2], vb[j].w & f[3]);
                    }
                    if (i + NW_AHEAD < U.stages) fetch(i + NW_AHEAD, va[j], vb[j], pl[j]);
                    const uint32_t st = seq % NW_STAGES;
                    if (!nw_wait_warp(&empty[2 * st + 1], ((seq / NW_STAGES) & 1u) ^ 1u, &gave_up)) { ok = false; break; }
                    const uint32_t base = b0 + st * NW_BSTAGE + ((uint32_t)(c ^ (row & 7)) << 4);
#pragma unroll
                    for (int b = 0; b < 3; b++) {
                        const uint32_t at = base + (uint32_t)(b * 32 + row) * 128u;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(va3[b].x),
                                     "r"(va3[b].y), "r"(va3[b].z), "r"(va3[b].w)
                                     : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 16u * 128u), "r"(vb3[b].x),
                                     "r"(vb3[b].y), "r"(vb3[b].z), "r"(vb3[b].w)
                                     : "memory");
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[2 * st]);
                    seq++;
                }
            }
        }
    } else if (warp < 16) {
        // ---- read-out: a thread per sample x; lanes of consecutive x are
        // consecutive slots
        const uint32_t my = tm + ((uint32_t)((warp - 12) * 32) << 16);
        // the genotype pair's number u (see the file comment) of (gx, gy) = (a, b)
        // and, query x panel, of (b, a)
        constexpr int UNIT[9] = {0, 2, 6, 4, 8, 5, 7, 3, 1}, UNIT_T[9] = {0, 4, 7, 2, 8, 3, 6, 5, 1};
        uint32_t n_acc = 0;
        const int nk = P.bins * J;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const NodeUnit U = node_unit<SEGS>(P, seg0, un);
            const int y = U.y, k = U.k, x = U.xb * 128 + (warp - 12) * 32 + lane;
            const int64_t idx = P.rect ? (int64_t)y * P.n_samples + x : (int64_t)y * (y + 1) / 2 + x;
            const bool store = x < (P.rect ? P.n_samples : y + 1) && idx >= P.idx0 && idx < P.idx1;
            const int64_t s = P.slot0 + (idx - P.idx0);
            double* out = P.w + (s >> 3) * P.group + (int64_t)(k * J) * 8 + (s & 7);
            if (U.stages == 0) {
                // an empty bin: zero weights, no product
                if (store)
                    for (int u = 0; u < 9; u++)
                        for (int j = 0; j < J; j++) out[((int64_t)u * nk + j) * 8] = 0.0;
                continue;
            }
            if (!nw_wait_warp(&acc_full, n_acc & 1u, &gave_up)) { ok = false; break; }
            n_acc++;
            tmem_fence_after();
#pragma unroll
            for (int ab = 0; ab < 9; ab++) {
                uint32_t r[32];
                tmem_load32(my + (ab / 3) * NW_N + (ab % 3) * 32, r);
                if (ab == 8) {
                    // every column is in registers: the next unit may start
                    tmem_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty);
                }
#pragma unroll
                for (int j = 0; j < J; j++) {
                    long long v = (int)r[j * L];
#pragma unroll
                    for (int d = 1; d < L; d++) v += (long long)(int)r[j * L + d] * (1ll << (8 * d));
                    double* o = out + ((int64_t)(P.rect ? UNIT_T[ab] : UNIT[ab]) * nk + j) * 8;
                    if (store) {
                        if (SEGS) atomicAdd(reinterpret_cast<unsigned long long*>(o), (unsigned long long)v);
                        else *o = (double)v;
                    }
                }
            }
        }
    } else {
        // ---- the issuing warps, a genotype of x each: every lane waits, one issues
        constexpr uint32_t idesc = idesc_i8(128, NW_N);
        const uint32_t a = warp - 16, d = tm + a * NW_N, a0 = tm + NW_TM_A + a * 16;
        uint32_t n_acc = 0;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const int stages = node_unit<SEGS>(P, seg0, un).stages;
            if (stages == 0) continue;
            if (!nw_wait_warp(&acc_empty, (n_acc & 1u) ^ 1u, &gave_up)) { ok = false; break; }
            n_acc++;
            tmem_fence_after();
            bool add = false;
            for (int i = 0; ok && i < stages; i++, seq++) {
                const uint32_t st = seq % NW_STAGES, phase = (seq / NW_STAGES) & 1u;
                const uint64_t bd = smem_desc_sw128(b0 + st * NW_BSTAGE);
#pragma unroll
                for (uint32_t half = 0; half < 2; half++) {
                    if (!nw_wait_warp(&full[2 * st + half], phase, &gave_up)) { ok = false; break; }
                    tmem_fence_after();
                    if (elect_one()) {
                        mma_i8_ts(d, a0 + st * 96 + half * 48, bd + 4 * half, idesc, add);
                        mma_i8_ts(d, a0 + st * 96 + half * 48 + 8, bd + 4 * half + 2, idesc, true);
                        mma_commit(smem_u32(&empty[2 * st + half]));
                    }
                    __syncwarp();
                    add = true;
                }
            }
            if (ok && elect_one()) mma_commit(smem_u32(&acc_full));
            __syncwarp();
        }
    }
    if (!ok && lane == 0) atomicAdd(P.stalled, 1ull);
    __syncwarp();
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    if (gave_up) nw_drain(&drained, warp);
    if (warp == 16) tmem_free<512>(tm);
}

// Weights formed in segments: 64-bit integers that start at zero and become
// doubles when every segment has been added.
template <bool CONVERT>
__global__ void node_segments_kernel(double* w, int64_t group, int32_t nk, int64_t slot0, int64_t n) {
    const int64_t per = (int64_t)NODE_UNITS * nk;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * per; e += (int64_t)gridDim.x * blockDim.x) {
        // slots fastest, as they lie
        const int64_t s = slot0 + e % n;
        double* p = w + (s >> 3) * group + (e / n) * 8 + (s & 7);
        *p = CONVERT ? (double)*reinterpret_cast<const long long*>(p) : 0.0;
    }
}

// --------------------------------------------------------- a chunk's slots

// A job's nodes.  The weights of eight slots lie together (64 KB for 14 bins):
// W of slot s at w[(s / 8) group + (u nk + i) 8 + s % 8], u a genotype pair, i a
// node.  With the slots of a node together instead (rows of 4 MB at 1024
// samples) every load of a pass went to another page: 25 ms of passes against
// 19 ms.
struct NodeDev {
    const double* w;
    int64_t group;
    const double* t;      // the nodes' frequencies (at most 1/2)
    double scale;         // what a unit of the (integer) weights stands for
    int32_t nk;           // nodes per genotype pair: bins x NODE_J
    int32_t pad;
};

struct NodeArgs : SlotArgs {
    const NodeDev* nodes;      // per job
    double* partial;           // NODE_PART values a slot
    int* sites;                // NODE_UNITS values a slot: the pair's sites by genotype pair
    const LogTable* log_table;
};
constexpr int NODE_PART = UNIT_VALS * NODE_UNITS;   // a pass's sums

__global__ void node_init_kernel(NodeArgs A, int n_seg, int n, unsigned long long max_waves) {
    init_slot(A, n_seg, n, max_waves);
}

// ------------------------------------------------------------------- passes

// d - eps at a node: the shape's polynomial (stream64 of kg_pair.cuh).
template <int SH>
__device__ __forceinline__ double node_poly(const double* k, double t, double ty, double q) {
    if (SH == 0) return t * fma(fma(fma(k[3], t, k[2]), t, k[1]), t, k[0]);
    if (SH == 1 || SH == 2) return q * fma(fma(k[2], t, k[1]), t, k[0]);
    if (SH == 3) return q * fma(q, k[3], fma(t, k[2], fma(ty, k[1], k[0])));
    return q * fma(q, k[1], k[0]);
}

// One genotype pair's nodes for one slot, every fourth node from part on: the
// moments of its shape (SH) and the objective sum, sum W log d or (DIFF) sum W
// log(d / d_old); the terms of stream64 with weights.  MIRROR: the pair sees 1 -
// t.  out: gradient moments, Hessian moments, objective, sites.
template <int SH>
struct NodeShape {
    static constexpr int NG = SH == 0 ? 4 : SH == 3 ? 4 : SH == 4 ? 2 : 3;
    static constexpr int NH = SH == 0 ? 7 : SH == 3 ? 9 : SH == 4 ? 3 : 5;
    static constexpr int NK = SH == 0 || SH == 3 ? 4 : SH == 4 ? 2 : 3;      // coefficients
    static constexpr int K0 = SH == 0 ? 0 : SH == 1 ? 4 : SH == 2 ? 7 : SH == 3 ? 10 : 14;   // the first in PassCoef
};

template <int SH, bool MIRROR, bool DIFF>
__device__ __forceinline__ void node_sums(const NodeDev& N, const double* __restrict__ w, const double* __restrict__ st,
                                          int part, const LogTable& T,
                                          double (&g)[NodeShape<SH>::NG], double (&h)[NodeShape<SH>::NH], double& F) {
    constexpr int NG = NodeShape<SH>::NG, NH = NodeShape<SH>::NH, NK = NodeShape<SH>::NK, K0 = NodeShape<SH>::K0;
    const double EPS = 1e-8;
    double k[NK], ks[NK];
#pragma unroll
    for (int i = 0; i < NK; i++) {
        k[i] = st[(NS_COEF + K0 + i) * NS_LANES];
        ks[i] = DIFF ? st[(NS_STEP + K0 + i) * NS_LANES] : 0.0;
    }
    F = 0.0;
#pragma unroll
    for (int i = 0; i < NG; i++) g[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NH; i++) h[i] = 0.0;
    auto node = [&](double W, double tl) {
        const double tu = 1.0 - tl, t = MIRROR ? tu : tl, ty = MIRROR ? tl : tu, q = t * ty, t2 = t * t;
        const double d = node_poly<SH>(k, t, ty, q) + EPS;
        const double rd = recip<true>(d);
        if (SH == 0) {
            const double t3 = t2 * t, t4 = t2 * t2;
            const double u = t * rd, v = u * W;
            g[0] += v; g[1] = fma(v, t, g[1]); g[2] = fma(v, t2, g[2]); g[3] = fma(v, t3, g[3]);
            const double v2 = v * u, v4 = v2 * t4;
            h[0] += v2; h[1] = fma(v2, t, h[1]); h[2] = fma(v2, t2, h[2]); h[3] = fma(v2, t3, h[3]);
            h[4] += v4; h[5] = fma(v4, t, h[5]); h[6] = fma(v4, t2, h[6]);
        } else if (SH == 1 || SH == 2) {
            const double u = q * rd, v = u * W;
            g[0] += v; g[1] = fma(v, t, g[1]); g[2] = fma(v, t2, g[2]);
            const double v2 = v * u, v22 = v2 * t2;
            h[0] += v2; h[1] = fma(v2, t, h[1]); h[2] += v22; h[3] = fma(v22, t, h[3]);
            h[4] = fma(v22, t2, h[4]);
        } else if (SH == 3) {
            const double u = q * rd, v = u * W;
            g[0] += v; g[1] = fma(v, ty, g[1]); g[2] = fma(v, t, g[2]); g[3] = fma(v, q, g[3]);
            const double v2 = v * u, vy = v2 * ty, vq = v2 * q;
            h[0] += v2; h[1] += vy; h[2] = fma(v2, t, h[2]); h[3] += vq;
            h[4] = fma(vy, ty, h[4]); h[5] = fma(v2, t2, h[5]);
            h[6] = fma(vq, ty, h[6]); h[7] = fma(vq, t, h[7]); h[8] = fma(vq, q, h[8]);
        } else {
            const double u = q * rd, v = u * W;
            g[0] += v; g[1] = fma(v, q, g[1]);
            const double v2 = v * u, vq = v2 * q;
            h[0] += v2; h[1] += vq; h[2] = fma(vq, q, h[2]);
        }
        if (DIFF) F = fma(W, node_neg_log1m(node_poly<SH>(ks, t, ty, q) * rd, T), F);
        else F = fma(W, node_log(d, T), F);
    };
    static_assert(NODE_J % 8 == 0, "two nodes a step for each of four parts");
    constexpr int step = 4 * 8;
    const double* wp = w + part * 8;
    const double* __restrict__ tp = N.t + part;
    double W0 = wp[0], W1 = wp[step], t0 = __ldg(tp), t1 = __ldg(tp + 4);
    for (int i = 0; i < N.nk; i += 8) {
        const double a0 = W0, a1 = W1, b0 = t0, b1 = t1;
        if (i + 8 < N.nk) {   // the next two nodes' weights and frequencies in flight
            wp += 2 * step;
            tp += 8;
            W0 = wp[0];
            W1 = wp[step];
            t0 = __ldg(tp);
            t1 = __ldg(tp + 4);
        }
        node(a0, b0);
        node(a1, b1);
    }
}

template <int SH, bool MIRROR>
__device__ __forceinline__ void node_task(const NodeArgs& A, const NodeDev& N, int s, int u, int kind, int part,
                                          bool write, const LogTable& T) {
    constexpr int NG = NodeShape<SH>::NG, NH = NodeShape<SH>::NH;
    const double* w = N.w + (s >> 3) * N.group + (int64_t)u * N.nk * 8 + (s & 7);
    const double* st = A.state + slot_at(s, NS_VALS);
    double g[NG], h[NH], F;
    if (kind == NP_DIFF) node_sums<SH, MIRROR, true>(N, w, st, part, T, g, h, F);
    else node_sums<SH, MIRROR, false>(N, w, st, part, T, g, h, F);
    // the four parts, in a fixed order
    auto all = [](double v) {
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        return v + __shfl_xor_sync(0xffffffffu, v, 16);
    };
    double C = 0.0;
    const bool first = __any_sync(0xffffffffu, kind == NP_FIRST);
    if (first) {
        for (int i = part; i < N.nk; i += 4) C += w[i * 8];
        C = all(C);
    }
    const double scale = N.scale;
    double* P = A.partial + slot_at(s, NODE_PART) + u * UNIT_VALS * NS_LANES;
#pragma unroll
    for (int i = 0; i < NG; i++) {
        const double v = all(g[i]) * scale;
        if (write && part == (i & 3)) P[i * NS_LANES] = v;
    }
#pragma unroll
    for (int i = 0; i < NH; i++) {
        const double v = all(h[i]) * scale;
        if (write && part == ((NG + i) & 3)) P[(NG + i) * NS_LANES] = v;
    }
    const double f = all(F) * scale;
    if (write && part == 3) P[(UNIT_VALS - 1) * NS_LANES] = f;
    if (first && write && part == 0) A.sites[slot_at(s, NODE_UNITS) + u * NS_LANES] = __double2int_rn(C * scale);
}

// A warp per (8 slots of the pass list, genotype pair): lane l takes every
// fourth node from l / 8 on of slot l % 8, so a warp's load of weights is 256
// bytes in a row while its slots are neighbours; four lanes a slot keep a pass over few
// slots short (a lone lane's 112 nodes took 48 us), two shuffles a moment add
// them.  Genotype-pair-major, so an SM's warps run one shape's code at a time.
// Bound by the FP64 pipe's issue.
extern "C" __global__ void __launch_bounds__(128, 5) node_pass_kernel(NodeArgs A) {
    __shared__ LogTable T;
    if (A.clk->stop) return;   // a device loop past its last wave
    if (threadIdx.x == 0) atomicMin(&A.clk->start[1], global_ns());
    const int lane = threadIdx.x & 31;
    const PhaseEnd pe{&A.clk->end[1], lane == 0};
    const int n = A.ctl->n[A.par], groups = (n + 7) >> 3;
    const int64_t tasks = (int64_t)groups * NODE_UNITS;
    if ((int64_t)blockIdx.x >= tasks) return;
    for (int i = threadIdx.x; i < (int)(sizeof(LogTable) / 16); i += blockDim.x)
        reinterpret_cast<double2*>(&T)[i] = reinterpret_cast<const double2*>(A.log_table)[i];
    __syncthreads();
    const int part = lane >> 3;
    // consecutive tasks go to different SMs, so a short list spreads
    for (int64_t task = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; task < tasks;
         task += (int64_t)gridDim.x * (blockDim.x >> 5)) {
        const int u = (int)(task / groups), i = (int)(task - (int64_t)u * groups) * 8 + (lane & 7);
        const bool write = i < n;
        const int s = A.list_cur[write ? i : n - 1];
        const int jk = A.count[s].w, kind = jk & 7;
        const NodeDev N = A.nodes[jk >> 3];
        switch (u) {
        case 0: node_task<0, false>(A, N, s, u, kind, part, write, T); break;
        case 1: node_task<0, true>(A, N, s, u, kind, part, write, T); break;
        case 2: node_task<1, false>(A, N, s, u, kind, part, write, T); break;
        case 3: node_task<1, true>(A, N, s, u, kind, part, write, T); break;
        case 4: node_task<2, false>(A, N, s, u, kind, part, write, T); break;
        case 5: node_task<2, true>(A, N, s, u, kind, part, write, T); break;
        case 6: node_task<3, false>(A, N, s, u, kind, part, write, T); break;
        case 7: node_task<3, true>(A, N, s, u, kind, part, write, T); break;
        default: node_task<4, false>(A, N, s, u, kind, part, write, T); break;
        }
    }
}

// --------------------------------------------------------------- the SQP step

// S = sum L r and the upper triangle T = sum L L' r^2 from the moments (rebuild
// of kg_pair.cuh, its indices known at compile time).
__device__ __forceinline__ void rebuild_upper(const double (&m)[NMOM], double (&S)[9], double (&T)[QP_Q]) {
    constexpr int e[9] = {1, 2, 2, 3, 2, 3, 2, 3, 4};
#pragma unroll
    for (int i = 0; i < 9; i++) {
        S[i] = m[e[i] - 1];
#pragma unroll
        for (int j = i; j < 9; j++) T[upper_at(i, j)] = m[4 + e[i] + e[j] - 2];
    }
    constexpr int cb[4] = {1, 2, 1, 2}, pb[4] = {0, 1, 1, 2}, i1[4] = {2, 3, 7, 8}, i2[4] = {4, 5, 7, 8};
    constexpr int ic[4] = {1, 3, 5, 8}, hc[4][4] = {{0, 1, 2, 3}, {1, 4, 3, 6}, {2, 3, 5, 7}, {3, 6, 7, 8}};
    constexpr int id[3] = {6, 7, 8}, cd[3] = {2, 1, 4}, pd[3] = {0, 0, 1};
#pragma unroll
    for (int a = 0; a < 4; a++) {
        S[i1[a]] += cb[a] * m[11 + pb[a]];
        S[i2[a]] += cb[a] * m[19 + pb[a]];
        S[ic[a]] += m[27 + a];
#pragma unroll
        for (int b = a; b < 4; b++) {
            T[upper_at(i1[a], i1[b])] += (double)(cb[a] * cb[b]) * m[14 + pb[a] + pb[b]];
            T[upper_at(i2[a], i2[b])] += (double)(cb[a] * cb[b]) * m[22 + pb[a] + pb[b]];
            T[upper_at(ic[a], ic[b])] += m[31 + hc[a][b]];
        }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        S[id[a]] += cd[a] * m[40 + pd[a]];
#pragma unroll
        for (int b = a; b < 3; b++) T[upper_at(id[a], id[b])] += (double)(cd[a] * cd[b]) * m[42 + pd[a] + pd[b]];
    }
}

// A pass's sums over nodes: two genotype pairs a shape, het-het one.
struct NodeSums {
    static constexpr bool FP32 = false, COEF = true;
    const NodeArgs& A;
    static __device__ double none() { return CUDART_NAN; }
    __device__ __forceinline__ void load(int s, int kind, double* st, double& obj, double (&g)[9], double (&T)[QP_Q],
                                         double& nsites) const {
        double m[NMOM];
        const double* P = A.partial + slot_at(s, NODE_PART);
        const int* sites = A.sites + slot_at(s, NODE_UNITS);
        constexpr int SD = NS_LANES;
        obj = 0.0;
#pragma unroll
        for (int u = 0; u < NODE_UNITS; u++) {
            const int sh = u >> 1, go = sh == 0 ? 0 : sh == 1 ? 11 : sh == 2 ? 19 : sh == 3 ? 27 : 40;
            const int nv = sh == 0 ? 11 : sh == 3 ? 13 : sh == 4 ? 5 : 8;
#pragma unroll
            for (int v = 0; v < 13; v++)
                if (v < nv) {
                    const double p = P[(u * UNIT_VALS + v) * SD];
                    m[go + v] = (u & 1) ? m[go + v] + p : p;
                }
            obj += P[(u * UNIT_VALS + UNIT_VALS - 1) * SD];
        }
        if (kind == NP_FIRST) {
            int64_t c = 0;
            for (int u = 0; u < NODE_UNITS; u++) c += sites[u * SD];
            nsites = (double)c;
            st[NS_N * SD] = nsites;
        } else {
            nsites = st[NS_N * SD];
        }
        rebuild_upper(m, g, T);
    }
    __device__ __forceinline__ void count(int s, int job, int gh, int, double, bool ill, unsigned long long* sum) const {
        const int* sites = A.sites + slot_at(s, NODE_UNITS);
        unsigned long long evals = 0;
#pragma unroll
        for (int sh = 0; sh < 5; sh++) {
            int c = sites[2 * sh * NS_LANES];
            if (sh < 4) c += sites[(2 * sh + 1) * NS_LANES];
            atomicAdd(&sum[7 + sh], (unsigned long long)c);
            evals += (unsigned long long)((sh == 4 ? 1 : 2) * flops_fp64(sh));
        }
        if (ill) atomicAdd(&sum[5], 1ull);   // the pairs that FP32 passes would hand to FP64
        atomicAdd(&sum[6], evals * (unsigned long long)A.nodes[job].nk * (unsigned long long)gh);
    }
};

extern "C" __global__ void __launch_bounds__(NA_THREADS) node_advance_kernel(NodeArgs A, int in_loop,
                                                                            cudaGraphConditionalHandle loop) {
    advance_wave(A, NodeSums{A}, in_loop, loop);
}

// ---------------------------------------------------------------------- CLS

// The CLS estimator of a pair (cls_finish of kg_wave.cu, src/coefficients.rs:
// 218-268), a thread per pair: the pair's summed likelihood rows are cubic and
// quartic in the frequency, so its nodes give them exactly; c = rows / (-M),
// the simplex QP on the cohort's Q (two-variable for a self pair), the Brier
// score and the condition estimate.
extern "C" __global__ void __launch_bounds__(NA_THREADS) node_cls_kernel(NodeArgs A, int n_seg, int n) {
    __shared__ double in[QP_IN * NA_THREADS];
    __shared__ unsigned long long sum[7];
    if (threadIdx.x < 7) sum[threadIdx.x] = 0ull;
    __syncwarp();
    double* my = in + threadIdx.x;
    for (int s = blockIdx.x * NA_THREADS + threadIdx.x; s < n; s += gridDim.x * NA_THREADS) {
        const PairSeg sg = seg_of(A.seg, n_seg, s);
        const CohortDev& co = A.cohorts[sg.job];
        const NodeDev N = A.nodes[sg.job];
        int64_t x, y;
        const int64_t row = job_pair(co, sg.idx0 + (s - sg.slot0), x, y);
        // sums of the shapes' monomials: A t^1..4, B w t^0..2, C w {1, ty, t, w}, D w {1, w}
        double m[16], sites[5];
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = 0.0;
#pragma unroll
        for (int k = 0; k < 5; k++) sites[k] = 0.0;
        for (int i = 0; i < N.nk; i++) {
            const double* w = N.w + (s >> 3) * N.group + i * 8 + (s & 7);
            const int un = N.nk * 8;
            const double t = __ldg(N.t + i), u = 1.0 - t, q = t * u, t2 = t * t, u2 = u * u;
            const double W[9] = {w[0], w[un], w[2 * un], w[3 * un], w[4 * un], w[5 * un], w[6 * un], w[7 * un], w[8 * un]};
            m[0] = fma(W[0], t, fma(W[1], u, m[0]));
            m[1] = fma(W[0], t2, fma(W[1], u2, m[1]));
            m[2] = fma(W[0], t2 * t, fma(W[1], u2 * u, m[2]));
            m[3] = fma(W[0], t2 * t2, fma(W[1], u2 * u2, m[3]));
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const double v0 = W[2 + 2 * b] * q, v1 = W[3 + 2 * b] * q;
                m[4 + 3 * b] += v0 + v1;
                m[5 + 3 * b] = fma(v0, t, fma(v1, u, m[5 + 3 * b]));
                m[6 + 3 * b] = fma(v0, t2, fma(v1, u2, m[6 + 3 * b]));
            }
            const double c0 = W[6] * q, c1 = W[7] * q, d0 = W[8] * q;
            m[10] += c0 + c1;
            m[11] = fma(c0, u, fma(c1, t, m[11]));
            m[12] = fma(c0, t, fma(c1, u, m[12]));
            m[13] = fma(c0 + c1, q, m[13]);
            m[14] += d0;
            m[15] = fma(d0, q, m[15]);
#pragma unroll
            for (int k = 0; k < 4; k++) sites[k] += W[2 * k] + W[2 * k + 1];
            sites[4] += W[8];
        }
        double S[9] = {m[0], m[1] + m[10], m[1] + m[4], m[2] + 2.0 * m[5] + m[11], m[1] + m[7],
                       m[2] + 2.0 * m[8] + m[12], m[1] + 2.0 * m[14], m[2] + m[5] + m[8] + m[14],
                       m[3] + 2.0 * (m[6] + m[9]) + m[13] + 4.0 * m[15]};
        Tune tq = A.tune;
        tq.qp_max_iter = co.max_iter > (uint64_t)INT_MAX ? INT_MAX : (int)co.max_iter;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            double v = S[k] * N.scale;
            if (co.cls_cmulti) v += co.cls_cmulti[row * 9 + k];   // its tri- and tetra-allelic rows
            my[(QP_Q + k) * NA_THREADS] = v / -co.cls_m;
#pragma unroll
            for (int j = k; j < 9; j++) my[upper_at(k, j) * NA_THREADS] = co.cls_q[k * 9 + j];
        }
        auto Q = [my](int i2, int j2) { return my[(i2 <= j2 ? upper_at(i2, j2) : upper_at(j2, i2)) * NA_THREADS]; };
        double d[9];
        int iters;
        if (x == y) {
            double e0 = 0.0, e6 = 0.0;
            iters = qp_simplex2(Q(0, 0), Q(0, 6), Q(0, 6), Q(6, 6), my[QP_Q * NA_THREADS], my[(QP_Q + 6) * NA_THREADS],
                                0.5, 0.5, tq, e0, e6);
#pragma unroll
            for (int k = 0; k < 9; k++) d[k] = k == 0 ? e0 : k == 6 ? e6 : 0.0;
        } else {
#pragma unroll
            for (int k = 0; k < 9; k++) d[k] = 1.0 / 9.0;
            iters = qp_simplex_thread<true>([my](int v) { return my[v * NA_THREADS]; }, tq, d);
        }
        double g[9], quad = 0.0, lin = 0.0;
#pragma unroll
        for (int r = 0; r < 9; r++) {
            double qd = 0.0;
#pragma unroll
            for (int j = 0; j < 9; j++) qd = fma(Q(r, j), d[j], qd);
            quad = fma(d[r], qd, quad);
            const double c = my[(QP_Q + r) * NA_THREADS];
            lin = fma(c, d[r], lin);
            g[r] = qd + c;
        }
        const double cond = condition_thread([my](int k) { return my[k * NA_THREADS]; }, d, g, tq.sqp_conv_tol);
        node_write_row(co.out + row, x, y, d, (quad + 2.0 * lin) + 1.0, (uint64_t)iters, cond);
        unsigned long long all = 0;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const unsigned long long c = (unsigned long long)__double2ll_rn(sites[k] * N.scale);
            all += c;
            atomicAdd(&sum[k], c);
        }
        atomicAdd(&sum[5], all);
        if ((uint64_t)iters >= co.max_iter) atomicAdd(&sum[6], 1ull);
    }
    __syncwarp();
    RunCounters* C = A.counters;
    if (threadIdx.x < 5) atomicAdd(&C->shape_sites[threadIdx.x], sum[threadIdx.x]);
    if (threadIdx.x == 5) {
        atomicAdd(&C->pair_sites, sum[5]);
        atomicAdd(&C->work_units, sum[5]);
    }
    if (threadIdx.x == 6 && sum[6]) atomicAdd(&C->nonconverged, sum[6]);
}

// ------------------------------------------------------------------- host

// The waves of a chunk as one graph launch (a WHILE node over two waves), kept
// between calls: it depends on the workspace's buffers and on what they are laid
// out for (the most slots and jobs so far), not on the cohort.  Capturing
// and instantiating it takes 0.25 ms: with the layout of the call itself, 64 x
// 10,000 sites took 1.01 ms again and again, and 1.26 ms among other sizes.
struct NodeEngine {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    std::vector<void*> key;
    uint64_t key_iterations = 0;
    int key_dev = -1;
    cudaStream_t key_st = nullptr;
    int64_t stride = 0;   // slots that the layout holds
    int jobs = 0;         // jobs that the tables hold
    DevBuf log_table;
    NodeArgs args[2]{};
    int pass_blocks = 0, advance_blocks = 0, cls_blocks = 0;
    void drop() {
        if (x) cudaGraphExecDestroy(x);
        if (g) cudaGraphDestroy(g);
        x = nullptr;
        g = nullptr;
        key.clear();
    }
    ~NodeEngine() {
        drop();
        for (auto& e : ev)
            if (e) cudaEventDestroy(e);
    }
    void wave(int par, int in_loop, cudaGraphConditionalHandle h, cudaStream_t st) const {
        node_pass_kernel<<<pass_blocks, 128, 0, st>>>(args[par]);
        node_advance_kernel<<<advance_blocks, NA_THREADS, 0, st>>>(args[par], in_loop, h);
    }
};

int run_nodes(const std::vector<PairJob>& jobs, const RunConfig& cfg, Workspace& ws, cudaStream_t st,
              kg_run_stats& stats, std::string& err) {
    if (!ws.nodes) ws.nodes = std::make_shared<NodeEngine>();
    NodeEngine& E = *ws.nodes;
    int dev = 0;
    KG_NODE_TRY(cudaGetDevice(&dev));
    if (ws.sm_count == 0) KG_NODE_TRY(cudaDeviceGetAttribute(&ws.sm_count, cudaDevAttrMultiProcessorCount, dev));
    const int n_jobs = (int)jobs.size();
    constexpr int J = NODE_J;
    const bool cls = jobs[0].method == ESTIMATOR_CLS;
    std::vector<CohortDev> table((size_t)n_jobs);
    int64_t total = 0;
    int nk_max = 0;
    uint64_t max_iter = cfg.iterations;
    for (int i = 0; i < n_jobs; i++) {
        table[i] = make_cohort_dev(jobs[i], cfg.iterations);
        table[i].pair_begin = total;
        total += jobs[i].count < 0 ? table[i].n_pairs : jobs[i].count;
        nk_max = std::max(nk_max, jobs[i].panel->nd_n * J);
        max_iter = std::max<uint64_t>(max_iter, table[i].max_iter);
    }
    // pairs in flight: all of them up to 2^20, or what half the free memory
    // (with what the workspace holds already) takes
    const size_t slot_bytes = sizeof(double) * (NODE_UNITS * UNIT_VALS + NS_VALS + 2) + sizeof(int4) +
                              sizeof(int) * (2 + NODE_UNITS);
    const size_t per_slot = sizeof(double) * NODE_UNITS * (size_t)nk_max + slot_bytes;
    int64_t cap = std::min<int64_t>(total, cfg.slots > 0 ? cfg.slots : (int64_t)1 << 20);
    const size_t held = ws.scratch.bytes + ws.slots.bytes;
    if ((size_t)cap * per_slot > held) {
        size_t fr = 0, tot = 0;
        KG_NODE_TRY(cudaMemGetInfo(&fr, &tot));
        cap = std::max<int64_t>(1, std::min<int64_t>(cap, (int64_t)((fr + held) / 2 / per_slot)));
    }
    const int64_t group = (int64_t)NODE_UNITS * nk_max * 8;
    KG_NODE_TRY((cudaError_t)ws.scratch.reserve(sizeof(double) * (size_t)group * ((cap + 31) / 32 * 4)));
    // the layout of the largest call so far, not rounded up
    int64_t stride = (cap + 31) / 32 * 32;
    if (stride < E.stride && slot_bytes * (size_t)E.stride <= ws.slots.bytes) stride = E.stride;
    KG_NODE_TRY((cudaError_t)ws.slots.reserve(slot_bytes * (size_t)stride));
    // (the tables are copied whole: no more than 256 jobs are kept for fewer)
    int job_cap = n_jobs;
    if (job_cap < E.jobs && E.jobs <= 256) job_cap = E.jobs;
    // control words, one buffer: {control, clock, run counters}
    const size_t off_clk = sizeof(SlotCtl), off_run = off_clk + sizeof(WaveClock);
    const size_t ctl_bytes = off_run + sizeof(RunCounters);
    KG_NODE_TRY((cudaError_t)ws.node_counts.reserve(ctl_bytes));
    const size_t off_nodes = sizeof(CohortDev) * job_cap, off_seg = off_nodes + sizeof(NodeDev) * job_cap;
    const size_t blob = off_seg + sizeof(PairSeg) * job_cap;
    KG_NODE_TRY((cudaError_t)ws.node_table.reserve(blob));
    KG_NODE_TRY((cudaError_t)ws.host.reserve(blob + sizeof(WaveClock) + sizeof(RunCounters)));
    char* counts = ws.node_counts.as<char>();
    char* dtab = ws.node_table.as<char>();
    char* htab = ws.host.as<char>();
    WaveClock* h_clk = reinterpret_cast<WaveClock*>(htab + blob);
    RunCounters* h_run = reinterpret_cast<RunCounters*>(h_clk + 1);
    const unsigned long long bound = wave_bound(max_iter, 1);   // without a caller's wave limit
    const char* hw = std::getenv("KESTREL_HOST_WAVES");
    const bool host_waves = hw && hw[0] == '1';
    const std::vector<void*> key{ws.slots.p, ws.node_counts.p, ws.node_table.p};
    if (E.key != key || E.stride != stride || E.jobs != job_cap || E.key_iterations != cfg.iterations || E.key_dev != dev || E.key_st != st) {
        E.drop();
        if (!E.log_table.p || E.key_dev != dev) {
            LogTable T;
            fill_log_table(T);
            E.log_table.release();
            KG_NODE_TRY((cudaError_t)E.log_table.reserve(sizeof(T)));
            KG_NODE_TRY(cudaMemcpy(E.log_table.p, &T, sizeof(T), cudaMemcpyHostToDevice));
        }
        NodeArgs A{};
        A.cohorts = reinterpret_cast<CohortDev*>(dtab);
        A.nodes = reinterpret_cast<NodeDev*>(dtab + off_nodes);
        A.seg = reinterpret_cast<PairSeg*>(dtab + off_seg);
        A.state = ws.slots.as<double>();
        A.partial = A.state + (size_t)(NS_VALS + 2) * stride;
        A.count = reinterpret_cast<int4*>(A.partial + (size_t)NODE_UNITS * UNIT_VALS * stride);
        A.sites = reinterpret_cast<int*>(A.count + stride);
        int* lists = A.sites + NODE_UNITS * stride;
        A.ctl = reinterpret_cast<SlotCtl*>(counts);
        A.clk = reinterpret_cast<WaveClock*>(counts + off_clk);
        A.counters = reinterpret_cast<RunCounters*>(counts + off_run);
        A.log_table = E.log_table.as<LogTable>();
        A.tune = make_tune(cfg.iterations);
        for (int par = 0; par < 2; par++) {
            E.args[par] = A;
            E.args[par].par = par;
            E.args[par].list_cur = lists + (par ? stride : 0);
            E.args[par].list_next = lists + (par ? 0 : stride);
        }
        int occ = 0;
        KG_NODE_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, node_pass_kernel, 128, 0));
        E.pass_blocks = ws.sm_count * std::max(1, occ);
        KG_NODE_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, node_advance_kernel, NA_THREADS, 0));
        E.advance_blocks = ws.sm_count * std::max(1, occ);
        KG_NODE_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, node_cls_kernel, NA_THREADS, 0));
        E.cls_blocks = ws.sm_count * std::max(1, occ);
        KG_NODE_TRY(cudaFuncSetAttribute(node_weights_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, NW_SMEM));
        KG_NODE_TRY(cudaFuncSetAttribute(node_weights_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, NW_SMEM));
        for (auto& e : E.ev)
            if (!e) KG_NODE_TRY(cudaEventCreate(&e));
        KG_NODE_TRY(wave_loop_graph(
            st, [&](int par, int in_loop, cudaGraphConditionalHandle h) { E.wave(par, in_loop, h, st); }, &E.g, &E.x));
        E.key = key;
        E.stride = stride;
        E.jobs = job_cap;
        E.key_iterations = cfg.iterations;
        E.key_dev = dev;
        E.key_st = st;
    }
    std::memcpy(htab, table.data(), sizeof(CohortDev) * n_jobs);
    KG_NODE_TRY(cudaMemsetAsync(counts, 0, ctl_bytes, st));
    NodeDev* h_nodes = reinterpret_cast<NodeDev*>(htab + off_nodes);
    PairSeg* h_seg = reinterpret_cast<PairSeg*>(htab + off_seg);
    RunCounters* d_run = reinterpret_cast<RunCounters*>(counts + off_run);
    const WaveClock* d_clk = reinterpret_cast<const WaveClock*>(counts + off_clk);
    int job = 0;
    int64_t at = jobs[0].first;   // the job's next pair, y-major
    bool limit_hit = false;
    double build_ms = 0.0;
    uint64_t waves = 0, launches = 0;
    while (job < n_jobs && !limit_hit) {
        // the next chunk of pairs
        int n_seg = 0;
        int64_t n = 0;
        while (job < n_jobs && n < cap) {
            const PairJob& jb = jobs[job];
            const int64_t end = jb.count < 0 ? table[job].n_pairs : jb.first + jb.count;
            const int64_t take = std::min<int64_t>(end - at, cap - n);
            if (take > 0) {
                const Cohort& c = *jb.panel;
                h_seg[n_seg] = PairSeg{at, (int32_t)n, (int32_t)take, job, 0};
                NodeDev& nd = h_nodes[job];
                nd.w = ws.scratch.as<double>();
                nd.group = group;
                nd.nk = c.nd_n * J;
                nd.t = c.nd_t.as<double>();
                nd.scale = std::ldexp(1.0, -(8 * NODE_L - 2));
                n_seg++;
                n += take;
                at += take;
            }
            if (at >= end) {
                job++;
                at = job < n_jobs ? jobs[job].first : 0;
            }
        }
        KG_NODE_TRY(cudaMemcpyAsync(dtab, htab, blob, cudaMemcpyHostToDevice, st));
        KG_NODE_TRY(cudaEventRecord(E.ev[0], st));
        for (int k = 0; k < n_seg; k++) {
            const PairSeg& g = h_seg[k];
            const Cohort& c = *jobs[g.job].panel;
            NodeProduct P;
            P.rect = jobs[g.job].kind == COHORT_RECT ? 1 : 0;
            P.planes = c.nd_planes.as<uint2>();
            P.planes_b = P.rect ? jobs[g.job].query->planes.as<uint2>() : P.planes;
            P.dig = c.nd_dig.as<int8_t>();
            P.bin = reinterpret_cast<const NodeBin*>(c.nd_bins.as<int>() + NODE_MAX_BINS);
            P.mp = c.nd_mp;
            P.words = c.nd_mp / 32;
            P.n_samples = (int32_t)c.n_samples;
            P.bins = c.nd_n;
            P.idx0 = g.idx0;
            P.idx1 = g.idx0 + g.n;
            P.slot0 = g.slot0;
            int64_t x, y0, y1;
            if (P.rect) {
                const int64_t nb = (P.n_samples + 127) >> 7;
                y0 = P.idx0 / P.n_samples;
                y1 = (P.idx1 - 1) / P.n_samples;
                P.first_unit = y0 * nb;
                P.n_yx = (y1 + 1) * nb - P.first_unit;
            } else {
                pair_of(P.idx0, x, y0);
                pair_of(P.idx1 - 1, x, y1);
                P.first_unit = yx_before(y0);
                P.n_yx = yx_before(y1 + 1) - P.first_unit;
            }
            P.w = ws.scratch.as<double>();
            P.group = group;
            P.stalled = &d_run->stalled_waits;
            P.seg = (int32_t)node_seg_stages(c.nd_mp / NODE_STAGE, P.n_yx, ws.sm_count);
            P.segs = node_segments(c.nd_mp / NODE_STAGE, P.seg);
            const int grid = (int)std::min<int64_t>(ws.sm_count, P.n_yx * (P.bins + P.segs - 1));
            const int sgrid = (int)std::min<int64_t>(((int64_t)g.n * NODE_UNITS * c.nd_n * J + 255) / 256, ws.sm_count * 8);
            if (P.segs == 1) {
                node_weights_kernel<false><<<grid, NW_THREADS, NW_SMEM, st>>>(P);
            } else {
                node_segments_kernel<false><<<sgrid, 256, 0, st>>>(P.w, group, c.nd_n * J, g.slot0, g.n);
                node_weights_kernel<true><<<grid, NW_THREADS, NW_SMEM, st>>>(P);
                node_segments_kernel<true><<<sgrid, 256, 0, st>>>(P.w, group, c.nd_n * J, g.slot0, g.n);
                launches += 2;
            }
        }
        launches += n_seg + 1;
        KG_NODE_TRY(cudaGetLastError());
        KG_NODE_TRY(cudaEventRecord(E.ev[1], st));
        if (cls) {
            const int grid = (int)std::min<int64_t>(E.cls_blocks, (n + NA_THREADS - 1) / NA_THREADS);
            node_cls_kernel<<<grid, NA_THREADS, 0, st>>>(E.args[0], n_seg, (int)n);
        } else {
            node_init_kernel<<<(int)((n + 127) / 128), 128, 0, st>>>(E.args[0], n_seg, (int)n,
                                                                     cfg.max_waves ? cfg.max_waves - waves : bound);
            if (host_waves) {
                for (uint64_t k = 0;; k++) {
                    E.wave((int)(k & 1), 0, cudaGraphConditionalHandle{}, st);
                    KG_NODE_TRY(cudaMemcpyAsync(h_clk, d_clk, sizeof(WaveClock), cudaMemcpyDeviceToHost, st));
                    KG_NODE_TRY(cudaStreamSynchronize(st));
                    launches += 2;
                    if (h_clk->stop) break;
                }
            } else {
                KG_NODE_TRY(cudaGraphLaunch(E.x, st));
            }
        }
        KG_NODE_TRY(cudaGetLastError());
        KG_NODE_TRY(cudaMemcpyAsync(h_clk, d_clk, sizeof(WaveClock) + sizeof(RunCounters), cudaMemcpyDeviceToHost, st));
        KG_NODE_TRY(cudaStreamSynchronize(st));
        if (!host_waves && !cls) launches += 4 * h_clk->iters;
        float ms = 0.f;
        KG_NODE_TRY(cudaEventElapsedTime(&ms, E.ev[0], E.ev[1]));
        build_ms += ms;
        waves += cls ? 1 : h_clk->waves;
        limit_hit = !cls && (h_clk->limit_hit != 0 || (cfg.max_waves && waves >= cfg.max_waves && job < n_jobs));
        if (h_run->stalled_waits) {
            err = "a device wait of the node weights ran out of its limit";
            return KG_ETIMEOUT;
        }
    }
    const RunCounters& rc = *h_run;
    stats.gh_passes = cls ? (uint64_t)total : rc.gh_passes;
    stats.obj_passes = stats.gh_passes;
    stats.fp64_passes = cls ? 0 : rc.gh_passes;   // every pass over nodes is FP64
    stats.fp64_pairs = rc.fp64_pairs;
    stats.pair_sites = rc.pair_sites;
    stats.work_units = rc.work_units;
    stats.launches = launches;
    stats.flops_fp64 = rc.flops_fp64;
    for (int k = 0; k < 5; k++) stats.shape_sites[k] = rc.shape_sites[k];
    stats.nonconverged = rc.nonconverged;
    stats.waves = waves;
    stats.slots = (uint64_t)cap;
    stats.admit_ms = build_ms;
    stats.pass_ms = (double)h_clk->acc[1] * 1e-6;
    stats.solve_ms = (double)h_clk->acc[2] * 1e-6;
    stats.pair_kernel_ms = stats.admit_ms + stats.pass_ms + stats.solve_ms;
    if (limit_hit) {
        err = "the wave loop reached its wave limit";
        return KG_ETIMEOUT;
    }
    if (rc.nosite_pairs) {
        err = "a pair has no jointly observed segregating site (its row is NaN)";
        return KG_ENOSITES;
    }
    return KG_OK;
}

}  // namespace kg
