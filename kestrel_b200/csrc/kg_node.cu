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
// CLS needs sum t^k, k <= 4, only: one interval [0, 1/2] is exact with five
// nodes, so its bins are equal runs of sites (to spread a small cohort over the
// SMs), all on that interval.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "kg_bulk.cuh"
#include "kg_engine.h"
#include "kg_node.h"
#include "kg_pair.cuh"
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

// A node's table entry at frequency t: t, 1 - t, t (1 - t), t^2 .. t^6.
constexpr int NODE_VALS = 8;

// A double bin: its first site (a multiple of NODE_STAGE), its stages.
struct NodeBin {
    int32_t start, stages;
};

int node_bins(bool cls, int64_t n_kept, int64_t n_samples, double t_min) {
    if (n_kept <= 0 || n_samples <= 0) return 0;
    if (cls) {
        if (!(t_min >= 0.0)) return 0;
        const int64_t by_work = (n_kept + 1023) / 1024, by_sms = 296 / n_samples + 1;
        return (int)std::max<int64_t>(1, std::min<int64_t>({by_work, by_sms, 16}));
    }
    if (!(t_min > 0.0) || t_min > 0.5) return 0;
    const double need = std::ceil(std::log(0.5 / t_min) / std::log(NODE_RATIO));
    if (!(need <= (double)NODE_MAX_BINS)) return 0;
    const int bins = std::max(1, (int)need);
    // below ten sites per node the lists win: 64 samples x 10,000 sites (14
    // bins, 1,008 nodes a pair) took 2.73 ms on lists and 3.28 ms on nodes, 201
    // x 33,333 (2,016 nodes of 24 bins) 41.6 against 6.6 ms
    if (n_kept < (int64_t)10 * NODE_UNITS * NODE_J * bins) return 0;
    return bins;
}

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
// the scatter's cursors) and the node points.
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
    for (int e = threadIdx.x; e < 2 * G.bins * J; e += blockDim.x) {
        const bool mirror = e >= G.bins * J;
        const int i = mirror ? e - G.bins * J : e, k = i / J, j = i - k * J;
        double lo, hi;
        bin_interval(G, k, lo, hi);
        const double tl = 0.5 * (lo + hi) - 0.5 * (hi - lo) * cospi((2 * j + 1) / (2.0 * J));
        const double x = mirror ? 1.0 - tl : tl, y = mirror ? tl : 1.0 - tl, x2 = x * x;
        double* o = t + (int64_t)e * NODE_VALS;
        o[0] = x;
        o[1] = y;
        o[2] = x * y;
        o[3] = x2;
        o[4] = x2 * x;
        o[5] = x2 * x2;
        o[6] = x2 * x2 * x;
        o[7] = x2 * x2 * x2;
    }
}

// Kept sites to their places: place[pos] = raw site, bit 31 set where the
// genotypes are exchanged (the order within a bin does not matter: the sums
// are integers); and the digits of the site's basis values.
__global__ void node_scatter_kernel(NodeGrid G, const double* __restrict__ p64, const int32_t* __restrict__ site_of,
                                    int* __restrict__ cursor, uint32_t* __restrict__ place, int8_t* __restrict__ dig,
                                    int64_t mp) {
    constexpr int J = NODE_J, L = NODE_L;
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= G.n_kept) return;
    const double p = p64[freq_index(s)];
    const int k = bin_of(G, s, p);
    const int pos = atomicAdd(&cursor[k], 1);
    const double t = fmin(p, 1.0 - p);
    place[pos] = (uint32_t)site_of[s] | (p > 0.5 ? 0x80000000u : 0u);
    double lo, hi;
    bin_interval(G, k, lo, hi);
    const double z = (t - 0.5 * (lo + hi)) / (0.5 * (hi - lo));
    // barycentric basis on the first-kind Chebyshev points z_j = -cos((2j+1) pi / 2J)
    double b[J], sum = 0.0;
    int hit = -1;
#pragma unroll
    for (int j = 0; j < J; j++) {
        const double dz = z + cospi((2 * j + 1) / (2.0 * J));
        const double w = ((j & 1) ? -1.0 : 1.0) * sinpi((2 * j + 1) / (2.0 * J));
        if (dz == 0.0) hit = j;
        b[j] = w / dz;
        sum += b[j];
    }
    const int64_t byte = (pos & ~31) | ((pos & 7) << 2) | ((pos >> 3) & 3);
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
// placed sites a time; the sample's codes are read through L1.
__global__ void node_pack_kernel(const uint8_t* __restrict__ raw, int64_t stride, const uint32_t* __restrict__ place,
                                 int64_t words, uint2* __restrict__ planes) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint8_t* row = raw + (int64_t)blockIdx.x * stride;
    uint2* out = planes + (int64_t)blockIdx.x * words;
    for (int64_t k = (int64_t)blockIdx.y * nw + w; k < words; k += (int64_t)gridDim.y * nw) {
        const uint32_t e = place[k * 32 + lane];
        unsigned c = 3u;
        if (e != 0xFFFFFFFFu) {
            c = row[e & 0x7FFFFFFFu];
            if ((e >> 31) && c < 3u) c = 2u - c;
        }
        const unsigned lo = __ballot_sync(0xffffffffu, c & 1u), hi = __ballot_sync(0xffffffffu, (c >> 1) & 1u);
        if (lane == 0) out[k] = make_uint2(lo, hi);
    }
}

int prepare_nodes(Cohort& c, const uint8_t* codes, int64_t stride, int bins, double t_min, cudaStream_t st,
                  std::string& err) {
    const int64_t mp = ((c.n_kept + NODE_STAGE - 1) / NODE_STAGE + bins) * NODE_STAGE;
    NodeGrid G;
    G.bins = bins;
    G.by_index = c.cls ? 1 : 0;
    // the bins end at the smallest frequency (a hair below, so that it lies inside)
    G.q = c.cls ? 1.0
                : std::min(1.0 / NODE_RATIO, std::pow(std::min(1.0, 2.0 * t_min) * (1.0 - 1e-12), 1.0 / bins));
    G.inv_log_q = c.cls ? 0.0 : 1.0 / std::log(G.q);
    G.n_kept = c.n_kept;
    const size_t head = sizeof(int) * NODE_MAX_BINS + sizeof(NodeBin) * NODE_MAX_BINS;
    KG_NODE_TRY((cudaError_t)c.nd_bins.reserve(head));
    KG_NODE_TRY((cudaError_t)c.nd_t.reserve(sizeof(double) * 2 * NODE_VALS * bins * NODE_J));
    KG_NODE_TRY((cudaError_t)c.nd_place.reserve(sizeof(uint32_t) * mp));
    KG_NODE_TRY((cudaError_t)c.nd_dig.reserve((size_t)32 * mp));
    KG_NODE_TRY((cudaError_t)c.nd_planes.reserve(sizeof(uint2) * (mp / 32) * c.n_samples));
    int* hist = c.nd_bins.as<int>();
    NodeBin* bin = reinterpret_cast<NodeBin*>(hist + NODE_MAX_BINS);
    KG_NODE_TRY(cudaMemsetAsync(hist, 0, sizeof(int) * NODE_MAX_BINS, st));
    KG_NODE_TRY(cudaMemsetAsync(c.nd_place.p, 0xFF, sizeof(uint32_t) * mp, st));
    KG_NODE_TRY(cudaMemsetAsync(c.nd_dig.p, 0, (size_t)32 * mp, st));
    const int grid = (int)((c.n_kept + 255) / 256);
    node_hist_kernel<<<grid, 256, 0, st>>>(G, c.p64.as<double>(), hist);
    node_layout_kernel<<<1, 256, 0, st>>>(G, hist, bin, c.nd_t.as<double>());
    node_scatter_kernel<<<grid, 256, 0, st>>>(G, c.p64.as<double>(), c.site_of.as<int32_t>(), hist,
                                              c.nd_place.as<uint32_t>(), c.nd_dig.as<int8_t>(), mp);
    // enough blocks to fill the SMs, few enough that a sample's row is read by few
    const int64_t words = mp / 32;
    const int parts = (int)std::max<int64_t>(1, std::min<int64_t>((words + 63) / 64, 1184 / c.n_samples + 1));
    node_pack_kernel<<<dim3((unsigned)c.n_samples, parts), 256, 0, st>>>(codes, stride, c.nd_place.as<uint32_t>(),
                                                                         words, c.nd_planes.as<uint2>());
    KG_NODE_TRY(cudaGetLastError());
    c.nd_n = bins;
    c.nd_mp = mp;
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
// Per stage of 128 sites: 12 instructions of 48 cycles; two stages, so the
// expansion of one runs under the products of the other.
constexpr int NW_THREADS = 416;          // 4 warps expand A, 4 expand B, 4 read out, 1 issues
constexpr int NW_N = 96;                 // B's rows: 3 genotypes of y x 32 columns
constexpr int NW_BSTAGE = NW_N * NODE_STAGE;
constexpr int NW_STAGES = 2;
constexpr uint32_t NW_TM_A = 320;        // tensor-memory column of A's stages (D: 0 .. 287)
constexpr int NW_SMEM = 120 * 1024;      // more than half an SM's: one block (it owns the tensor memory)

struct NodeProduct {
    const uint2* planes;       // [sample][words]
    const int8_t* dig;         // [32][mp]
    const NodeBin* bin;
    int64_t words, mp;
    int32_t n_samples;         // rows of the planes
    int32_t bins;
    int64_t idx0, idx1;        // the pairs (x <= y) of this chunk: y (y + 1) / 2 + x
    int64_t slot0;             // slot of pair idx0 within w's columns
    int64_t y0, first_unit, n_yx;   // first y; its first (y, x block) in the count from y = 0; how many
    double* w;
    int64_t stride;
    unsigned long long* stalled;
};

// (y, block of 128 samples x) number u, counted from y = 0: y has y / 128 + 1.
__host__ __device__ inline int64_t yx_before(int64_t y) {
    const int64_t q = y >> 7;
    return 64 * q * (q + 1) + (y - (q << 7)) * (q + 1);
}
__device__ __forceinline__ void decode_yx(int64_t u, int& y, int& xb) {
    int64_t q = (int64_t)((sqrt(1.0 + (double)u / 16.0) - 1.0) * 0.5);
    while (q > 0 && 64 * q * (q + 1) > u) q--;
    while (64 * (q + 1) * (q + 2) <= u) q++;
    const int64_t r = u - 64 * q * (q + 1);
    y = (int)((q << 7) + r / (q + 1));
    xb = (int)(r % (q + 1));
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
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__global__ void __launch_bounds__(NW_THREADS, 1) node_weights_kernel(NodeProduct P) {
    constexpr int J = NODE_J, L = NODE_L;
    extern __shared__ __align__(1024) unsigned char nw_smem[];
    __shared__ __align__(8) uint64_t full[NW_STAGES], empty[NW_STAGES], acc_full, acc_empty;
    __shared__ uint32_t tm_slot;
    __shared__ int gave_up;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t b0 = (smem_u32(nw_smem) + 1023u) & ~1023u;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NW_STAGES; i++) {
            mbar_init(&full[i], 8);     // the eight expanding warps
            mbar_init(&empty[i], 1);
        }
        mbar_init(&acc_full, 1);
        mbar_init(&acc_empty, 4);
        gave_up = 0;
        fence_mbar_init();
    }
    if (warp == 12) tmem_alloc<512>(smem_u32(&tm_slot));
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tm = tm_slot;
    const int64_t n_units = P.n_yx * P.bins;
    uint32_t seq = 0;    // stages so far
    bool ok = true;
    if (warp < 4) {
        // ---- A: a thread per sample x
        const uint32_t my = tm + ((uint32_t)(warp * 32) << 16) + NW_TM_A;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const int k = (int)(un / P.n_yx);
            int y, xb;
            decode_yx(P.first_unit + (un - k * P.n_yx), y, xb);
            const NodeBin bn = P.bin[k];
            const int x = xb * 128 + warp * 32 + lane;
            const bool live = x < P.n_samples;
            const uint4* src = reinterpret_cast<const uint4*>(P.planes + (int64_t)(live ? x : 0) * P.words + (bn.start >> 5));
            uint4 v0 = src[0], v1 = src[1];
            for (int i = 0; i < bn.stages; i++, seq++) {
                const uint32_t lo[4] = {v0.x, v0.z, v1.x, v1.z}, hi[4] = {v0.y, v0.w, v1.y, v1.w};
                if (i + 1 < bn.stages) {
                    v0 = src[2 * i + 2];
                    v1 = src[2 * i + 3];
                }
                const uint32_t st = seq % NW_STAGES;
                if (!nw_wait_warp(&empty[st], ((seq / NW_STAGES) & 1u) ^ 1u, &gave_up)) { ok = false; break; }
                tmem_fence_after();
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    uint32_t r[32];
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        uint32_t m = a == 0 ? ~(lo[w] | hi[w]) : a == 1 ? lo[w] & ~hi[w] : hi[w] & ~lo[w];
                        if (!live) m = 0u;
#pragma unroll
                        for (int q = 0; q < 8; q++) r[8 * w + q] = (m >> q) & 0x01010101u;
                    }
                    tmem_store32(my + st * 96 + a * 32, r);
                }
                tmem_store_wait();
                tmem_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[st]);
            }
        }
    } else if (warp < 8) {
        // ---- B: thread (row, 16-site piece); rows row and row + 16 of the
        // 32 columns, for the three genotypes of y
        const int tid = threadIdx.x - 128, c = tid & 7, row = tid >> 3;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const int k = (int)(un / P.n_yx);
            int y, xb;
            decode_yx(P.first_unit + (un - k * P.n_yx), y, xb);
            const NodeBin bn = P.bin[k];
            const int8_t* d0 = P.dig + (int64_t)row * P.mp + bn.start + 16 * c;
            const uint2* py = P.planes + (int64_t)y * P.words + (bn.start >> 5) + (c >> 1);
            uint4 va = *reinterpret_cast<const uint4*>(d0), vb = *reinterpret_cast<const uint4*>(d0 + 16 * P.mp);
            uint2 pl = py[0];
            for (int i = 0; i < bn.stages; i++, seq++) {
                const uint4 da = va, db = vb;
                const uint32_t lo = pl.x, hi = pl.y;
                if (i + 1 < bn.stages) {
                    va = *reinterpret_cast<const uint4*>(d0 + (int64_t)(i + 1) * NODE_STAGE);
                    vb = *reinterpret_cast<const uint4*>(d0 + 16 * P.mp + (int64_t)(i + 1) * NODE_STAGE);
                    pl = py[4 * (i + 1)];
                }
                const uint32_t st = seq % NW_STAGES;
                if (!nw_wait_warp(&empty[st], ((seq / NW_STAGES) & 1u) ^ 1u, &gave_up)) { ok = false; break; }
                const uint32_t base = b0 + st * NW_BSTAGE + ((uint32_t)(c ^ (row & 7)) << 4);
#pragma unroll
                for (int b = 0; b < 3; b++) {
                    const uint32_t m = (b == 0 ? ~(lo | hi) : b == 1 ? lo & ~hi : hi & ~lo) >> (4 * (c & 1));
                    uint32_t f[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) f[q] = ((m >> q) & 0x01010101u) * 255u;
                    const uint32_t at = base + (uint32_t)(b * 32 + row) * 128u;
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(da.x & f[0]),
                                 "r"(da.y & f[1]), "r"(da.z & f[2]), "r"(da.w & f[3])
                                 : "memory");
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 16u * 128u), "r"(db.x & f[0]),
                                 "r"(db.y & f[1]), "r"(db.z & f[2]), "r"(db.w & f[3])
                                 : "memory");
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[st]);
            }
        }
    } else if (warp < 12) {
        // ---- read-out: a thread per sample x; lanes of consecutive x are
        // consecutive slots
        const uint32_t my = tm + ((uint32_t)((warp - 8) * 32) << 16);
        // the genotype pair's number u (see the file comment) of (gx, gy) = (a, b)
        constexpr int UNIT[9] = {0, 2, 6, 4, 8, 5, 7, 3, 1};
        uint32_t n_acc = 0;
        const int nk = P.bins * J;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const int k = (int)(un / P.n_yx);
            int y, xb;
            decode_yx(P.first_unit + (un - k * P.n_yx), y, xb);
            if (P.bin[k].stages == 0) {
                // an empty bin: zero weights, no product
                const int x = xb * 128 + (warp - 8) * 32 + lane;
                const int64_t idx = (int64_t)y * (y + 1) / 2 + x;
                if (x <= y && idx >= P.idx0 && idx < P.idx1)
                    for (int u = 0; u < 9; u++)
                        for (int j = 0; j < J; j++)
                            P.w[((int64_t)u * nk + k * J + j) * P.stride + P.slot0 + (idx - P.idx0)] = 0.0;
                continue;
            }
            if (!nw_wait_warp(&acc_full, n_acc & 1u, &gave_up)) { ok = false; break; }
            n_acc++;
            tmem_fence_after();
            const int x = xb * 128 + (warp - 8) * 32 + lane;
            const int64_t idx = (int64_t)y * (y + 1) / 2 + x;
            const bool store = x <= y && idx >= P.idx0 && idx < P.idx1;
            double* out = P.w + (int64_t)(k * J) * P.stride + P.slot0 + (idx - P.idx0);
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
                    if (store) out[((int64_t)UNIT[ab] * nk + j) * P.stride] = (double)v;
                }
            }
        }
    } else if (lane == 0) {
        // ---- the issuing thread
        constexpr uint32_t idesc = idesc_i8(128, NW_N);
        uint32_t n_acc = 0;
        for (int64_t un = blockIdx.x; ok && un < n_units; un += gridDim.x) {
            const NodeBin bn = P.bin[un / P.n_yx];
            if (bn.stages == 0) continue;
            if (!nw_wait(&acc_empty, (n_acc & 1u) ^ 1u, &gave_up)) { ok = false; break; }
            n_acc++;
            tmem_fence_after();
            for (int i = 0; i < bn.stages; i++, seq++) {
                const uint32_t st = seq % NW_STAGES;
                if (!nw_wait(&full[st], (seq / NW_STAGES) & 1u, &gave_up)) { ok = false; break; }
                tmem_fence_after();
                const uint64_t bd = smem_desc_sw128(b0 + st * NW_BSTAGE);
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int a = 0; a < 3; a++)
                        mma_i8_ts(tm + a * NW_N, tm + NW_TM_A + st * 96 + a * 32 + 8 * q, bd + 2 * q, idesc,
                                  (i | q) != 0);
                mma_commit(smem_u32(&empty[st]));
            }
            if (ok) mma_commit(smem_u32(&acc_full));
        }
    }
    if (!ok && lane == 0) atomicAdd(P.stalled, 1ull);
    __syncwarp();
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    if (warp == 12) tmem_free<512>(tm);
}

// ------------------------------------------------------- first state, passes

// A run of one job's pairs (y-major: y (y + 1) / 2 + x) in consecutive slots.
struct NodeSeg {
    int64_t idx0;
    int32_t slot0, n, job, pad;
};

// Thread per slot: the pair's state before its first pass; thread 0 readies
// the wave counters and the clock.
__global__ void node_init_kernel(WaveArgs A, const NodeSeg* __restrict__ seg, int n_seg, int n,
                                 unsigned long long max_waves) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) {
        *A.wc_cur = WaveCounts{};
        *A.wc_next = WaveCounts{};
        A.wc_cur->n_pass = n;
        for (int i = 0; i < 3; i++) {
            A.clk->start[i] = ~0ull;
            A.clk->end[i] = 0ull;
        }
        A.clk->stop = 0;
        A.clk->waves = 0;
        A.clk->iters = 0;
        A.clk->max_waves = max_waves;
    }
    if (s >= n) return;
    int lo = 0, hi = n_seg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (seg[mid].slot0 <= s) lo = mid;
        else hi = mid - 1;
    }
    const NodeSeg g = seg[lo];
    const int64_t idx = g.idx0 + (s - g.slot0);
    int64_t y = (int64_t)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
    while (y > 0 && y * (y + 1) / 2 > idx) y--;
    while ((y + 1) * (y + 2) / 2 <= idx) y++;
    const int64_t x = idx - y * (y + 1) / 2;
    const CohortDev& co = A.cohorts[g.job];
    SlotState& S = A.slots[s];
    S.k = co.pair_begin + x * co.n_x - x * (x - 1) / 2 + (y - x);
    S.x = x;
    S.y = y;
    S.cohort = g.job;
    // two units a shape, one for het-het (UNIT in node_weights_kernel)
    for (int i = 0; i < 5; i++) S.ustart[i] = 2 * i;
    S.ustart[5] = NODE_UNITS;
    S.n = 0;
    S.lists64 = 1;
    S.fp64 = 1;
    S.near_count = 0;
    S.bls = 0;
    S.escalated = 0;
    S.gh = 0;
    S.f64p = 0;
    S.diffp = 0;
    S.it = 0;
    S.f = 0.0;
    double x0[9];
    for (int i = 0; i < 9; i++) x0[i] = x == y ? 0.0 : 1.0 / 9.0;
    if (x == y) { x0[0] = 0.5; x0[6] = 0.5; }
    normalise9(x0);
    for (int i = 0; i < 9; i++) { S.xc[i] = x0[i]; S.xt[i] = x0[i]; }
    S.ev = EV_INIT;
    S.kind = co.method == ESTIMATOR_CLS ? PASS_CLS64 : PASS_FP64;
    make_coef(x0, S.c64);
    S.status = SLOT_PASS;
    A.pass_cur[s] = s;
}

// 1 / d to an ulp or so: the hardware's approximation and one cubic Newton step.
__device__ __forceinline__ double node_rcp(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d, r, 1.0);
    return fma(fma(e, e, e), r, r);
}

// log d for eps <= d < 2 by table (Tang, ACM TOMS 16, 1990): d = 2^e m, c the
// reciprocal of the middle of m's 1/128 interval, log d = e log 2 - log c +
// log1p(m c - 1), the last by its series (|m c - 1| < 2^-8: the first term left
// out is below 3e-18).  The library's log is 30 FP64 instructions, this 9.
constexpr int LOG_CELLS = 128, LOG_EXPS = 64;
struct LogTable {
    double2 cell[LOG_CELLS];   // {c, -log c}
    double exp2[LOG_EXPS];     // (e - 40) log 2
};
__device__ __forceinline__ void fill_log_table(LogTable& T) {
    for (int i = threadIdx.x; i < LOG_CELLS; i += blockDim.x) {
        const double c = 1.0 / (1.0 + (i + 0.5) / LOG_CELLS);
        T.cell[i] = make_double2(c, -log(c));
    }
    for (int i = threadIdx.x; i < LOG_EXPS; i += blockDim.x) T.exp2[i] = (i - 40) * 0.69314718055994530942;
}
__device__ __forceinline__ double node_log(double d, const LogTable& T) {
    const int hi = __double2hiint(d);
    const double m = __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(d));
    const double2 c = T.cell[(hi >> 13) & (LOG_CELLS - 1)];
    const double r = fma(m, c.x, -1.0);
    double s = fma(r, -1.0 / 6.0, 0.2);
    s = fma(r, s, -0.25);
    s = fma(r, s, 1.0 / 3.0);
    s = fma(r, s, -0.5);
    s = fma(r * r, s, r);
    return (T.exp2[((hi >> 20) - 1023 + 40) & (LOG_EXPS - 1)] + c.y) + s;
}

// One genotype pair's nodes for one slot: the moments of its shape (SH) and the
// sum of W log d; the terms of stream64 with weights.  MIRROR: the pair sees 1
// - t.  The logarithms of four nodes are added before they join their sum, whose
// rounding is kept (two-sum): the Armijo test near convergence compares
// objectives to their last bits.  scale: what an integer weight stands for.
template <int SH, bool MIRROR>
__device__ __forceinline__ void node_unit(const NodeDev& N, const double* __restrict__ w, const PassCoef& K, double* P,
                                          int* cnt, bool write, bool count, const LogTable& T) {
    constexpr int NG = SH == 0 ? 4 : SH == 3 ? 4 : SH == 4 ? 2 : 3;
    constexpr int NH = SH == 0 ? 7 : SH == 3 ? 9 : SH == 4 ? 3 : 5;
    const double EPS = 1e-8;
    double k0, k1, k2 = 0.0, k3 = 0.0;
    if (SH == 0) { k0 = K.a[0]; k1 = K.a[1]; k2 = K.a[2]; k3 = K.a[3]; }
    if (SH == 1) { k0 = K.b1[0]; k1 = K.b1[1]; k2 = K.b1[2]; }
    if (SH == 2) { k0 = K.b2[0]; k1 = K.b2[1]; k2 = K.b2[2]; }
    if (SH == 3) { k0 = K.c[0]; k1 = K.c[1]; k2 = K.c[2]; k3 = K.c[3]; }
    if (SH == 4) { k0 = K.d[0]; k1 = K.d[1]; }
    double g[NG], h[NH], F = 0.0, Fl = 0.0;
#pragma unroll
    for (int i = 0; i < NG; i++) g[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NH; i++) h[i] = 0.0;
    const double2* __restrict__ tab = reinterpret_cast<const double2*>(N.t) + (MIRROR ? (NODE_VALS / 2) * N.nk : 0);
    const int64_t step = N.stride;
    auto node = [&](double W, const double2* __restrict__ e) {
        const double2 e0 = __ldg(e), e1 = __ldg(e + 1);
        const double t = e0.x, ty = e0.y, q = e1.x, t2 = e1.y;
        double d;
        if (SH == 0) {
            const double2 e2 = __ldg(e + 2), e3 = __ldg(e + 3);
            d = fma(t, fma(fma(fma(k3, t, k2), t, k1), t, k0), EPS);
            const double u = t * node_rcp(d), v = u * W;
            g[0] += v; g[1] = fma(v, t, g[1]); g[2] = fma(v, t2, g[2]); g[3] = fma(v, e2.x, g[3]);
            const double v2 = v * u;
            h[0] += v2; h[1] = fma(v2, t, h[1]); h[2] = fma(v2, t2, h[2]); h[3] = fma(v2, e2.x, h[3]);
            h[4] = fma(v2, e2.y, h[4]); h[5] = fma(v2, e3.x, h[5]); h[6] = fma(v2, e3.y, h[6]);
        } else if (SH == 1 || SH == 2) {
            const double2 e2 = __ldg(e + 2);
            d = fma(q, fma(fma(k2, t, k1), t, k0), EPS);
            const double u = q * node_rcp(d), v = u * W;
            g[0] += v; g[1] = fma(v, t, g[1]); g[2] = fma(v, t2, g[2]);
            const double v2 = v * u;
            h[0] += v2; h[1] = fma(v2, t, h[1]); h[2] = fma(v2, t2, h[2]); h[3] = fma(v2, e2.x, h[3]);
            h[4] = fma(v2, e2.y, h[4]);
        } else if (SH == 3) {
            d = fma(q, fma(q, k3, fma(t, k2, fma(ty, k1, k0))), EPS);
            const double u = q * node_rcp(d), v = u * W;
            g[0] += v; g[1] = fma(v, ty, g[1]); g[2] = fma(v, t, g[2]); g[3] = fma(v, q, g[3]);
            const double v2 = v * u, vy = v2 * ty, vq = v2 * q;
            h[0] += v2; h[1] += vy; h[2] = fma(v2, t, h[2]); h[3] += vq;
            h[4] = fma(vy, ty, h[4]); h[5] = fma(v2, t2, h[5]);
            h[6] = fma(vq, ty, h[6]); h[7] = fma(vq, t, h[7]); h[8] = fma(vq, q, h[8]);
        } else {
            d = fma(q, fma(q, k1, k0), EPS);
            const double u = q * node_rcp(d), v = u * W;
            g[0] += v; g[1] = fma(v, q, g[1]);
            const double v2 = v * u, vq = v2 * q;
            h[0] += v2; h[1] += vq; h[2] = fma(vq, q, h[2]);
        }
        return W * node_log(d, T);
    };
    static_assert(NODE_J % 4 == 0, "nodes come in fours");
    const double* wp = w;
    double W0 = wp[0], W1 = wp[step], W2 = wp[2 * step], W3 = wp[3 * step];
    for (int i = 0; i < N.nk; i += 4) {
        const double a0 = W0, a1 = W1, a2 = W2, a3 = W3;
        if (i + 4 < N.nk) {   // the next four nodes' weights in flight
            wp += 4 * step;
            W0 = wp[0]; W1 = wp[step]; W2 = wp[2 * step]; W3 = wp[3 * step];
        }
        const double2* e = tab + (NODE_VALS / 2) * i;
        const double f = (node(a0, e) + node(a1, e + 4)) + (node(a2, e + 8) + node(a3, e + 12));
        const double s = F + f, z = s - F;
        Fl += (F - (s - z)) + (f - z);
        F = s;
    }
    if (!write) return;
    const double scale = N.scale;
#pragma unroll
    for (int i = 0; i < NG; i++) P[i] = g[i] * scale;
#pragma unroll
    for (int i = 0; i < NH; i++) P[NG + i] = h[i] * scale;
    P[UNIT_VALS - 1] = (F + Fl) * scale;
    if (count) {
        double C = 0.0;
        for (int i = 0; i < N.nk; i++) C += w[(int64_t)i * step];
        *cnt = __double2int_rn(C * scale);
    }
}

// The CLS moments (cls_stream64) of one genotype pair's nodes.
template <int SH, bool MIRROR>
__device__ __forceinline__ void node_unit_cls(const NodeDev& N, const double* __restrict__ w, double* P, int* cnt,
                                              bool write) {
    constexpr int NG = SH == 0 ? 4 : SH == 3 ? 4 : SH == 4 ? 2 : 3;
    constexpr int NH = SH == 0 ? 7 : SH == 3 ? 9 : SH == 4 ? 3 : 5;
    double g[NG], C = 0.0;
#pragma unroll
    for (int i = 0; i < NG; i++) g[i] = 0.0;
    const double2* __restrict__ tab = reinterpret_cast<const double2*>(N.t) + (MIRROR ? (NODE_VALS / 2) * N.nk : 0);
    for (int i = 0; i < N.nk; i++) {
        const double W = w[(int64_t)i * N.stride];
        const double2 e0 = __ldg(tab + (NODE_VALS / 2) * i), e1 = __ldg(tab + (NODE_VALS / 2) * i + 1);
        const double t = e0.x, ty = e0.y, q = e1.x, t2 = e1.y;
        if (SH == 0) {
            const double v = W * t;
            g[0] += v; g[1] = fma(v, t, g[1]); g[2] = fma(v, t2, g[2]); g[3] = fma(v * t2, t, g[3]);
        } else if (SH == 1 || SH == 2) {
            const double v = W * q;
            g[0] += v; g[1] = fma(v, t, g[1]); g[2] = fma(v, t2, g[2]);
        } else if (SH == 3) {
            const double v = W * q;
            g[0] += v; g[1] = fma(v, ty, g[1]); g[2] = fma(v, t, g[2]); g[3] = fma(v, q, g[3]);
        } else {
            const double v = W * q;
            g[0] += v; g[1] = fma(v, q, g[1]);
        }
        C += W;
    }
    if (!write) return;
    const double scale = N.scale;
#pragma unroll
    for (int i = 0; i < NG; i++) P[i] = g[i] * scale;
#pragma unroll
    for (int i = 0; i < NH; i++) P[NG + i] = 0.0;
    P[UNIT_VALS - 1] = 0.0;
    *cnt = __double2int_rn(C * scale);
}

template <int SH, bool MIRROR>
__device__ __forceinline__ void node_task(const WaveArgs& A, const SlotState& S, int s, int u, bool write,
                                          const LogTable& T) {
    const NodeDev N = A.nodes[S.cohort];
    const double* w = N.w + (int64_t)u * N.nk * N.stride + (s - N.slot0);
    double* P = A.partial + ((int64_t)s * A.max_units + u) * UNIT_VALS;
    int* cnt = A.node_cnt + (int64_t)s * NODE_UNITS + u;
    if (S.kind == PASS_CLS64) node_unit_cls<SH, MIRROR>(N, w, P, cnt, write);
    else node_unit<SH, MIRROR>(N, w, S.c64, P, cnt, write, S.ev == EV_INIT, T);
}

// A warp per (32 slots of the pass list, genotype pair), a thread per slot:
// the weights are stored slot-fastest, so a warp's loads are whole sectors,
// the node's frequency is the same for all lanes, and no sum crosses lanes.
// Genotype-pair-major, so an SM's warps run one shape's code at a time.  Bound
// by the FP64 pipe (the reciprocal and the logarithm are most of a node's
// operations).
extern "C" __global__ void __launch_bounds__(128, 4) node_pass_kernel(WaveArgs A) {
    __shared__ LogTable T;
    if (A.clk->stop) return;   // a device loop past its last wave
    fill_log_table(T);
    __syncthreads();
    if (threadIdx.x == 0) atomicMin(&A.clk->start[1], global_ns());
    const int lane = threadIdx.x & 31;
    const PhaseEnd pe{&A.clk->end[1], lane == 0};
    const int n = A.wc_cur->n_pass, groups = (n + 31) >> 5;
    const int64_t tasks = (int64_t)groups * NODE_UNITS;
    // consecutive tasks go to different SMs, so a short list spreads
    for (int64_t task = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; task < tasks;
         task += (int64_t)gridDim.x * (blockDim.x >> 5)) {
        const int u = (int)(task / groups), i = (int)(task - (int64_t)u * groups) * 32 + lane;
        const bool write = i < n;
        const int s = A.pass_cur[write ? i : n - 1];
        const SlotState& S = A.slots[s];
        switch (u) {
        case 0: node_task<0, false>(A, S, s, u, write, T); break;
        case 1: node_task<0, true>(A, S, s, u, write, T); break;
        case 2: node_task<1, false>(A, S, s, u, write, T); break;
        case 3: node_task<1, true>(A, S, s, u, write, T); break;
        case 4: node_task<2, false>(A, S, s, u, write, T); break;
        case 5: node_task<2, true>(A, S, s, u, write, T); break;
        case 6: node_task<3, false>(A, S, s, u, write, T); break;
        case 7: node_task<3, true>(A, S, s, u, write, T); break;
        default: node_task<4, false>(A, S, s, u, write, T); break;
        }
    }
}

// ------------------------------------------------------------------- host

// The waves of a chunk as one graph launch (a WHILE node over two waves), kept
// between calls: it depends on the workspace's buffers only, not on the cohort.
struct NodeEngine {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    std::vector<void*> key_bufs;
    uint64_t key_iterations = 0;
    int key_dev = -1;
    cudaStream_t key_st = nullptr;
    WaveArgs args[2]{};
    int pass_blocks = 0, solve_blocks = 0, qp_blocks = 0, step_blocks = 0;
    void drop() {
        if (x) cudaGraphExecDestroy(x);
        if (g) cudaGraphDestroy(g);
        x = nullptr;
        g = nullptr;
    }
    ~NodeEngine() {
        drop();
        for (auto& e : ev)
            if (e) cudaEventDestroy(e);
    }
    void wave(int par, cudaStream_t st) const {
        const WaveArgs& A = args[par];
        node_pass_kernel<<<pass_blocks, 128, 0, st>>>(A);
        wave_solve_kernel<<<solve_blocks, 128, WAVE_WPB * WARP_SMEM, st>>>(A);
        wave_qp_kernel<<<qp_blocks, QP_THREADS, 0, st>>>(A);
        wave_step_kernel<<<step_blocks, 128, 0, st>>>(A);
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
    std::vector<CohortDev> table((size_t)n_jobs);
    int64_t total = 0;
    int nk_max = 0;
    uint64_t max_iter = cfg.iterations;
    for (int i = 0; i < n_jobs; i++) {
        table[i] = make_cohort_dev(jobs[i], cfg.iterations);
        table[i].pair_begin = total;
        total += table[i].n_pairs;
        nk_max = std::max(nk_max, jobs[i].panel->nd_n * J);
        max_iter = std::max<uint64_t>(max_iter, table[i].max_iter);
    }
    // pairs in flight: all of them up to 2^20, or what half the free memory
    // (with what the workspace holds already) takes
    const size_t per_slot = sizeof(double) * NODE_UNITS * ((size_t)nk_max + UNIT_VALS) + sizeof(SlotState) +
                            sizeof(double) * QP_VALS + sizeof(int) * (3 + NODE_UNITS);
    size_t fr = 0, tot = 0;
    int64_t cap = std::min<int64_t>(total, cfg.slots > 0 ? cfg.slots : (int64_t)1 << 20);
    const size_t held = ws.scratch.bytes + ws.slots.bytes + ws.partial.bytes + ws.qp.bytes;
    if ((size_t)cap * per_slot > held) {
        KG_NODE_TRY(cudaMemGetInfo(&fr, &tot));
        cap = std::max<int64_t>(1, std::min<int64_t>(cap, (int64_t)((fr + held) / 2 / per_slot)));
    }
    const int64_t stride = (cap + 31) / 32 * 32;
    KG_NODE_TRY((cudaError_t)ws.scratch.reserve(sizeof(double) * NODE_UNITS * (size_t)nk_max * stride));
    KG_NODE_TRY((cudaError_t)ws.partial.reserve(sizeof(double) * NODE_UNITS * UNIT_VALS * (size_t)cap));
    KG_NODE_TRY((cudaError_t)ws.slots.reserve(sizeof(SlotState) * (size_t)cap));
    KG_NODE_TRY((cudaError_t)ws.qp.reserve((sizeof(double) * QP_VALS + sizeof(int)) * (size_t)cap));
    KG_NODE_TRY((cudaError_t)ws.lists_a.reserve(sizeof(int) * 2 * (size_t)cap));
    KG_NODE_TRY((cudaError_t)ws.lists_b.reserve(sizeof(int) * NODE_UNITS * (size_t)cap));
    // counters, one buffer: {wave counts x 2, task and queue words, live, clock,
    // run counters, finished pairs per job}
    const size_t off_live = sizeof(WaveCounts) * 2 + 64, off_clk = (off_live + sizeof(LiveQueue) + 15) & ~(size_t)15;
    const size_t off_run = off_clk + sizeof(WaveClock), off_done = off_run + sizeof(RunCounters);
    KG_NODE_TRY((cudaError_t)ws.node_counts.reserve(off_done + sizeof(unsigned long long) * n_jobs));
    const size_t off_nodes = sizeof(CohortDev) * n_jobs, off_seg = off_nodes + sizeof(NodeDev) * n_jobs;
    const size_t blob = off_seg + sizeof(NodeSeg) * n_jobs;
    KG_NODE_TRY((cudaError_t)ws.node_table.reserve(blob));
    KG_NODE_TRY((cudaError_t)ws.host.reserve(blob + sizeof(WaveClock) + sizeof(RunCounters)));
    char* counts = ws.node_counts.as<char>();
    char* dtab = ws.node_table.as<char>();
    char* htab = ws.host.as<char>();
    WaveClock* h_clk = reinterpret_cast<WaveClock*>(htab + blob);
    RunCounters* h_run = reinterpret_cast<RunCounters*>(h_clk + 1);
    // without a caller's wave limit, one that only bounds a loop that would not
    // end: a pair takes at most (1 + backtracks) passes per iteration
    const unsigned long long bound = 2ull * (max_iter + 2) * 16ull + 64ull;
    const char* hw = std::getenv("KESTREL_HOST_WAVES");
    const bool host_waves = hw && hw[0] == '1';
    const std::vector<void*> bufs{ws.scratch.p, ws.partial.p, ws.slots.p, ws.qp.p, ws.lists_a.p, ws.lists_b.p,
                                  ws.node_counts.p, ws.node_table.p, reinterpret_cast<void*>(off_nodes), reinterpret_cast<void*>((size_t)cap)};
    const bool same = E.key_bufs == bufs && E.key_iterations == cfg.iterations &&
                      E.key_dev == dev && E.key_st == st;
    if (!same) {
        E.drop();
        WaveArgs A{};
        A.cohorts = reinterpret_cast<CohortDev*>(dtab);
        A.nodes = reinterpret_cast<NodeDev*>(dtab + off_nodes);
        A.live = reinterpret_cast<LiveQueue*>(counts + off_live);
        unsigned long long* words = reinterpret_cast<unsigned long long*>(counts + sizeof(WaveCounts) * 2);
        A.admit_task = reinterpret_cast<int*>(words);
        A.queue = words + 1;
        A.pass_task = words + 2;
        A.clk = reinterpret_cast<WaveClock*>(counts + off_clk);
        A.counters = reinterpret_cast<RunCounters*>(counts + off_run);
        A.cohort_done = reinterpret_cast<unsigned long long*>(counts + off_done);
        A.precision = KG_PREC_FP32C;
        A.slots = ws.slots.as<SlotState>();
        A.n_slots = (int)cap;
        A.partial = ws.partial.as<double>();
        A.max_units = NODE_UNITS;
        A.tune = make_tune(cfg.iterations);
        A.qp_buf = ws.qp.as<double>();
        A.qp_list = reinterpret_cast<int*>(A.qp_buf + (size_t)QP_VALS * cap);
        A.unit_elems = UNIT_ELEMS;
        A.node_cnt = ws.lists_b.as<int>();
        for (int par = 0; par < 2; par++) {
            WaveArgs& W = E.args[par];
            W = A;
            W.pass_cur = ws.lists_a.as<int>() + (par ? cap : 0);
            W.pass_next = ws.lists_a.as<int>() + (par ? 0 : cap);
            W.wc_cur = reinterpret_cast<WaveCounts*>(counts) + par;
            W.wc_next = reinterpret_cast<WaveCounts*>(counts) + (par ^ 1);
        }
        int occ = 0;
        KG_NODE_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, node_pass_kernel, 128, 0));
        E.pass_blocks = ws.sm_count * std::max(1, occ);
        KG_NODE_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, wave_solve_kernel, 128, WAVE_WPB * WARP_SMEM));
        E.solve_blocks = ws.sm_count * std::max(1, occ);
        KG_NODE_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, wave_qp_kernel, QP_THREADS, 0));
        E.qp_blocks = ws.sm_count * std::max(1, occ);
        KG_NODE_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, wave_step_kernel, 128, 0));
        E.step_blocks = ws.sm_count * std::max(1, occ);
        KG_NODE_TRY(cudaFuncSetAttribute(node_weights_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NW_SMEM));
        for (auto& e : E.ev)
            if (!e) KG_NODE_TRY(cudaEventCreate(&e));
        E.key_bufs.clear();
        KG_NODE_TRY(cudaGraphCreate(&E.g, 0));
        cudaGraphConditionalHandle h;
        KG_NODE_TRY(cudaGraphConditionalHandleCreate(&h, E.g, 1, cudaGraphCondAssignDefault));
        cudaGraphNodeParams np{};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        cudaGraphNode_t node;
        KG_NODE_TRY(cudaGraphAddNode(&node, E.g, nullptr, 0, &np));
        cudaGraph_t body = np.conditional.phGraph_out[0];
        KG_NODE_TRY(cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        for (int par = 0; par < 2; par++) {
            E.wave(par, st);
            wave_end_kernel<<<1, 32, 0, st>>>(E.args[par], par, h, 0);
        }
        cudaGraph_t captured = nullptr;
        const cudaError_t ce = cudaGetLastError();
        const cudaError_t ee = cudaStreamEndCapture(st, &captured);
        KG_NODE_TRY(ce);
        KG_NODE_TRY(ee);
        KG_NODE_TRY(cudaGraphInstantiate(&E.x, E.g, 0));
        E.key_bufs = bufs;
        E.key_iterations = cfg.iterations;
        E.key_dev = dev;
        E.key_st = st;
    }
    std::memcpy(htab, table.data(), sizeof(CohortDev) * n_jobs);
    KG_NODE_TRY(cudaMemsetAsync(counts, 0, off_done + sizeof(unsigned long long) * n_jobs, st));
    NodeDev* h_nodes = reinterpret_cast<NodeDev*>(htab + off_nodes);
    NodeSeg* h_seg = reinterpret_cast<NodeSeg*>(htab + off_seg);
    RunCounters* d_run = reinterpret_cast<RunCounters*>(counts + off_run);
    int job = 0;
    int64_t at = 0;   // the job's next pair, y-major
    bool limit_hit = false;
    double build_ms = 0.0, pass_ms = 0.0, solve_ms = 0.0;
    uint64_t waves = 0, launches = 0;
    while (job < n_jobs && !limit_hit) {
        // the next chunk of pairs
        int n_seg = 0;
        int64_t n = 0;
        std::vector<int> in;
        while (job < n_jobs && n < cap) {
            const int64_t np = table[job].n_pairs, take = std::min<int64_t>(np - at, cap - n);
            if (take > 0) {
                const Cohort& c = *jobs[job].panel;
                h_seg[n_seg] = NodeSeg{at, (int32_t)n, (int32_t)take, job, 0};
                NodeDev& nd = h_nodes[job];
                nd.w = ws.scratch.as<double>();
                nd.stride = stride;
                nd.slot0 = 0;
                nd.nk = c.nd_n * J;
                nd.t = c.nd_t.as<double>();
                nd.scale = std::ldexp(1.0, -(8 * NODE_L - 2));
                in.push_back(job);
                n_seg++;
                n += take;
                at += take;
            }
            if (at == np) {
                job++;
                at = 0;
            }
        }
        KG_NODE_TRY(cudaMemcpyAsync(dtab, htab, blob, cudaMemcpyHostToDevice, st));
        KG_NODE_TRY(cudaEventRecord(E.ev[0], st));
        for (int k = 0; k < n_seg; k++) {
            const Cohort& c = *jobs[in[k]].panel;
            const NodeSeg& g = h_seg[k];
            NodeProduct P;
            P.planes = c.nd_planes.as<uint2>();
            P.dig = c.nd_dig.as<int8_t>();
            P.bin = reinterpret_cast<const NodeBin*>(c.nd_bins.as<int>() + NODE_MAX_BINS);
            P.mp = c.nd_mp;
            P.words = c.nd_mp / 32;
            P.n_samples = (int32_t)c.n_samples;
            P.bins = c.nd_n;
            P.idx0 = g.idx0;
            P.idx1 = g.idx0 + g.n;
            P.slot0 = g.slot0;
            auto y_of = [](int64_t idx) {
                int64_t y = (int64_t)((std::sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
                while (y > 0 && y * (y + 1) / 2 > idx) y--;
                while ((y + 1) * (y + 2) / 2 <= idx) y++;
                return y;
            };
            P.y0 = y_of(P.idx0);
            P.first_unit = yx_before(P.y0);
            P.n_yx = yx_before(y_of(P.idx1 - 1) + 1) - P.first_unit;
            P.w = ws.scratch.as<double>();
            P.stride = stride;
            P.stalled = &d_run->stalled_waits;
            const int grid = (int)std::min<int64_t>(ws.sm_count, P.n_yx * P.bins);
            node_weights_kernel<<<grid, NW_THREADS, NW_SMEM, st>>>(P);
        }
        node_init_kernel<<<(int)((n + 127) / 128), 128, 0, st>>>(
            E.args[0], reinterpret_cast<const NodeSeg*>(dtab + off_seg), n_seg, (int)n,
            cfg.max_waves ? cfg.max_waves - waves : bound);
        KG_NODE_TRY(cudaGetLastError());
        KG_NODE_TRY(cudaEventRecord(E.ev[1], st));
        launches += n_seg + 1;
        const WaveClock* d_clk = reinterpret_cast<const WaveClock*>(counts + off_clk);
        if (host_waves) {
            for (uint64_t k = 0;; k++) {
                E.wave((int)(k & 1), st);
                wave_end_kernel<<<1, 32, 0, st>>>(E.args[k & 1], 0, cudaGraphConditionalHandle{}, 0);
                KG_NODE_TRY(cudaMemcpyAsync(h_clk, d_clk, sizeof(WaveClock), cudaMemcpyDeviceToHost, st));
                KG_NODE_TRY(cudaStreamSynchronize(st));
                launches += 5;
                if (h_clk->stop) break;
            }
        } else {
            KG_NODE_TRY(cudaGraphLaunch(E.x, st));
        }
        KG_NODE_TRY(cudaMemcpyAsync(h_clk, d_clk, sizeof(WaveClock) + sizeof(RunCounters), cudaMemcpyDeviceToHost, st));
        KG_NODE_TRY(cudaStreamSynchronize(st));
        if (!host_waves) launches += 10 * h_clk->iters;
        float ms = 0.f;
        KG_NODE_TRY(cudaEventElapsedTime(&ms, E.ev[0], E.ev[1]));
        build_ms += ms;
        waves += h_clk->waves;
        limit_hit = h_clk->limit_hit != 0 || (cfg.max_waves && waves >= cfg.max_waves && job < n_jobs);
        if (h_run->stalled_waits) {
            err = "a device wait of the node weights ran out of its limit";
            return KG_ETIMEOUT;
        }
    }
    pass_ms = (double)h_clk->acc[1] * 1e-6;
    solve_ms = (double)h_clk->acc[2] * 1e-6;
    const RunCounters& rc = *h_run;
    stats.gh_passes = rc.gh_passes;
    stats.obj_passes = rc.obj_passes;
    stats.fp64_passes = rc.fp64_passes;
    stats.fp64_pairs = rc.fp64_pairs;
    stats.pair_sites = rc.pair_sites;
    stats.work_units = rc.work_units;
    stats.launches = launches;
    stats.flops_fp32 = rc.flops_fp32;
    stats.flops_fp64 = rc.flops_fp64;
    for (int k = 0; k < 5; k++) stats.shape_sites[k] = rc.shape_sites[k];
    stats.nonconverged = rc.nonconverged;
    stats.waves = waves;
    stats.slots = (uint64_t)cap;
    stats.admit_ms = build_ms;
    stats.pass_ms = pass_ms;
    stats.solve_ms = solve_ms;
    stats.pair_kernel_ms = build_ms + pass_ms + solve_ms;
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
