// kg_node.h — pairs estimated from frequency nodes instead of site lists
// (host-side interface of kg_node.cu).
//
// Every sum an SQP pass forms over a pair's sites (src/jacquard/objective.rs:
// 9-20, grad_hess.rs:13-41) is, within one genotype-pair shape, a sum of a
// smooth function phi of the site's allele frequency t.  phi is one of log d, r
// t^k, r^2 t^k with d = eps + L.Delta, Delta on the simplex, whose
// singularities keep a distance from t that grows with min(t, 1 - t).  So the
// cohort's sites go into narrow frequency bins, in each bin phi is replaced by its
// interpolant through a few Chebyshev nodes, and
//   sum over the pair's sites of phi(t_s) = sum over nodes of W_node phi(t_node),
//   W_node = sum over those sites of l_node(t_s)  (l: the Lagrange basis).
// The weights W do not depend on Delta: they are formed once per pair, and every
// pass then evaluates 9 x (nodes per bin) x (bins) points instead of all sites.
// W of all pairs is a matrix product of genotype indicators with indicators
// times l, which kg_node.cu runs on the tensor cores in exact integers.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "kg_engine.h"

namespace kg {

// Nodes per bin, signed 8-bit digits of l's fixed-point value (2^-30), and the
// largest ratio of a bin's ends.  The interpolation error is then below 2e-10
// of a site's log d and 1.1e-10 of its gradient term x_i L_i / d anywhere on the
// simplex, and its mean over a bin's sites below 5e-13, against the 6e-8 of a FP32
// site term.  (With 2^(1/4) it is ten times lower, and no row of 1,024 samples x
// 100,000 sites is nearer to the FP64 form's, 9.6e-9 at most on both: where the two stop
// decides; but a third more nodes: 18.8 against 15.0 ms of passes, 13.3 against
// 13.0 ms of weights.)  The FP64 form keeps its site
// lists: with 12 nodes and 5 digits it ran 2.4 times as fast and 1e-13
// accurate, but within 1e-9 of the list form's rows only where no pair's last
// line search hangs on an ulp of the objective.
constexpr int NODE_J = 8, NODE_L = 4;
constexpr double NODE_RATIO = 1.2599210498948732;   // 2^(1/3)
constexpr int NODE_MAX_BINS = 64;
constexpr int NODE_UNITS = 9;        // genotype pairs (gx, gy)
constexpr int NODE_STAGE = 128;      // sites per tile of the product; a bin's sites are padded to it

// Stages that one 32-bit accumulator adds up at most: a site's digit is -128 at
// the least, and 2^16 x 128 x 128 = 2^30.
constexpr int NODE_SEG_STAGES = 1 << 16;
// The stages of a segment for a cohort of `stages` stages and `units` (y, x block)
// pairs.  With few pairs the fullest bin is one SM's work from end to end: 2
// samples x 3,000,000 sites took 3.9 ms of weights, in segments 0.23; eight units an SM
// even the blocks out (two, four, eight, sixteen: 3.67, 2.72, 2.73, 2.67 ms for 32 x
// 3,000,000, CLS 3.58, 3.01, 2.73, 2.76; whole bins 6.17 and 3.57).  Below 2,048
// stages, or with more pairs than half the SMs, the segments' two further passes over
// the weights cost what they save.
inline int64_t node_seg_stages(int64_t stages, int64_t units, int sms) {
    if (stages < 2048 || 2 * units > sms) return NODE_SEG_STAGES;
    const int64_t fair = (stages * units + 8 * sms - 1) / (8 * sms);
    return fair < 128 ? 128 : fair > NODE_SEG_STAGES ? NODE_SEG_STAGES : fair;
}
// The segments that a bin of up to `stages` stages takes at `seg` a segment.
inline int node_segments(int64_t stages, int64_t seg) { return (int)((stages + seg - 1) / seg); }
static_assert((int64_t)NODE_SEG_STAGES * NODE_STAGE * 128 < ((int64_t)1 << 31), "32-bit sums");

// Whether a prepared cohort's pairs run on nodes, given its kept sites and
// their smallest min(p, 1 - p), and the bins that takes (0: it does not: a
// frequency outside 0..1, or below 1/2 x 2^(-64/3) = 1.9e-7, the end of 64 bins).
// Nodes win at any size and range measured.  Whole calls of 2 samples x 300 sites took
// 0.50 ms against 1.35 ms on lists, 64 x 1,200 0.95 against 1.93, 600 x 300 9.0
// against 30.4, 600 x 10,000 11.3 against 43.2 ms, with frequencies from 0.05 up (10
// bins).  A pass costs the bins, not the sites, so wide ranges at few sites are
// nearest to the lists: from 4e-7 up (61 bins) 1,024 x 10 took 37 against 46 ms on
// the device, 1,024 x 100 62 against 170, 1,024 x 300 68 against 88, 64 x 40 0.90
// against 3.0, 1,024 x 30,000 80 against 198.
int node_bins(bool cls, int64_t n_kept, int64_t n_samples, double t_min);

// After the kept sites are compacted: bins, node points, digits and the
// samples' planes in bin order (c.nd_*).  codes: device byte codes.
int prepare_nodes(Cohort& c, const uint8_t* codes, int64_t stride, int bins, cudaStream_t st, std::string& err);

// A query's rows against a node-prepared panel (prepare_query for site lists).
int prepare_query_nodes(const Cohort& panel, QueryPlanes& q, const uint8_t* codes, int64_t n_rows, int64_t row_stride,
                        const uint8_t* site_mask, cudaStream_t st, std::string& err);

// All jobs (over node-prepared cohorts; queries by prepare_query_nodes) of one
// call.
int run_nodes(const std::vector<PairJob>& jobs, const RunConfig& cfg, Workspace& ws, cudaStream_t st,
              kg_run_stats& stats, std::string& err);

}  // namespace kg
