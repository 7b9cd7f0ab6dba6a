// kg_advance.cuh — the SQP between two passes, a thread per pair: pairs in
// slots, waves of a pass kernel (frequency nodes in kg_node.cu, soft
// likelihoods in kg_soft.cu) and the advance step here, as one graph launch.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>

#include <string>

#include "kg_pair.cuh"
#include "kg_qp1.cuh"
#include "kg_wave.cuh"

namespace kg {

// A run of one job's pairs (y-major: y (y + 1) / 2 + x; query x panel: x n_y +
// y) in consecutive slots.
struct PairSeg {
    int64_t idx0;
    int32_t slot0, n, job, pad;
};

// Per-slot values lie in blocks of 32 slots, value-major inside: value v of
// slot s, of V values, at [(s / 32) V 32 + v 32 + s % 32].
constexpr int NS_LANES = 32;
__host__ __device__ __forceinline__ int64_t slot_at(int s, int values) {
    return (int64_t)(s >> 5) * (values * NS_LANES) + (s & 31);
}

// A slot's SQP state (src/sqp.rs:49-93) between its passes.
enum : int {
    NS_XC = 0,        // accepted point
    NS_XT = 9,        // point of the pending pass
    NS_P = 18,        // search direction
    NS_F = 27,        // objective at xc
    NS_GP = 28,       // g . p
    NS_ALPHA = 29,
    NS_N = 30,        // the pair's sites
    NS_COEF = 31,     // PassCoef at xt (16)
    NS_STEP = 47,     // PassCoef of the step (16), or the step itself (9): difference passes
    NS_VALS = 63
};
constexpr int NS_COEFS = (int)(sizeof(PassCoef) / sizeof(double));
static_assert(NS_COEFS == 16, "PassCoef: a 4, b1 3, b2 3, c 4, d 2");

// The waves' control words.
struct SlotCtl {
    int n[2];              // pending passes of the even and the odd waves
    unsigned int ticket;   // blocks of the advance kernel that are done
    int n_seg;             // runs of the chunk
    unsigned long long max_waves;
};

// Kinds of a pending pass: the pair's first, direct objective, objective
// change; for passes that are not FP64 by themselves, an FP64 one and the FP64
// re-evaluation of an accepted point.
enum : int { NP_FIRST = 0, NP_DIRECT = 1, NP_DIFF = 2, NP_FP64 = 3, NP_REEVAL = 4 };

struct SlotArgs {
    const CohortDev* cohorts;
    const PairSeg* seg;        // the chunk's runs (ctl->n_seg)
    double* state;             // NS_VALS values a slot
    int4* count;               // {iterations, backtracks | near count << 8 | FP64 passes << 16, passes, job * 8 + kind}
    int* list_cur;             // slots with a pending pass
    int* list_next;
    int par;                   // 0: even waves
    SlotCtl* ctl;
    WaveClock* clk;
    RunCounters* counters;
    Tune tune;
};

__device__ __forceinline__ PairSeg seg_of(const PairSeg* seg, int n_seg, int s) {
    int lo = 0, hi = n_seg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (seg[mid].slot0 <= s) lo = mid;
        else hi = mid - 1;
    }
    return seg[lo];
}

__host__ __device__ inline void pair_of(int64_t idx, int64_t& x, int64_t& y) {
    y = (int64_t)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
    while (y > 0 && y * (y + 1) / 2 > idx) y--;
    while ((y + 1) * (y + 2) / 2 <= idx) y++;
    x = idx - y * (y + 1) / 2;
}

// The samples of a job's pair idx, and its output row.
__device__ __forceinline__ int64_t job_pair(const CohortDev& co, int64_t idx, int64_t& x, int64_t& y) {
    if (co.kind == COHORT_RECT) {
        x = idx / co.n_y;
        y = idx - x * co.n_y;
        return idx;
    }
    pair_of(idx, x, y);
    return x * co.n_x - x * (x - 1) / 2 + (y - x);
}

__device__ __forceinline__ void node_write_row(kg_output* o, int64_t x, int64_t y, const double* d, double obj,
                                               uint64_t iters, double cond) {
    o->x = (uint64_t)x;
    o->y = (uint64_t)y;
#pragma unroll
    for (int i = 0; i < 9; i++) o->jacquard[i] = d[i];
    o->obj = obj;
    o->iters = iters;
    o->cond = cond;
}

__device__ __forceinline__ void store_coef(double* v, const double* x) {
    PassCoef k;
    make_coef(x, k);
    const double* c = reinterpret_cast<const double*>(&k);
#pragma unroll
    for (int i = 0; i < NS_COEFS; i++) v[i * NS_LANES] = c[i];
}

// The step xt - xc of a difference pass, less its part along xc: both points
// add up to 1 only to an ulp, and the objective would change by that ulp (its
// slope along x itself is -1) where the step's own change is smaller still.
__host__ __device__ __forceinline__ void difference_step(const double* xt, const double* xc, double (&d)[9]) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        d[i] = xt[i] - xc[i];
        s += d[i];
    }
#pragma unroll
    for (int i = 0; i < 9; i++) d[i] = fma(-s, xc[i], d[i]);
}

template <bool COEF>
__device__ __forceinline__ void store_step(double* v, const double* xt, const double* xc) {
    double d[9];
    difference_step(xt, xc, d);
    if (COEF) {
        store_coef(v, d);
    } else {
#pragma unroll
        for (int i = 0; i < 9; i++) v[i * NS_LANES] = d[i];
    }
}

// Thread per slot: the pair's state before its first pass; thread 0 readies
// the control words and the clock.
__device__ __forceinline__ void init_slot(const SlotArgs& A, int n_seg, int n, unsigned long long max_waves) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) {
        A.ctl->n[0] = n;
        A.ctl->n[1] = 0;
        A.ctl->ticket = 0;
        A.ctl->n_seg = n_seg;
        A.ctl->max_waves = max_waves;
        for (int i = 0; i < 3; i++) {
            A.clk->start[i] = ~0ull;
            A.clk->end[i] = 0ull;
        }
        A.clk->stop = 0;
        A.clk->waves = 0;
        A.clk->iters = 0;
    }
    if (s >= n) return;
    const PairSeg g = seg_of(A.seg, n_seg, s);
    const CohortDev& co = A.cohorts[g.job];
    int64_t x, y;
    job_pair(co, g.idx0 + (s - g.slot0), x, y);
    const bool self_pair = co.kind == COHORT_TRIANGLE && x == y;
    double x0[9];
    for (int i = 0; i < 9; i++) x0[i] = self_pair ? 0.0 : 1.0 / 9.0;
    if (self_pair) { x0[0] = 0.5; x0[6] = 0.5; }
    normalise9(x0);
    double* st = A.state + slot_at(s, NS_VALS);
#pragma unroll
    for (int i = 0; i < 9; i++) st[(NS_XT + i) * NS_LANES] = x0[i];
    store_coef(st + NS_COEF * NS_LANES, x0);   // (soft likelihoods do not read them)
    A.count[s] = make_int4(0, 0, 0, 8 * g.job + NP_FIRST);
    A.list_cur[s] = s;
}

constexpr int NA_THREADS = 32;   // one warp a block: few slots spread over the SMs

// One slot: returns the kind of its next pass, or -1 when its row is written.
// my: the thread's column of the shared memory; sum: the block's counters; src:
// where the pass's sums come from (Sums::FP32: its passes are FP32, and a pair
// whose condition estimate exceeds COND_RECHECK, or whose KKT residual stalls
// below 1e-6 three times, goes on in FP64).
template <class Sums>
__device__ __forceinline__ int advance_slot(const SlotArgs& A, const Sums& src, int s, double* my,
                                            unsigned long long* sum) {
    const Tune& tu = A.tune;
    constexpr int SD = NS_LANES;
    double* st = A.state + slot_at(s, NS_VALS);
    const int4 ct = A.count[s];
    const int kind = ct.w & 7, job = ct.w >> 3, bls = ct.y & 0xFF;
    int near_count = (ct.y >> 8) & 0xFF;
    const int f64p = Sums::FP32 ? min((ct.y >> 16) + (kind >= NP_FP64 ? 1 : 0), 0x7FFF) : 0;
    const bool fp64 = f64p > 0;
    // ---- the sums, and H and g from them
    double xt[9], g[9], obj, nsites;
    {
        double T[QP_Q];
        src.load(s, kind, st, obj, g, T, nsites);
        const double rn = 1.0 / nsites;
#pragma unroll
        for (int k = 0; k < QP_Q; k++) my[k * NA_THREADS] = quot(T[k], nsites, rn);
#pragma unroll
        for (int k = 0; k < 9; k++) g[k] = quot(-g[k], nsites, rn);
    }
#pragma unroll
    for (int k = 0; k < 9; k++) xt[k] = st[(NS_XT + k) * SD];
    const int gh = ct.z + 1;
    int it = ct.x;
    double f;
    int next = -1;   // the kind of the next pass (-1: the pair is done)
    bool trial_again = false;
    if (kind == NP_FIRST || kind == NP_REEVAL) {
        f = -obj / nsites;
    } else {
        // Armijo (src/sqp.rs:294): a difference pass has the objective's
        // change itself, which the test resolves far below an ulp of f
        const double f0 = st[NS_F * SD], alpha = st[NS_ALPHA * SD], gp = st[NS_GP * SD];
        const double bar = alpha * (tu.bls_sufficient_decrease * gp);
        const double df = -obj / nsites;
        f = kind == NP_DIFF ? f0 + df : df;
        const bool accept = kind == NP_DIFF ? df <= bar : f <= f0 + bar;
        if (!accept && bls + 1 != tu.bls_max_iter) {
            trial_again = true;
            const double a2 = alpha * tu.bls_step_size_reduce;
            double xc[9], sum_x = 0.0;
#pragma unroll
            for (int k = 0; k < 9; k++) {
                xc[k] = st[(NS_XC + k) * SD];
                xt[k] = xc[k] + a2 * st[(NS_P + k) * SD];
                sum_x += xt[k];
            }
#pragma unroll
            for (int k = 0; k < 9; k++) {
                xt[k] = xt[k] / sum_x;
                st[(NS_XT + k) * SD] = xt[k];
            }
            st[NS_ALPHA * SD] = a2;
            next = fp64 ? NP_FP64 : fabs(a2 * gp) < DIFF_BELOW ? NP_DIFF : NP_DIRECT;
            if (Sums::COEF) store_coef(st + NS_COEF * SD, xt);
            if (next == NP_DIFF) store_step<Sums::COEF>(st + NS_STEP * SD, xt, xc);
            A.count[s] = make_int4(it, (bls + 1) | (near_count << 8) | (f64p << 16), gh, 8 * job + next);
        } else {
            it++;
        }
    }
    if (!trial_again) {
        // ---- the accepted point
        const CohortDev& co = A.cohorts[job];
        double resid = 0.0, cond = CUDART_NAN;
        const bool none = nsites == 0.0, last = (uint64_t)it >= co.max_iter;
        const bool conv = !none && !last && kkt_ok(xt, g, tu.sqp_conv_tol, &resid);
        if (conv) cond = condition_thread([my](int k) { return my[k * NA_THREADS]; }, xt, g, tu.sqp_conv_tol);
        bool recheck = false;
        if (Sums::FP32 && !none && !last && !fp64 && (conv || resid < 1e-6)) {
            near_count += conv ? 0 : 1;
            recheck = conv ? !(cond <= COND_RECHECK) : near_count >= 3;
        }
        if (recheck) {
            // the same point again, in FP64; the pair stays FP64
            next = NP_REEVAL;
            A.count[s] = make_int4(it, near_count << 8, gh, 8 * job + next);
            atomicAdd(&sum[5], 1ull);
        } else if (none || last || conv) {
            const PairSeg sg = seg_of(A.seg, A.ctl->n_seg, s);
            int64_t x, y;
            const int64_t row = job_pair(co, sg.idx0 + (s - sg.slot0), x, y);
            if (none) {
#pragma unroll
                for (int k = 0; k < 9; k++) xt[k] = Sums::none();
                f = CUDART_NAN;
            }
            node_write_row(co.out + row, x, y, xt, f, none ? 0 : last ? co.max_iter : (uint64_t)it, cond);
            // the counters of the call
            if (none) {
                atomicAdd(&sum[0], 1ull);
            } else {
                atomicAdd(&sum[1], (unsigned long long)gh);
                atomicAdd(&sum[2], (unsigned long long)nsites);
                atomicAdd(&sum[3], (unsigned long long)nsites * (unsigned long long)gh);
                if (last) atomicAdd(&sum[4], 1ull);
                src.count(s, job, gh, f64p, nsites, conv && !(cond <= COND_RECHECK), sum);
            }
        } else {
            // ---- the QP and the step (src/sqp.rs:78-90)
            auto H = [my](int i2, int j2) { return my[(i2 <= j2 ? upper_at(i2, j2) : upper_at(j2, i2)) * NA_THREADS]; };
#pragma unroll
            for (int r = 0; r < 9; r++) {
                double hx = 0.0;
#pragma unroll
                for (int j = 0; j < 9; j++) hx = fma(H(r, j), xt[j], hx);
                my[(QP_Q + r) * NA_THREADS] = g[r] - hx;
                st[(NS_XC + r) * SD] = xt[r];
            }
            st[NS_F * SD] = f;
            double y[9];
#pragma unroll
            for (int k = 0; k < 9; k++) y[k] = xt[k];
            qp_simplex_thread<true>([my](int v) { return my[v * NA_THREADS]; }, tu, y);
            // g . p with p = y - x; the first trial point x + p, normalised
            double gp = 0.0, sum_x = 0.0, p[9];
#pragma unroll
            for (int k = 0; k < 9; k++) {
                p[k] = y[k] - xt[k];
                gp = fma(g[k], p[k], gp);
                y[k] = xt[k] + p[k];
                sum_x += y[k];
            }
#pragma unroll
            for (int k = 0; k < 9; k++) {
                st[(NS_P + k) * SD] = p[k];
                y[k] = y[k] / sum_x;
                st[(NS_XT + k) * SD] = y[k];
            }
            st[NS_GP * SD] = gp;
            st[NS_ALPHA * SD] = 1.0;
            next = fp64 ? NP_FP64 : fabs(gp) < DIFF_BELOW ? NP_DIFF : NP_DIRECT;
            if (Sums::COEF) store_coef(st + NS_COEF * SD, y);
            if (next == NP_DIFF) store_step<Sums::COEF>(st + NS_STEP * SD, y, xt);
            A.count[s] = make_int4(it, (near_count << 8) | (f64p << 16), gh, 8 * job + next);
        }
    }
    return next;
}

// Everything between two passes of a slot, a thread per slot: its moments,
// the Armijo accept test (a rejected trial backs off and takes the next pass),
// the KKT test, at convergence the condition estimate and the row, else the
// simplex QP and the next trial point.  The state and the sums are blocked by 32
// slots, so a warp's loads and stores are whole sectors; H and c go
// through shared memory (432 bytes a thread) into the QP.  One kernel instead
// of the list form's solve, QP and step kernels: nothing is written between
// them and a wave over few slots waits for one launch.  Bound by the FP64
// chains of the QP (nine pivots one after the other, up to ten times).  The
// last block to finish ends the wave: it adds the phase times and decides
// whether the loop goes on.
template <class Sums>
__device__ __forceinline__ void advance_wave(const SlotArgs& A, const Sums& src, int in_loop,
                                             cudaGraphConditionalHandle loop) {
    __shared__ double in[QP_IN * NA_THREADS];
    __shared__ unsigned long long sum[12];
    if (A.clk->stop) {   // a device loop past its last wave
        if (in_loop && A.par && blockIdx.x == 0 && threadIdx.x == 0) {
            A.clk->iters++;
            cudaGraphSetConditional(loop, 0u);
        }
        return;
    }
    const int n = A.ctl->n[A.par];
    if (threadIdx.x < 12) sum[threadIdx.x] = 0ull;
    if (threadIdx.x == 0 && (int)blockIdx.x * NA_THREADS < n) atomicMin(&A.clk->start[2], global_ns());
    __syncwarp();
    double* my = in + threadIdx.x;
    for (int base = blockIdx.x * NA_THREADS; base < n; base += gridDim.x * NA_THREADS) {
        const bool live = base + (int)threadIdx.x < n;
        const int s = A.list_cur[live ? base + threadIdx.x : n - 1];
        const int next = live ? advance_slot(A, src, s, my, sum) : -1;
        __syncwarp();
        // slots with another pass join the next wave's list, in this list's order
        const unsigned more = __ballot_sync(0xffffffffu, next >= 0);
        int at = 0;
        if (threadIdx.x == 0 && more) at = atomicAdd(&A.ctl->n[A.par ^ 1], __popc(more));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (next >= 0) A.list_next[at + __popc(more & ((1u << threadIdx.x) - 1u))] = s;
    }
    __syncwarp();
    if (threadIdx.x < 12 && sum[threadIdx.x]) {
        RunCounters* C = A.counters;
        const unsigned long long v = sum[threadIdx.x];
        switch (threadIdx.x) {
        case 0: atomicAdd(&C->nosite_pairs, v); break;
        case 1: atomicAdd(&C->gh_passes, v); break;
        case 2: atomicAdd(&C->pair_sites, v); break;
        case 3: atomicAdd(&C->work_units, v); break;
        case 4: atomicAdd(&C->nonconverged, v); break;
        case 5: atomicAdd(&C->fp64_pairs, v); break;
        case 6: atomicAdd(&C->flops_fp64, v); break;
        default: atomicAdd(&C->shape_sites[threadIdx.x - 7], v); break;
        }
    }
    __syncwarp();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&A.ctl->ticket, 1u) != gridDim.x - 1) return;
    // ---- the wave's end
    __threadfence();
    WaveClock* c = A.clk;
    volatile SlotCtl* ctl = A.ctl;
    const unsigned long long now = global_ns();
    const unsigned long long p0 = *reinterpret_cast<volatile unsigned long long*>(&c->start[1]);
    const unsigned long long p1 = *reinterpret_cast<volatile unsigned long long*>(&c->end[1]);
    const unsigned long long s0 = *reinterpret_cast<volatile unsigned long long*>(&c->start[2]);
    if (p1 > p0) c->acc[1] += p1 - p0;
    if (now > s0) c->acc[2] += now - s0;
    c->waves++;
    unsigned int stop = 0;
    if (ctl->n[A.par ^ 1] == 0) {
        stop = 1;
    } else if (c->waves >= ctl->max_waves) {
        stop = 1;
        c->limit_hit = 1;
    }
    c->stop = stop;
    ctl->n[A.par] = 0;
    ctl->ticket = 0;
    for (int k = 0; k < 3; k++) {
        c->start[k] = ~0ull;
        c->end[k] = 0ull;
    }
    if (in_loop && A.par) {
        c->iters++;
        cudaGraphSetConditional(loop, stop ? 0u : 1u);
    }
}

// Waves that no pair needs more of, which only bound a loop that would not end: at
// most (1 + backtracks) passes per iteration, in each of its forms (FP32 and FP64).
inline unsigned long long wave_bound(uint64_t iterations, int forms) {
    const uint64_t most = 1ull << 50;   // whatever the caller asks for, the product does not wrap
    return (unsigned long long)forms * ((iterations < most ? iterations : most) + 2) * 32ull + 64ull;
}

// The waves as one graph launch: a WHILE node over an even and an odd wave.
// wave(par, in_loop, handle) launches one on st, which captures.  Returns a
// CUDA error.
template <class Wave>
inline cudaError_t wave_loop_graph(cudaStream_t st, const Wave& wave, cudaGraph_t* g, cudaGraphExec_t* x) {
    cudaError_t e = cudaGraphCreate(g, 0);
    if (e != cudaSuccess) return e;
    cudaGraphConditionalHandle h;
    e = cudaGraphConditionalHandleCreate(&h, *g, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) return e;
    cudaGraphNodeParams np{};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    e = cudaGraphAddNode(&node, *g, nullptr, 0, &np);
    if (e != cudaSuccess) return e;
    e = cudaStreamBeginCaptureToGraph(st, np.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                      cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    for (int par = 0; par < 2; par++) wave(par, 1, h);
    cudaGraph_t captured = nullptr;
    const cudaError_t ce = cudaGetLastError(), ee = cudaStreamEndCapture(st, &captured);
    if (ce != cudaSuccess) return ce;
    if (ee != cudaSuccess) return ee;
    return cudaGraphInstantiate(x, *g, 0);
}

}  // namespace kg
