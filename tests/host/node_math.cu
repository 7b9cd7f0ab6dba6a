// The scalar functions of the passes over frequency nodes against long double,
// for the tests of them: on the host, or with the argument "device" on the GPU.
// Prints, per function, the largest error as a fraction of its bound (see
// tests/test_node_math.py) and the argument it occurs at.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "kg_advance.cuh"
#include "kg_log.cuh"
#include "kg_node.h"
#include "kg_qp1.cuh"

enum { RECIP, LOG, LOG1M, STEP, N_FN };

__host__ __device__ inline double value(int fn, double a, const kg::LogTable& T) {
    return fn == RECIP ? kg::recip<true>(a) : fn == LOG ? kg::node_log(a, T) : kg::node_neg_log1m(a, T);
}

__global__ void values_kernel(int fn, const double* a, double* v, int n, const kg::LogTable* T) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = value(fn, a[i], *T);
}

__global__ void steps_kernel(const double* xt, const double* xc, double* v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d[9];
    kg::difference_step(xt + 9 * i, xc + 9 * i, d);
    for (int k = 0; k < 9; k++) v[9 * i + k] = d[k];
}

template <class T>
static T* upload(const T* h, size_t n) {
    T* d = nullptr;
    if (cudaMalloc(&d, n * sizeof(T)) != cudaSuccess ||
        cudaMemcpy(d, h, n * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
        std::fprintf(stderr, "no device memory\n");
        std::exit(2);
    }
    return d;
}
static std::vector<double> download(const double* d, size_t n) {
    std::vector<double> h(n);
    if (cudaMemcpy(h.data(), d, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) std::exit(2);
    return h;
}

int main(int argc, char** argv) {
    const bool device = argc > 1 && !std::strcmp(argv[1], "device");
    kg::LogTable T;
    kg::fill_log_table(T);
    const kg::LogTable* dT = device ? upload(&T, 1) : nullptr;
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    const int n = 1 << 20;
    const long double U = 0x1p-53L;   // half an ulp, relative
    for (int fn = 0; fn < STEP; fn++) {
        std::vector<double> a(n), v(n);
        for (int i = 0; i < n; i++) {
            const double r = u(rng);
            if (fn == RECIP) a[i] = std::exp2(600.0 * r - 300.0) * (i & 1 ? 1.0 : -1.0);
            else if (fn == LOG) a[i] = i < 64 ? 1.0 + (i - 32) * 0x1p-40 : std::exp2(-32.0 + 63.9 * r);
            else if (i & 1) a[i] = (i & 2 ? 1.0 : -1.0) * std::exp2(-60.0 + 54.0 * r);   // the series
            else a[i] = 1.0 - std::exp2(-27.5 + 55.0 * r);   // d_old / d from 5e-9 to 1.9e8
        }
        if (device) {
            double* da = upload(a.data(), n);
            double* dv = upload(v.data(), n);
            values_kernel<<<n / 256, 256>>>(fn, da, dv, n, dT);
            v = download(dv, n);
        } else {
            for (int i = 0; i < n; i++) v[i] = value(fn, a[i], T);
        }
        long double worst = 0.0L;
        double at = 0.0;
        for (int i = 0; i < n; i++) {
            const long double x = a[i];
            const long double want = fn == RECIP ? 1.0L / x : fn == LOG ? logl(x) : -log1pl(-x);
            const long double bound = fn == RECIP ? 2.0L * U * fabsl(want)
                                      : fn == LOG ? 4.0L * U * (1.0L + fabsl(want))
                                      : fabsl(x) <= 0.015625L ? 1e-15L * fabsl(want)
                                                              // the argument 1 - z is rounded to its ulp
                                                              : 4.0L * U * (1.0L + fabsl(want)) + 2.0L * U;
            const long double e = fabsl((long double)v[i] - want) / bound;
            if (!(e <= worst)) {
                worst = e;
                at = a[i];
            }
        }
        std::printf("%s %.4Lf %.17g\n", fn == RECIP ? "recip" : fn == LOG ? "log" : "neg_log1m", worst, at);
    }
    // steps of 1e-3 to 1e-9 between points of the simplex
    const int m = 1 << 16;
    std::vector<double> xt(9 * m), xc(9 * m), d(9 * m);
    for (int i = 0; i < m; i++) {
        const double len = std::pow(10.0, -3.0 - 6.0 * u(rng));
        double s = 0.0, t = 0.0;
        for (int k = 0; k < 9; k++) s += xc[9 * i + k] = u(rng) < 0.3 ? 0.0 : u(rng);
        if (s == 0.0) s = xc[9 * i] = 1.0;
        for (int k = 0; k < 9; k++) xc[9 * i + k] /= s;
        for (int k = 0; k < 9; k++) t += xt[9 * i + k] = xc[9 * i + k] * (1.0 + len * (u(rng) - 0.5));
        for (int k = 0; k < 9; k++) xt[9 * i + k] /= t;
    }
    if (device) {
        double *a = upload(xt.data(), xt.size()), *b = upload(xc.data(), xc.size()), *v = upload(d.data(), d.size());
        steps_kernel<<<m / 256, 256>>>(a, b, v, m);
        d = download(v, d.size());
    } else {
        for (int i = 0; i < m; i++) {
            double o[9];
            kg::difference_step(&xt[9 * i], &xc[9 * i], o);
            std::memcpy(&d[9 * i], o, sizeof(o));
        }
    }
    long double worst = 0.0L;
    for (int i = 0; i < m; i++) {
        long double sum = 0.0L, big = 0.0L, was = 0.0L;
        for (int k = 0; k < 9; k++) {
            sum += d[9 * i + k];
            was += (long double)xt[9 * i + k] - xc[9 * i + k];
            big += fabsl((long double)xt[9 * i + k] - xc[9 * i + k]);
        }
        // the step's own roundings, twice, and the part taken out times the sum's ulps
        const long double e = fabsl(sum) / (4.0L * U * big + 16.0L * U * fabsl(was) + 0x1p-1000L);
        worst = e > worst ? e : worst;
    }
    std::printf("step %.4Lf\n", worst);
    // the bound of a call's waves grows with its iteration limit, up to the largest
    unsigned long long last = 0;
    double wrapped = 0.0;
    for (int b = 0; b < 64; b++)
        for (uint64_t it : {((uint64_t)1 << b) - 2 * (b > 0), ((uint64_t)1 << b) - 1, (uint64_t)1 << b, ~(uint64_t)0 >> (63 - b)}) {
            const unsigned long long w = kg::wave_bound(it, 2);
            const uint64_t least = it < 1ull << 40 ? it : 1ull << 40;
            if (w / 11 < least || w / 22 < least || w + 4096 < last) wrapped = 2.0;
            last = w;
        }
    std::printf("wave_bound %.4f\n", wrapped);
    // no segment of a bin, cut into equal parts as the kernel cuts it, has more digits of
    // -128 than 32 bits hold, up to the most sites that places allow
    double sums = 0.0;
    for (int64_t stages : {1ll, 127ll, 2047ll, 2048ll, 2049ll, 65535ll, 65536ll, 65537ll, 131071ll, 131072ll, 131073ll, 156251ll, 16777215ll})
        for (int64_t units : {1ll, 2ll, 73ll, 74ll, 75ll, 4608ll, 1ll << 40}) {
            const int64_t seg = kg::node_seg_stages(stages, units, 148);
            const int64_t parts = kg::node_segments(stages, seg);
            int64_t last = 0;
            for (int64_t k = 0; k < parts; k++) {
                const int64_t end = stages * (k + 1) / parts, n = end - last;
                const double sum = (double)n * kg::NODE_STAGE * 128.0 / 2147483648.0;
                if (n < 1) sums = 2.0;
                if (sum > sums) sums = sum;
                last = end;
            }
            if (last != stages) sums = 2.0;
        }
    std::printf("segments %.4f\n", sums);
    return 0;
}
