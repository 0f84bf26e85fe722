// FP64 forward for short vectors, n and d known at compile time.
//
// The FP64 pipe takes a warp instruction every 16 clocks per SM whatever the number of its
// active lanes, so what counts is that all lanes work and that every SM has some.  A CTA
// takes E entries; the E * n^d output elements of a mode are dealt to its threads in rounds
// (element q of the CTA belongs to entry q / n^d), so that lanes idle in the last warp only,
// whatever n^d is.  A small batch is spread over all SMs with one element per thread.  Modes
// run in place in shared memory, each element the k-ascending FMA chain of the other kernels:
// bitwise the same value.
//
// What bounds it: the FP64 pipe for large batches (1.02-1.19 of 1.25 TFLOP/s from n^d = 25 up),
// two dependent trips to memory, the barriers and the chain of d n additions for small ones.
// The kernels with a power-of-two team per entry left lanes idle (d = 2, n = 5: 131 -> 96 us at
// 200000 entries) and packed a small batch into few CTAs (d = 4, n = 4, 200 entries: 22.2 ->
// 4.8 us); n = 9 and 10 had one CTA per entry (d = 2, n = 10, 60000 entries: 310 -> 212 us).
#pragma once
#include "fwd_kernels.cuh"

namespace kgb {

constexpr int f64_pow(int b, int e) { return e <= 0 ? 1 : b * f64_pow(b, e - 1); }

template <int NN, int D> struct F64 {
    static constexpr int N = f64_pow(NN, D), P = NN * NN, F = N / NN;
    static constexpr int VS = (N + 1) / 2 * 2, FS = D * P;  // doubles per entry: vector, factors
    static constexpr int threads = N <= 1024 ? 256 : 512;
    static_assert(N <= 4 * threads, "vector too long");
};

// a.teams_per_cta entries per CTA, at most R elements per thread.  (Every warp runs through the
// code of all R rounds: with two rounds in the code of four, n = 2, d = 5, 8192 entries take
// 12.1 us instead of 8.3.)
template <int NN, int D, int R>
__global__ void __launch_bounds__(F64<NN, D>::threads, 1024 / F64<NN, D>::threads)
    fwd_f64_kernel(const FwdArgs<double, double> a)
{
    using K = F64<NN, D>;
    constexpr int N = K::N, P = K::P, F = K::F;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int T = blockDim.x, tid = threadIdx.x, E = a.teams_per_cta;
    double *const X = reinterpret_cast<double *>(smem_raw), *const M = X + E * K::VS;
    const long long e0 = (long long)blockIdx.x * E;
    const int ne = a.nb - e0 < E ? (int)(a.nb - e0) : E, total = ne * N;
    const double *const *in = a.in + e0;
    const double *const *mats = a.mats + e0 * D;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int q = tid + j * T;
        if (q < total) cp_async<8>(X + q / N * K::VS + q % N, in[q / N] + q % N);
    }
#pragma unroll 4
    for (int f = tid; f < ne * K::FS; f += T) {
        const int m = f / P, el = f % P;
        cp_async<8>(M + f, mats[m] + el % NN + (size_t)(el / NN) * a.stride);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    double y[R];
#pragma unroll
    for (int i = D - 1; i >= 0; --i) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int q = tid + j * T;
            if (q < total) {
                const int en = q / N, p = q % N, c = p / NN, r = p % NN;  // row r of fibre c
                double x[NN];
                load_fibre<double, NN>(X + en * K::VS + c * NN, x);
                const double *const A = M + en * K::FS + i * P + r;
                double s = 0.0;
#pragma unroll
                for (int k = 0; k < NN; ++k) s = fma(A[k * NN], x[k], s);
                y[j] = s;
            }
        }
        if (i > 0) __syncthreads();
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int q = tid + j * T;
            if (q < total) {
                const int en = q / N, p = q % N, at = p / NN + p % NN * F;
                if (i > 0)
                    X[en * K::VS + at] = y[j];
                else
                    atomic_add<double>(a.out[e0 + en] + at, y[j]);
            }
        }
        if (i > 0) __syncthreads();
    }
}

struct F64Info {
    const void *fn[3] = {};  // at most 1, 2 and 4 elements per thread (null: fewer than n^d per CTA)
    int n = 0, d = 0;  // of the instantiation
    int threads = 0, entry_bytes = 0;
};
F64Info f64_lookup(int n, int d);  // fn[2] == nullptr where there is no instantiation

}  // namespace kgb
