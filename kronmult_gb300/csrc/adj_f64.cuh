// FP64 adjoint, n and d known at compile time (adj_kernels.cuh has the definitions of p_i, q_i
// and the gradients, and the layouts).
//
// As in fwd_f64_kernel a CTA takes E entries and deals their elements to its threads in rounds,
// so that lanes idle in the last warp only and a small batch is spread over all SMs.  The
// p-sweep keeps every p_i in shared memory; then for every mode i one phase adds the
// contraction of q_i and p_i to the factor gradient and computes q_{i+1} into registers.  A
// contraction item is a pair (r, k) of an entry; S lanes share it (t = lane mod S, + S, ..)
// where the CTA has more threads than pairs, and add up by shuffles.  Both gradients go out
// with additions in L2, one per entry: no sums across entries, no slices in shared memory.
//
// What bounds it: the FP64 pipe for large batches (1.0-1.19 of 1.25 TFLOP/s), the 3 d phases'
// barriers and dependent additions for small ones.  Against the element kernels with a
// power-of-two team per entry: d = 3, n = 6 820 -> 735 us at 40000 entries, 20.4 -> 7.3 at 16;
// d = 4, n = 8 1058 -> 716 at 1000; d = 2, n = 4 43 -> 28 at 40000; d = 4, n = 4 20.9 -> 8.1 at
// 16.
#pragma once
#include "adj_kernels.cuh"
#include "f64_kernels.cuh"

namespace kgb {

template <int NN, int D> struct AdjF64 {
    static constexpr int N = f64_pow(NN, D), P = NN * NN, R = N / NN;
    static constexpr int VS = (N + 1) / 2 * 2, FS = (D * P + 1) / 2 * 2;
    static constexpr int ES = (D + 1) * VS + FS;  // doubles per entry: p_0 .. p_{D-1}, q, factors
    static constexpr int threads = N <= 1024 ? 256 : N <= 2048 ? 512 : 1024;
    static_assert(N <= 4 * threads, "vector too long");
};

// a.teams_per_cta entries per CTA, at most ROUNDS elements per thread, a.slices lanes (a power
// of two) per contraction item
template <int NN, int D, int ROUNDS>
__global__ void __launch_bounds__(AdjF64<NN, D>::threads, 1024 / AdjF64<NN, D>::threads)
    adj_f64_kernel(const AdjArgs<double> a)
{
    using K = AdjF64<NN, D>;
    constexpr int N = K::N, P = K::P, R = K::R, VS = K::VS, ES = K::ES;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *const base = reinterpret_cast<double *>(smem_raw);
    const int T = blockDim.x, tid = threadIdx.x, E = a.teams_per_cta;
    const long long e0 = (long long)blockIdx.x * E;
    const int ne = a.nb - e0 < E ? (int)(a.nb - e0) : E, total = ne * N;
    const bool want_gA = a.gmats != nullptr, want_gin = a.gin != nullptr;
#pragma unroll
    for (int j = 0; j < ROUNDS; ++j) {
        const int q = tid + j * T;
        if (q < total) {
            const int en = q / N, p = q % N;
            double *const s = base + en * ES + p;
            if (want_gA) cp_async<8>(s + (D - 1) * VS, a.in[e0 + en] + p);
            cp_async<8>(s + D * VS, a.gout[e0 + en] + p);
        }
    }
#pragma unroll 4
    for (int f = tid; f < ne * D * P; f += T) {
        const int en = f / (D * P), m = f % (D * P), el = m % P;
        cp_async<8>(base + en * ES + (D + 1) * VS + m, a.mats[(e0 + en) * D + m / P] + el % NN + (size_t)(el / NN) * a.stride);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (want_gA) {
#pragma unroll
        for (int i = D - 1; i >= 1; --i) {
#pragma unroll
            for (int j = 0; j < ROUNDS; ++j) {
                const int q = tid + j * T;
                if (q < total) {
                    const int en = q / N, p = q % N, c = p / NN, r = p % NN;  // row r of fibre c
                    double *const s = base + en * ES;
                    double x[NN];
                    load_fibre<double, NN>(s + i * VS + c * NN, x);
                    const double *const A = s + (D + 1) * VS + i * P + r;
                    double y = 0.0;
#pragma unroll
                    for (int k = 0; k < NN; ++k) y = fma(A[k * NN], x[k], y);
                    s[(i - 1) * VS + c + r * R] = y;
                }
            }
            __syncthreads();
        }
    }
    const int S = a.slices;
    constexpr int kChains = R >= 16 ? 4 : R >= 8 ? 2 : 1;
    double z[ROUNDS];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        if (want_gA) {
            const int items = ne * P * S;
            for (int w0 = tid - tid % 32; w0 < items; w0 += T) {  // whole warps: they shuffle
                const int w = w0 + tid % 32, sl = w % S, pr = w / S;
                const int en = pr / P, el = pr % P, r = el % NN, k = el / NN;
                double sum = 0.0;
                if (w < items) {
                    const double *const s = base + en * ES;
                    const double *const q = s + D * VS + R * r, *const p = s + i * VS + k;
                    // at least kChains chains of additions, as the kernels that sum in slices have (d = 3,
                    // n = 6: error 2.75e-16 with two, 2.62e-16 with four)
                    if (S == 1) {
                        double part[kChains] = {};
#pragma unroll 2
                        for (int t = 0; t + kChains <= R; t += kChains) {
#pragma unroll
                            for (int c = 0; c < kChains; ++c) part[c] = fma(q[t + c], p[NN * (t + c)], part[c]);
                        }
#pragma unroll
                        for (int c = 0; c < R % kChains; ++c) part[c] = fma(q[R / kChains * kChains + c], p[NN * (R / kChains * kChains + c)], part[c]);
#pragma unroll
                        for (int h = kChains / 2; h > 0; h /= 2)
#pragma unroll
                            for (int c = 0; c < h; ++c) part[c] += part[c + h];
                        sum = part[0];
                    } else if (S == 2 && kChains == 4) {
                        double odd = 0.0;
#pragma unroll 4
                        for (int t = sl; t < R; t += 4) {
                            sum = fma(q[t], p[NN * t], sum);
                            if (t + 2 < R) odd = fma(q[t + 2], p[NN * (t + 2)], odd);
                        }
                        sum += odd;
                    } else {
#pragma unroll 4
                        for (int t = sl; t < R; t += S) sum = fma(q[t], p[NN * t], sum);
                    }
                }
                for (int o = S / 2; o > 0; o /= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (w < items && sl == 0) {
                    double *const g = a.gmats[(e0 + en) * D + i];
                    if (g != nullptr) atomic_add<double>(g + r + (size_t)k * a.gstride, sum);
                }
            }
        }
        if (i + 1 < D || want_gin) {
#pragma unroll
            for (int j = 0; j < ROUNDS; ++j) {
                const int q = tid + j * T;
                if (q < total) {
                    const int en = q / N, p = q % N, t = p / NN, r = p % NN;
                    const double *const s = base + en * ES;
                    const double *const A = s + (D + 1) * VS + i * P + r * NN, *const Q = s + D * VS + t;
                    double y = 0.0;
#pragma unroll
                    for (int k = 0; k < NN; ++k) y = fma(A[k], Q[R * k], y);
                    z[j] = y;
                }
            }
        }
        if (i + 1 < D) {
            __syncthreads();
#pragma unroll
            for (int j = 0; j < ROUNDS; ++j) {
                const int q = tid + j * T;
                if (q < total) base[q / N * ES + D * VS + q % N] = z[j];
            }
            __syncthreads();
        } else if (want_gin) {
#pragma unroll
            for (int j = 0; j < ROUNDS; ++j) {
                const int q = tid + j * T;
                if (q < total) atomic_add<double>(a.gin[e0 + q / N] + q % N, z[j]);
            }
        }
    }
}

struct AdjF64Info {
    const void *fn[3] = {};  // at most 1, 2 and 4 elements per thread (null: fewer than n^d per CTA)
    int n = 0, d = 0;  // of the instantiation
    int threads = 0, entry_bytes = 0;
};
AdjF64Info adj_f64_lookup(int n, int d);  // fn[2] == nullptr where there is no instantiation

}  // namespace kgb
