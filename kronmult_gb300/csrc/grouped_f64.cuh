// Deterministic FP64 groups of short vectors (grouped.cuh has the units, runs and partial
// slots): the short vectors' forward (f64_kernels.cuh) over the sorted entries, one unit per
// CTA in steps of E entries.
//
// After a step's last mode its results lie in shared memory, and the entries of a run are added
// to the output (or to the run's partial slot, which the first one stores) in entry order by one
// thread per element, with additions in L2: no FP64-pipe instruction for the sums.  Steps of a
// unit are ordered by barriers.
//
// Against the persistent kernels (run sums in L2 as well): d = 6, n = 3, 56340 entries 1412 -> 1371
// us, d = 3, n = 6, 83871 630 -> 583, d = 2, n = 2, 120000 66 -> 17; bound by the FP64 pipe (84-90 %)
// but for the last wave and the partial sums of runs that cross units.
#pragma once
#include "f64_kernels.cuh"
#include "grouped.cuh"

namespace kgb {

// a.team_elems: entries per step (E); a.unit a multiple of it
template <int NN, int D, int R>
__global__ void __launch_bounds__(F64<NN, D>::threads, 1024 / F64<NN, D>::threads) gq_f64_det_kernel(const GqArgs a)
{
    using K = F64<NN, D>;
    constexpr int N = K::N, P = K::P, F = K::F;
    constexpr bool kOwn = N >= 128;  // threads own positions over all entries, else over one run
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int T = blockDim.x, tid = threadIdx.x, E = a.team_elems;
    double *const X = reinterpret_cast<double *>(smem_raw), *const M = X + E * K::VS;
    double **const dst = reinterpret_cast<double **>(M + E * K::FS);  // where each entry is added
    unsigned char *const head = reinterpret_cast<unsigned char *>(dst + E);  // 1: first of its run in this step; 2: stored
    const double *const *const mats = reinterpret_cast<const double *const *>(a.mats);
    const double *const *const in = reinterpret_cast<const double *const *>(a.in);
    const long long u = blockIdx.x, b = u * a.unit, e = b + a.unit < a.nb ? b + a.unit : a.nb;
    const unsigned long long before = b > 0 ? a.keys[b - 1] : 0, after = e < a.nb ? a.keys[e] : 0;
    double *const slots = static_cast<double *>(a.partial) + 2 * u * N;
#pragma unroll 1
    for (long long e0 = b; e0 < e; e0 += E) {
        const int ne = e - e0 < E ? (int)(e - e0) : E, total = ne * N;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int q = tid + j * T;
            if (q < total) cp_async<8>(X + q / N * K::VS + q % N, in[e0 + q / N] + q % N);
        }
#pragma unroll 4
        for (int f = tid; f < ne * K::FS; f += T) {
            const int m = f / P, el = f % P;
            cp_async<8>(M + f, mats[e0 * D + m] + el % NN + (size_t)(el / NN) * a.stride);
        }
        cp_async_commit();
        for (int en = tid; en < ne; en += T) {
            const unsigned long long key = a.keys[e0 + en];
            const bool first = e0 + en == b || a.keys[e0 + en - 1] != key, low = key == before, high = key == after;
            dst[en] = low ? slots : high ? slots + N : reinterpret_cast<double *>(static_cast<uintptr_t>(key));
            head[en] = (first || en == 0 ? 1 : 0) | (first && (low || high) ? 2 : 0);
        }
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
            __syncthreads();
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const int q = tid + j * T;
                if (q < total) X[q / N * K::VS + q % N / NN + q % N % NN * F] = y[j];
            }
            __syncthreads();
        }
        if constexpr (kOwn) {
            for (int p = tid; p < N; p += T) {
                for (int en = 0; en < ne; ++en) {
                    const double v = X[en * K::VS + p];
                    if (head[en] & 2)
                        dst[en][p] = v;
                    else
                        atomic_add<double>(dst[en] + p, v);
                }
            }
        } else {
#pragma unroll 1
            for (int q = tid; q < total; q += T) {
                int en = q / N;
                if (!(head[en] & 1)) continue;
                double *const o = dst[en] + q % N;
                if (head[en] & 2)
                    *o = X[en * K::VS + q % N];
                else
                    atomic_add<double>(o, X[en * K::VS + q % N]);
                for (++en; en < ne && !(head[en] & 1); ++en) atomic_add<double>(o, X[en * K::VS + q % N]);
            }
        }
        __syncthreads();
    }
}

struct GqF64Info {
    GqFn fn[3] = {};  // at most 1, 2 and 4 elements per thread (null: fewer than n^d per CTA)
    int n = 0, d = 0;  // of the instantiation
    int threads = 0, entry_bytes = 0;
};
GqF64Info gq_f64_lookup(int n, int d);  // fn[2] == nullptr where there is no instantiation

}  // namespace kgb
