// FP32 vectors beyond shared memory, n known at compile time: two passes through the
// workspace, both in register blocks.
//
// Pass 1 (fwd_block_kernel, UNITS) applies the fastest d - D2 axes to every chunk of
// n^(d-D2) consecutive values and stores it to the workspace.  Pass 2 (here) applies the
// last D2 axes: the n^D2 values that share a fast position lie C = n^(d-D2) apart, one lane
// holds them all in registers, and a warp's lanes take 32 consecutive positions, so that
// every row it reads and every row it adds to is 128 contiguous bytes.  Warps work alone
// (no barrier across warps): a warp's next tile of n^D2 rows and its factors are copied
// (cp.async, two slots) while the current one is computed, and run sums stay in tensor
// memory until the output or the tile changes.
//
// Against one mode per shared-memory round trip in both passes (split_kernels.cuh): n = 8,
// d = 6, 3905 entries 4954 -> 2746 us, 20 -> 36 TFLOP/s; pass 1 takes two thirds of it.
// Neither pass is at a limit of the memory (4.2-4.5 TB/s, workspace included) or of the FMA
// pipe (48 %): 64 values per thread leave 12 warps per SM to cover the waits for the copies,
// the shared-memory round trips between the two parts of pass 1 and their barriers.
#pragma once
#include "block_kernels.cuh"

namespace kgb {

// axes of pass 2, by n: at most 64 values per lane
constexpr int col_axes(int n) { return n == 2 ? 6 : n <= 4 ? 3 : 2; }

template <int NN> struct Col {
    static constexpr int D2 = col_axes(NN), V = blk_pow(NN, D2), P = NN * NN, P4 = (P + 3) / 4 * 4;
    static constexpr int warps = 4, threads = 32 * warps, ctas = V > 40 ? 3 : 4;
    static constexpr int SLOT = 32 * V + D2 * P4;  // floats per warp and slot
    static constexpr int smem = warps * 2 * SLOT * (int)sizeof(float);
    // entries in one FP32 run sum: a warp's share in one chain of additions (270 entries) made
    // the error of n = 8, d = 6, 781 entries per output 3.1e-7 normwise, with this cap 2.1e-7
    static constexpr int run_max = 32;
    static constexpr int cols = V <= 32 ? 32 : 64;
};

template <int NN, int ST = 1> __device__ __forceinline__ void col_modes(float (&x)[Col<NN>::V], unsigned fac)
{
    if constexpr (ST < Col<NN>::V) {
        constexpr int NF = Col<NN>::V / NN, GB = NN == 2 ? 8 : NN == 4 ? 16 : NF;
        blk_mode<NN, Col<NN>::V, ST, GB>(x, fac);
        col_modes<NN, ST * NN>(x, fac - 4u * Col<NN>::P4);
    }
}

// A warp's work: chunks [first, first of the next warp) of a.chunks, chunk c being
// entries [c % cpt * chunk_len, + chunk_len) of tile c / cpt; FP64 outputs: run sums (in
// FP32) are cut at chunk edges.
template <typename TO, int NN>
__global__ void __launch_bounds__(Col<NN>::threads, Col<NN>::ctas) fwd_column_kernel(const FwdArgs<float, TO> a)
{
    using K = Col<NN>;
    constexpr int V = K::V, P = K::P, D2 = K::D2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_tmem;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *const base = reinterpret_cast<float *>(smem_raw) + warp * 2 * K::SLOT;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (unsigned)__cvta_generic_to_shared(&s_tmem)),
                     "n"(K::cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = s_tmem + ((unsigned)warp << 21);

    const int C = a.split_C, nb = (int)a.nb, len = a.chunk_len, cpt = (nb + len - 1) / len;
    const int g = blockIdx.x * K::warps + warp, share = a.entries_per_team;
    const int more = (int)a.chunks - share * (int)(gridDim.x * K::warps);
    struct Spot {  // an entry of a tile; `end`: where its chunk ends
        int c, tile, e, end;
    };
    const int c_end = (g + 1) * share + (g + 1 < more ? g + 1 : more);
    auto step = [&](Spot s) {
        if (++s.e == s.end && ++s.c < c_end) {
            if (s.e == nb) s.e = 0, ++s.tile;
            s.end = s.e + len < nb ? s.e + len : nb;
        }
        return s;
    };
    // lane 0: the workspace, 1: the output, 2 + i: factor i
    auto load_ptr = [&](const Spot &s) {
        unsigned long long p = 0;
        if (s.c < c_end) {
            if (lane == 0) p = (unsigned long long)reinterpret_cast<uintptr_t>(a.ws[s.e]);
            if (lane == 1) p = (unsigned long long)reinterpret_cast<uintptr_t>(a.out[s.e]);
            if (lane >= 2 && lane < 2 + D2)
                p = (unsigned long long)reinterpret_cast<uintptr_t>(a.mats[(size_t)s.e * a.d + (lane - 2)]);
        }
        return p;
    };
    const bool rows16 = C % 4 == 0;
    auto copy = [&](int slot, const Spot &s, unsigned long long ptr) {
        float *const X = base + slot * K::SLOT, *const F = X + 32 * V;
        const float *const src =
            reinterpret_cast<const float *>(__shfl_sync(0xffffffffu, ptr, 0)) + s.tile * 32;
        const int left = C - s.tile * 32;  // columns of the tile, if fewer than 32
        if (rows16 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
            const int j = lane % 8 * 4;
            if (j < left) {
#pragma unroll
                for (int h = 0; h < V; h += 4)
                    if (V % 4 == 0 || h + lane / 8 < V)
                        cp_async<16>(X + (h + lane / 8) * 32 + j, src + (size_t)(h + lane / 8) * C + j);
            }
        } else if (lane < left) {
#pragma unroll 8
            for (int h = 0; h < V; ++h) cp_async<4>(X + h * 32 + lane, src + (size_t)h * C + lane);
        }
#pragma unroll
        for (int j0 = 0; j0 < D2 * P; j0 += 32) {
            const int j = j0 + lane, i = j < D2 * P ? j / P : 0, el = j - i * P;
            const float *const m = reinterpret_cast<const float *>(__shfl_sync(0xffffffffu, ptr, 2 + i));
            if (j < D2 * P) cp_async<4>(F + i * K::P4 + el, m + el % NN + (size_t)(el / NN) * a.stride);
        }
        cp_async_commit();
    };

    Spot cur;
    cur.c = g * share + (g < more ? g : more);
    cur.tile = cur.c / cpt;
    cur.e = (cur.c - cur.tile * cpt) * len;
    cur.end = cur.e + len < nb ? cur.e + len : nb;
    if (cur.c < c_end) {
        unsigned long long ptr = load_ptr(cur);
        TO *o = reinterpret_cast<TO *>(__shfl_sync(0xffffffffu, ptr, 1));
        copy(0, cur, ptr);
        Spot next = step(cur);
        ptr = load_ptr(next);
        int slot = 0;
        int run = 0;  // entries in the current sum
        while (true) {
            const bool have = next.c < c_end;
            cp_async_wait_all();
            __syncwarp();  // this tile complete, the other slot's reads done
            TO *const o_next = reinterpret_cast<TO *>(__shfl_sync(0xffffffffu, ptr, 1));
            const Spot now = cur;
            if (have) {
                copy(slot ^ 1, next, ptr);
                cur = next;
                next = step(next);
                ptr = load_ptr(next);
            }
            const bool fresh = run == 0;
            const bool last = !have || o_next != o || cur.tile != now.tile ||
                              (sizeof(TO) == 8 ? cur.c != now.c : run + 1 == K::run_max);
            const float *const X = base + slot * K::SLOT;
            float x[V];
#pragma unroll
            for (int h = 0; h < V; ++h) x[h] = X[h * 32 + lane];
            col_modes<NN>(x, (unsigned)__cvta_generic_to_shared(X + 32 * V + (D2 - 1) * K::P4));
            if (!fresh) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                blk_tm_add<V>(tmem, x, false, false);
            }
            if (last) {
                if (now.tile * 32 + lane < C) {
                    TO *const p = o + now.tile * 32 + lane;
#pragma unroll
                    for (int h = 0; h < V; ++h) atomic_add<TO>(p + (size_t)h * C, blk_out<TO>(x[h]));
                }
                __syncwarp();
            } else {
                blk_tm_st<V>(tmem, x);
            }
            if (!have) break;
            run = last ? 0 : run + 1;
            o = o_next;
            slot ^= 1;
        }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "n"(K::cols) : "memory");
    }
}

struct ColInfo {
    const void *fn = nullptr;
    int block = 0, smem = 0, cols = 0;
};
// fn == nullptr where there is no instantiation
template <typename TO> ColInfo col_lookup(int n);
BlkInfo units_lookup(int n, int d1);

}  // namespace kgb
