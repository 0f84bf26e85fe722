// FP32 forward in register blocks, n and d known at compile time.
//
// The vector stays in its natural order in shared memory and every mode is applied in
// place along its own axis (no index rotation), so all shared-memory offsets are
// immediates.  The d axes are taken in passes of M axes from the fastest one: in a pass a
// thread owns blocks of n^M values (one fibre per axis of the pass through every value),
// loads them, applies the pass's modes in registers and stores them where they came from.
// Only the thread itself touches those positions, so a pass needs one barrier, after its
// stores.  The last pass adds into the run sums instead of storing.  Each output is the
// same k-ascending FMA chain, in the same mode order, as the one-mode-per-step kernels':
// bitwise the same value per entry.
//
// What bounds it: the register-file side of shared memory.  A load moves 128 bytes per
// cycle into registers, and a thread reads the n x n factor of a mode once per batch of
// fibres it holds, so a factor value has to meet as many fibres as the registers can hold.
// Hence whole blocks per thread with all their fibres in one batch (GB), two blocks per
// thread (G) where n is small (in packed FP32 pairs, the factor value duplicated in
// registers), and the run sums of entries with one output kept in tensor memory, which
// FP32 kernels leave idle, instead of V more registers per thread.
//
// E entries of T = ceil(n^(d-M) / G) threads share a CTA: n = 3, 5, 6, 7, 9, 10 leave no
// power-of-two teams, and whole-CTA teams of E * T threads keep 84-99 % of the lanes busy.
// Two slots per entry: the next entry's vector and factors are copied (cp.async) while the
// current one is computed, from pointers that were themselves copied one entry earlier.
//
// Bank conflicts: in the pass over the fastest axes consecutive threads own consecutive
// blocks and read them with the widest loads whose stride in load units is odd (blocks are
// padded to make it so where n^M is a multiple of 8); in the other passes consecutive
// threads own consecutive positions.
//
// Measured against the kernels that apply one mode (n = 2, 4, 8: two) per shared-memory pass,
// FP32: d = 4, n = 5, 35007 entries 89.6 -> 46.4 us (DRAM sectors 67 % of peak at a stride of
// 67); d = 6, n = 4, 36864 entries 207 -> 200 us; d = 2, n = 3, 200000 entries 34.9 -> 19.8; d = 3,
// n = 6, 200000 entries 160 -> 100; FP64 outputs, d = 4, n = 8, 32768 entries 268 -> 219 us.  With
// 64 values per thread (168 registers, 12 warps per SM) the FMA pipe is 45-56 % busy and DRAM
// 45-54 %: register-port conflicts stall dispatch for about a quarter of the cycles.
#pragma once
#include <type_traits>
#include "fwd_kernels.cuh"

namespace kgb {

// tensor memory is allocated in powers of two of at least 32 columns
constexpr int tmem_cols(int used) { return used <= 32 ? 32 : used <= 64 ? 64 : used <= 128 ? 128 : used <= 256 ? 256 : 512; }

constexpr int blk_pow(int b, int e) { return e <= 0 ? 1 : b * blk_pow(b, e - 1); }

// One way to run (n, d): axes per pass (M), blocks per thread (G: 1, or 2 in packed pairs),
// fibres (or fibre pairs) whose outputs are held at once (GB), warps per group (W), groups
// per CTA (C) and CTAs per SM.
template <int NN_, int D_, int M_, int G_, int GB_, int W_, int C_, int CTAS_> struct BlkCfg {
    static constexpr int NN = NN_, D = D_, M = M_, G = G_, GB = GB_, W = W_, C = C_, ctas = CTAS_;
};

// Batches that fill the GPU: whole blocks of two or three axes per thread.
template <int NN, int D> struct BlkLarge;
template <int D> struct BlkLarge<2, D> : BlkCfg<2, D, (D <= 5 ? 3 : 4), 1, (D <= 5 ? 4 : 8), 1, 4, 8> {};
template <int D> struct BlkLarge<3, D> : BlkCfg<3, D, (D >= 5 ? 3 : 2), (D == 6 ? 2 : 1), (D >= 5 ? 9 : 3), 1, 4, (D == 6 ? 3 : D >= 7 ? 4 : D == 5 ? 5 : 8)> {};
template <int D> struct BlkLarge<4, D> : BlkCfg<4, D, (D >= 5 ? 3 : D == 2 ? 1 : 2), 1, (D == 6 ? 8 : D >= 5 ? 16 : D == 2 ? 1 : 4), 1, (D == 6 ? 2 : 4), (D == 6 ? 6 : D >= 5 ? 3 : 8)> {};
template <int D> struct BlkLarge<5, D> : BlkCfg<5, D, (D == 2 ? 1 : 2), (D == 5 ? 2 : 1), (D == 2 ? 1 : 5), 1, 4, (D == 2 ? 8 : D == 3 ? 4 : D == 4 ? 5 : 3)> {};
template <int D> struct BlkLarge<6, D> : BlkCfg<6, D, (D == 2 ? 1 : 2), 1, (D == 2 ? 1 : 6), (D >= 4 ? 8 : 1), (D >= 4 ? 1 : 4), (D >= 4 ? 2 : D == 2 ? 8 : 4)> {};
template <int D> struct BlkLarge<7, D> : BlkCfg<7, D, (D == 2 ? 1 : 2), 1, (D == 2 ? 1 : 7), (D == 4 ? 8 : 1), (D == 4 ? 1 : 4), (D == 4 ? 2 : D == 2 ? 8 : 4)> {};
template <int D> struct BlkLarge<8, D> : BlkCfg<8, D, (D == 2 ? 1 : 2), 1, (D == 2 ? 1 : 8), 1, (D == 4 ? 2 : 4), (D == 2 || D == 4 ? 6 : 3)> {};
template <int D> struct BlkLarge<9, D> : BlkCfg<9, D, (D <= 2 ? 1 : 2), 1, (D <= 2 ? 1 : D == 3 ? 5 : 3), 1, (D == 4 ? 3 : 4), (D <= 2 ? 4 : D == 3 ? 2 : 3)> {};
template <int D> struct BlkLarge<10, D> : BlkCfg<10, D, (D <= 2 ? 1 : 2), 1, (D <= 2 ? 1 : 5), 1, 4, (D <= 2 ? 4 : 2)> {};
// Small batches, where latency counts: one fibre per thread (n = 4: one pair of axes).
template <int NN, int D>
struct BlkSmall : BlkCfg<NN, D, (NN == 4 ? 2 : 1), 1, (NN == 4 ? 4 : 1), 1, 4, (NN >= 9 ? 4 : NN == 8 ? 6 : 8)> {};

template <typename Tn> struct Blk {
    static constexpr int NN = Tn::NN, D = Tn::D;
    static constexpr int N = blk_pow(NN, D);
    static constexpr int M = Tn::M < D ? Tn::M : D;
    static constexpr int V0 = blk_pow(NN, M);                    // values per block
    static constexpr int G = M < D ? Tn::G : 1;                  // blocks per thread
    static constexpr int V = V0 * G;                             // values per thread
    static constexpr int T = (N / V0 + G - 1) / G;               // threads per entry
    static constexpr int W = T > 32 * Tn::W ? (T + 31) / 32 : Tn::W;  // warps per group
    static constexpr int EW = 32 * W / T < 32 ? 32 * W / T : 32;      // entries per group
    static constexpr int C = Tn::W * Tn::C >= W ? Tn::W * Tn::C / W : 1;  // groups per CTA
    static constexpr int threads = 32 * W * C;
    static constexpr int ctas = Tn::W * Tn::C >= W ? Tn::ctas : 1;
    static constexpr int LW = V0 % 4 == 0 ? 4 : (V0 % 2 == 0 ? 2 : 1);  // floats per load in the first pass
    static constexpr int VP = (V0 / LW) % 2 == 0 ? V0 + LW : V0;        // padded block
    static constexpr bool copy16 = N % 4 == 0 && (LW == 4 || VP == V0);  // whole 16-byte chunks
    // odd n: a vector starts (address / 4) mod 4 floats into its slot, so that its 16-byte
    // chunks are copied whole; single-pass vectors (one thread each) are copied by value
    static constexpr bool shifted = NN % 2 == 1 && T > 1;
    // floats per vector slot; the entries of a group a multiple of about T banks apart, so
    // that their threads share the banks in the strided passes
    static constexpr int vs_min = copy16 || shifted ? (shifted ? (N + 6) / 4 * 4 : (N / V0 * VP + 3) / 4 * 4) : N / V0 * VP;
    static constexpr int vs_mod = (T + 3) / 4 * 4;
    static constexpr int VS = T > 1 && EW > 1 ? vs_min + ((vs_mod - vs_min) % 32 + 32) % 32 : vs_min;
    static constexpr int P4 = 4 * ((NN * NN + 3) / 4);                      // one staged factor
    static constexpr int FS = D * P4 / 4 % 2 == 0 ? D * P4 + 4 : D * P4;    // an entry's factors
    static constexpr int SLOT = (EW * VS + 3) / 4 * 4 + EW * FS;            // floats per staging slot of a group
    static constexpr int passes = (D + M - 1) / M;
    // tensor-memory columns of run sums: V per group of four warps
    static constexpr int cols_used = V * ((threads + 127) / 128);
    static_assert(cols_used <= 512, "tensor memory");
    // FP32 outputs: a second level of run sums, where all resident CTAs have room for it
    template <typename TO>
    static constexpr bool two_levels = sizeof(TO) == 4 && 2 * cols_used <= 512 && tmem_cols(2 * cols_used) * ctas <= 512;
    // batches of several waves of CTAs (plan_block)
    template <typename TO> static constexpr bool guided = sizeof(TO) == 8 ? T > 8 : T >= 8 && !two_levels<TO> && N <= 4096;
    template <typename TO> static constexpr int cols = tmem_cols(two_levels<TO> ? 2 * cols_used : cols_used);
    static_assert(C <= 15 || W == 1, "named barriers");
    static __host__ __device__ constexpr int phys(int p) { return VP == V0 ? p : p / V0 * VP + p % V0; }
    using X = std::conditional_t<G == 2, f2, float>;  // one value, or the same value of two blocks
};

// barrier of a group (its warps are consecutive)
template <int W, int C> __device__ __forceinline__ void blk_sync(int group)
{
    if constexpr (W == 1)
        __syncwarp();
    else if constexpr (C == 1)
        __syncthreads();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(32 * W) : "memory");
}

// 16 bytes of a factor at shared-memory address s (volatile: read again by the next batch
// of fibres, not kept in registers)
__device__ __forceinline__ void blk_ld_factor(unsigned s, float *m)
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(m[0]), "=f"(m[1]), "=f"(m[2]), "=f"(m[3])
                 : "r"(s));
}
__device__ __forceinline__ float blk_fma(float m, float x, float y) { return fmaf(m, x, y); }
__device__ __forceinline__ f2 blk_fma(float m, f2 x, f2 y) { return f2_fma(f2_pack(m, m), x, y); }
__device__ __forceinline__ float blk_zero(float) { return 0.f; }
__device__ __forceinline__ f2 blk_zero(f2) { return f2_pack(0.f, 0.f); }

// mode product on the axis of stride ST of a thread's values, in place: fibre f's element
// k is x[(f / ST) * ST * NN + f % ST + k * ST].  `fac`: shared address of the factor.
template <int NN, int NX, int ST, int GB, typename X>
__device__ __forceinline__ void blk_mode(X (&x)[NX], unsigned fac)
{
    constexpr int NF = NX / NN, P4 = (NN * NN + 3) / 4 * 4;
#pragma unroll
    for (int f0 = 0; f0 < NF; f0 += GB) {
        X y[GB][NN];
        float m[P4];
#pragma unroll
        for (int k = 0; k < NN; ++k) {
#pragma unroll
            for (int r = 0; r < NN; ++r) {
                const int j = k * NN + r;
                if (j % 4 == 0) blk_ld_factor(fac + 4u * j, m + j);
            }
#pragma unroll
            for (int g = 0; g < GB; ++g) {
                const int f = f0 + g;
                if (f < NF) {
                    const X xk = x[f / ST * ST * NN + f % ST + k * ST];
#pragma unroll
                    for (int rr = 0; rr < NN; ++rr) {
                        // there and back: the factor value at a turn meets two values in a row
                        // (fewer register-port conflicts: d = 3, n = 6 106 -> 100 us, d = 4,
                        // n = 8 103 -> 101, no shape slower)
                        const int r = g % 2 ? NN - 1 - rr : rr;
                        y[g][r] = blk_fma(m[k * NN + r], xk, k == 0 ? blk_zero(xk) : y[g][r]);
                    }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < GB; ++g) {
            const int f = f0 + g;
            if (f < NF) {
#pragma unroll
                for (int r = 0; r < NN; ++r) x[f / ST * ST * NN + f % ST + r * ST] = y[g][r];
            }
        }
    }
}

// Pass P over axes [D - first - axes, D - first): blocks of NB = n^axes values, step apart,
// G * V0 / NB of them per thread.
template <typename CF, int P> struct BlkPass {
    using B = Blk<CF>;
    static constexpr int NN = CF::NN, D = CF::D;
    static constexpr int first = P * B::M;                            // axes below the pass
    static constexpr int axes = D - first < B::M ? D - first : B::M;  // axes of the pass
    static constexpr int NB = blk_pow(NN, axes);
    static constexpr int NG = B::V / NB;   // blocks per thread
    static constexpr int NH = NG / B::G;   // blocks (G = 1) or pairs of blocks (G = 2) per thread
    static constexpr int items = B::N / NB;
    static constexpr int Q = blk_pow(NN, first);
    static constexpr int step = P == 0 ? 1 : B::phys(Q);  // p > 0: Q is a multiple of V0 wherever blocks are padded
    static_assert(B::VP == B::V0 || P == 0 || Q % B::V0 == 0, "padded blocks stay whole");
    // whether block i exists for every thread, and for thread t
    static constexpr bool whole(int i) { return B::T * (i + 1) <= items; }
    static __host__ __device__ __forceinline__ bool has(int t, int i) { return whole(i) || t + B::T * i < items; }
    // position of block i of thread t in the staged layout (a block that does not exist:
    // the last one, which is then only read)
    static __host__ __device__ __forceinline__ int base(int t, int i)
    {
        int idx = t + B::T * i;
        if (!whole(i) && idx >= items) idx = items - 1;
        if constexpr (P == 0) {
            return idx * B::VP;
        } else if constexpr (items == Q) {
            return B::VP == B::V0 || Q == B::V0 ? idx : B::phys(idx);
        } else if constexpr (B::T % Q == 0 && B::T * NG == items) {
            return B::phys(t / Q * NB * Q + t % Q) + i * B::phys(B::T / Q * NB * Q);
        } else {
            return B::phys(idx / Q * NB * Q + idx % Q);
        }
    }
};

// NB values of one block between shared memory and v (contiguous for P = 0: wide accesses)
template <int NB, int LW, int STEP> __device__ __forceinline__ void blk_load(const float *p, float (&v)[NB])
{
#pragma unroll
    for (int j = 0; j < NB; j += LW) {
        if constexpr (LW == 4) {
            const float4 u = *reinterpret_cast<const float4 *>(p + j);
            v[j] = u.x, v[j + 1] = u.y, v[j + 2] = u.z, v[j + 3] = u.w;
        } else if constexpr (LW == 2) {
            const float2 u = *reinterpret_cast<const float2 *>(p + j);
            v[j] = u.x, v[j + 1] = u.y;
        } else {
            v[j] = p[j * STEP];
        }
    }
}
template <int NB, int LW, int STEP> __device__ __forceinline__ void blk_store(float *p, const float (&v)[NB])
{
#pragma unroll
    for (int j = 0; j < NB; j += LW) {
        if constexpr (LW == 4)
            *reinterpret_cast<float4 *>(p + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        else if constexpr (LW == 2)
            *reinterpret_cast<float2 *>(p + j) = make_float2(v[j], v[j + 1]);
        else
            p[j * STEP] = v[j];
    }
}

__device__ __forceinline__ void blk_split(float x, float &lo, float &) { lo = x; }
__device__ __forceinline__ void blk_split(f2 x, float &lo, float &hi) { f2_unpack(x, lo, hi); }

// One pass's values between shared memory and registers: x[ib * NB + m] is value m of block
// ib (and of block ib + NH).
template <typename CF, int P>
__device__ __forceinline__ void blk_load_pass(typename Blk<CF>::X (&x)[Blk<CF>::V0], const float *vec, int t)
{
    using B = Blk<CF>;
    using W = BlkPass<CF, P>;
    constexpr int NB = W::NB, LW = P == 0 ? B::LW : 1;
#pragma unroll
    for (int ib = 0; ib < W::NH; ++ib) {
        float lo[NB];
        blk_load<NB, LW, W::step>(vec + W::base(t, ib), lo);
        if constexpr (B::G == 2) {
            float hi[NB];
            blk_load<NB, LW, W::step>(vec + W::base(t, ib + W::NH), hi);
#pragma unroll
            for (int m = 0; m < NB; ++m) x[ib * NB + m] = f2_pack(lo[m], hi[m]);
        } else {
#pragma unroll
            for (int m = 0; m < NB; ++m) x[ib * NB + m] = lo[m];
        }
    }
}
template <typename CF, int P>
__device__ __forceinline__ void blk_store_pass(const typename Blk<CF>::X (&x)[Blk<CF>::V0], float *vec, int t)
{
    using B = Blk<CF>;
    using W = BlkPass<CF, P>;
    constexpr int NB = W::NB, LW = P == 0 ? B::LW : 1;
#pragma unroll
    for (int ib = 0; ib < W::NH; ++ib) {
        float lo[NB], hi[NB];
#pragma unroll
        for (int m = 0; m < NB; ++m) blk_split(x[ib * NB + m], lo[m], hi[m]);
        if (W::has(t, ib)) blk_store<NB, LW, W::step>(vec + W::base(t, ib), lo);
        if constexpr (B::G == 2) {
            if (W::has(t, ib + W::NH)) blk_store<NB, LW, W::step>(vec + W::base(t, ib + W::NH), hi);
        }
    }
}
// AXES modes, the first on the block's fastest axis; `fac`: the first mode's factor, the
// following ones P4 floats below
template <typename CF, int AXES>
__device__ __forceinline__ void blk_modes(typename Blk<CF>::X (&x)[Blk<CF>::V0], unsigned fac)
{
    using B = Blk<CF>;
    constexpr int GB = CF::GB, NN = CF::NN;
    blk_mode<NN, B::V0, 1, GB>(x, fac);
    if constexpr (AXES > 1) blk_mode<NN, B::V0, NN, GB>(x, fac - 4u * B::P4);
    if constexpr (AXES > 2) blk_mode<NN, B::V0, NN * NN, GB>(x, fac - 8u * B::P4);
    if constexpr (AXES > 3) blk_mode<NN, B::V0, NN * NN * NN, GB>(x, fac - 12u * B::P4);
    if constexpr (AXES > 4) blk_mode<NN, B::V0, NN * NN * NN * NN, GB>(x, fac - 16u * B::P4);
}

// Passes P .. of one entry; the last one's results stay in x.  Threads without work (t
// beyond the entry's, or no entry) compute on whatever lies in their slot and store
// nothing.
template <typename CF, int P>
__device__ __forceinline__ void blk_passes(typename Blk<CF>::X (&x)[Blk<CF>::V0], float *vec, unsigned fac, int t,
                                           bool active, int group)
{
    using B = Blk<CF>;
    using W = BlkPass<CF, P>;
    constexpr int D = CF::D;
    constexpr int top = D - 1 - W::first;
    if constexpr (P == 0 && D == 2 * B::M && B::V0 >= 49) {
        // two like passes: one copy of the modes' code (a block's modes are 10-40 KB of
        // instructions: unrolled, the passes wait for instruction fetches)
#pragma unroll 1
        for (int p = 0; p < 2; ++p) {
            if (p == 0)
                blk_load_pass<CF, 0>(x, vec, t);
            else
                blk_load_pass<CF, 1>(x, vec, t);
            blk_modes<CF, B::M>(x, fac + 4u * B::P4 * (p == 0 ? D - 1 : B::M - 1));
            if (p == 0) {
                if (active) blk_store_pass<CF, 0>(x, vec, t);
                blk_sync<B::W, B::C>(group);
            }
        }
    } else {
        blk_load_pass<CF, P>(x, vec, t);
        blk_modes<CF, W::axes>(x, fac + 4u * B::P4 * top);
        if constexpr (P + 1 < B::passes) {
            if (active) blk_store_pass<CF, P>(x, vec, t);
            blk_sync<B::W, B::C>(group);
            blk_passes<CF, P + 1>(x, vec, fac, t, active, group);
        }
    }
}

// A sum in the output's type.  FP64: the float's bits moved into place, exactly cvt's result
// for normal floats; the conversion instruction runs on the FP64 pipe, at 2 values per
// clock and SM half as long as the modes of a vector take.
template <typename TO> __device__ __forceinline__ TO blk_out(float v)
{
    if constexpr (sizeof(TO) == 4) {
        return v;
    } else {
        const unsigned u = __float_as_uint(v);
        if ((u & 0x7fffffffu) - 0x00800000u >= 0x7f000000u) return (TO)v;  // zero, subnormal, infinite, NaN
        return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
    }
}

// one vector into its slot by SZ threads of rank `rank` < SZ (asynchronous); vectors of
// B::shifted layouts start blk_shift(src) floats into the slot
__device__ __forceinline__ int blk_shift(const float *src) { return (int)(reinterpret_cast<uintptr_t>(src) >> 2) & 3; }
template <typename B, int SZ> __device__ __forceinline__ void blk_copy_vec(float *dst, const float *src, int rank)
{
    constexpr int N = B::N;
    if constexpr (B::shifted) {
        const int sh = blk_shift(src), end = (N + sh) / 4;
        const float *s0 = src - sh;
#pragma unroll
        for (int i = 0; i < (N / 4 + SZ) / SZ; ++i) {
            const int c = rank + SZ * i;
            if ((c > 0 || sh == 0) && c < end) cp_async<16>(dst + 4 * c, s0 + 4 * c);
        }
        // the values before the first whole chunk and after the last one
        if (rank < 3) {
            if (rank < ((4 - sh) & 3)) cp_async<4>(dst + sh + rank, src + rank);
            if (rank < ((N + sh) & 3)) cp_async<4>(dst + 4 * end + rank, s0 + 4 * end + rank);
        }
    } else if (B::copy16 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
#pragma unroll
        for (int i = 0; i < (N / 4 + SZ - 1) / SZ; ++i) {
            const int c = rank + SZ * i;
            if ((i + 1) * SZ <= N / 4 || c < N / 4) cp_async<16>(dst + B::phys(4 * c), src + 4 * c);
        }
    } else {
#pragma unroll
        for (int i = 0; i < (N + SZ - 1) / SZ; ++i) {
            const int p = rank + SZ * i;
            if ((i + 1) * SZ <= N || p < N) cp_async<4>(dst + B::phys(p), src + p);
        }
    }
}

// Copies the factors of a group's entries: the elements (r, k) of a factor over consecutive
// lanes, PP factors (of PP teams) at a time.
template <typename CF> struct BlkFactorLanes {
    using B = Blk<CF>;
    static constexpr int P = CF::NN * CF::NN, EW = B::EW, W = B::W;
    static constexpr int PP = P >= 32 ? 1 : (32 / P < EW ? 32 / P : EW), RR = (P + 31) / 32;
    int sub, el;
    size_t off[RR];
    __device__ __forceinline__ BlkFactorLanes(int lane, int stride)
    {
        sub = P >= 32 ? 0 : lane / P;
        el = P >= 32 ? lane : lane - sub * P;
#pragma unroll
        for (int h = 0; h < RR; ++h) off[h] = (el + 32 * h) % CF::NN + (size_t)((el + 32 * h) / CF::NN) * stride;
    }
    __device__ __forceinline__ void one(float *dst, const float *m) const
    {
#pragma unroll
        for (int h = 0; h < RR; ++h)
            if (32 * h + 32 <= P || el + 32 * h < P) cp_async<4>(dst + el + 32 * h, m + off[h]);
    }
    // gw: the warp's rank in its group; ptr(i, j): factor i of team j (all lanes call it)
    template <typename F> __device__ __forceinline__ void copy(float *dst, int gw, int ew, F ptr) const
    {
#pragma unroll
        for (int i = 0; i < CF::D; ++i) {
            if constexpr (EW <= PP) {  // the warps of a group share the modes
                if (W == 1 || i % W == gw) {
                    const float *m = ptr(i, sub < EW ? sub : 0);
                    if (sub < EW && m) one(dst + sub * B::FS + i * B::P4, m);
                }
            } else {
#pragma unroll 1
                for (int j0 = gw * PP; j0 < ew; j0 += W * PP) {
                    const int j = j0 + sub;
                    const float *m = ptr(i, j < ew ? j : 0);
                    if (sub < PP && j < ew && m) one(dst + j * B::FS + i * B::P4, m);
                }
            }
        }
    }
};

// ---- run sums in tensor memory: each thread's V values in its own lane --------------

template <int NUM> __device__ __forceinline__ void blk_tm_ld1(unsigned a, float *r)
{
    if constexpr (NUM == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
                       "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]),
                       "=f"(r[15])
                     : "r"(a));
    else if constexpr (NUM == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                     : "r"(a));
    else if constexpr (NUM == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(a));
    else if constexpr (NUM == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=f"(r[0]), "=f"(r[1]) : "r"(a));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=f"(r[0]) : "r"(a));
}
template <int NUM> __device__ __forceinline__ void blk_tm_st1(unsigned a, const float *r)
{
    if constexpr (NUM == 16)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(a),
                     "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]),
                     "f"(r[9]), "f"(r[10]), "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15])
                     : "memory");
    else if constexpr (NUM == 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(a), "f"(r[0]),
                     "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]) : "memory");
    else if constexpr (NUM == 4)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(r[0]), "f"(r[1]),
                     "f"(r[2]), "f"(r[3]) : "memory");
    else if constexpr (NUM == 2)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(a), "f"(r[0]), "f"(r[1]) : "memory");
    else
        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(a), "f"(r[0]) : "memory");
}
constexpr int blk_tm_piece(int left) { return left >= 16 ? 16 : left >= 8 ? 8 : left >= 4 ? 4 : left >= 2 ? 2 : 1; }
template <int NV, int AT = 0> __device__ __forceinline__ void blk_tm_ld(unsigned a, float (&r)[NV])
{
    if constexpr (AT < NV) {
        constexpr int NUM = blk_tm_piece(NV - AT);
        blk_tm_ld1<NUM>(a + AT, r + AT);
        blk_tm_ld<NV, AT + NUM>(a, r);
    }
}
template <int NV, int AT = 0> __device__ __forceinline__ void blk_tm_st(unsigned a, const float (&r)[NV])
{
    if constexpr (AT < NV) {
        constexpr int NUM = blk_tm_piece(NV - AT);
        blk_tm_st1<NUM>(a + AT, r + AT);
        blk_tm_st<NV, AT + NUM>(a, r);
    }
}

// y += the lane's sums (y alone where `fresh`; `mixed`: some lane of the warp is fresh),
// at most 16 sums of 64 in registers at a time (d = 4, n = 8, FP64 outputs, 32768 entries: 242
// -> 234 us; d = 6, n = 4 196.8 -> 195.1), 32 of more
template <int NV, int AT = 0>
__device__ __forceinline__ void blk_tm_add(unsigned a, float (&y)[NV], bool fresh, bool mixed)
{
    if constexpr (AT < NV) {
        constexpr int CH0 = NV < 64 ? NV : NV == 64 ? 16 : 32, CH = NV - AT < CH0 ? NV - AT : CH0;
        float s[CH];
        blk_tm_ld<CH>(a + AT, s);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < CH; ++j) asm volatile("" : "+f"(s[j]));  // no use before the wait
        if (mixed) {
#pragma unroll
            for (int j = 0; j < CH; ++j) y[AT + j] = fresh ? y[AT + j] : s[j] + y[AT + j];
        } else {
#pragma unroll
            for (int j = 0; j < CH; ++j) y[AT + j] = s[j] + y[AT + j];
        }
        blk_tm_add<NV, AT + CH>(a, y, fresh, mixed);
    }
}

// a.team_size teams per group are in use (at most EW; one entry at a time per team).
// UNITS: pass 1 of vectors beyond shared memory.  An "entry" is then a unit, one of the
// split_R chunks of n^D consecutive values of an entry; a.chunks units, their fastest D of
// a.d axes, and the results are stored to the same place of the entry's workspace.
template <typename TO, typename CF, bool UNITS = false>
__global__ void __launch_bounds__(Blk<CF>::threads, Blk<CF>::ctas) fwd_block_kernel(const FwdArgs<float, TO> a)
{
    using B = Blk<CF>;
    constexpr int D = CF::D;
    constexpr int V = B::V, V0 = B::V0, T = B::T, N = B::N, VS = B::VS, FS = B::FS, EW = B::EW, W = B::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_tmem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = warp / W, gw = warp - group * W, grank = gw * 32 + lane;
    const int slots = a.prefetch ? 2 : 1;
    float *base = reinterpret_cast<float *>(smem_raw) + (size_t)group * slots * B::SLOT;

    // `ew` teams of every group are in use; team g of all takes `share` chunks of entries,
    // the first `more` teams one more.  (kGuided, several waves: the teams beyond the first one take
    // a.later_share each.)  Run sums (in FP32) are of at most chunk_len (8 or fewer)
    // entries.  FP64 outputs: they are cut at chunk edges, so that they are fixed by the batch.
    // FP32 outputs: a chunk is an entry; a sum of chunk_len of them is added to the output, or
    // (kTwo) to the run's whole sum, every 8 entries of the team's share.
    constexpr bool kCuts = sizeof(TO) == 8, kTwo = !UNITS && B::template two_levels<TO>;
    static_assert(!UNITS || (!kCuts && T >= 8), "units are stored as FP32 by large teams");
    const int ew = a.team_size;
    const long long teams = (long long)gridDim.x * (blockDim.x / (32 * W)) * ew;
    const long long team0 = ((long long)blockIdx.x * (blockDim.x / (32 * W)) + group) * ew;
    const long long chunks = kCuts || UNITS ? a.chunks : a.nb;
    const int share = a.entries_per_team;
    constexpr bool kGuided = !UNITS && B::template guided<TO>;
    const bool waves = kGuided && a.first_ctas > 0;
    const long long first = waves ? (long long)a.first_ctas * (blockDim.x / (32 * W)) * ew : teams;
    const long long more = waves ? 0 : chunks - share * teams;
    auto chunk_of = [&](long long g) {
        if constexpr (kGuided) {
            if (g > first) {
                const long long c = first * share + (g - first) * a.later_share;
                return c < chunks ? c : chunks;
            }
        }
        return g * share + (g < more ? g : more);
    };
    auto entry_of = [&](long long c) {
        if constexpr (!kCuts) return c;
        return c * a.chunk_len < a.nb ? c * a.chunk_len : a.nb;
    };
    // the most entries of any team, and whether sums outlive an entry
    const int most = kGuided && team0 >= first ? a.later_share : share + (more > 0 ? 1 : 0);
    const int iters = kCuts ? most * a.chunk_len : most;
    const bool sums = !UNITS && a.chunk_len > 1 && (kCuts || iters > 2);
    // The next CTA of a kernel that can allocate tensor memory starts on this SM only when
    // this one gives up its right to: at once where nothing is allocated (held to the end,
    // it left one CTA per SM: d = 4, n = 4, 5000 entries 10.0 us).
    if (!UNITS && !sums && warp == 0) asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    if (sums) {
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(&s_tmem)),
                         "n"(B::template cols<TO>)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    const unsigned tmem = sums ? s_tmem + ((unsigned)(warp & 3) << 21) + (unsigned)(warp >> 2) * V : 0u;
    // this thread's team and rank in it
    const int team = grank / T, t = grank - team * T;
    const bool mine = team < ew;
    const long long c0 = mine ? chunk_of(team0 + team) : 0, e0 = mine ? entry_of(c0) : 0;
    const int count = mine ? (int)(entry_of(chunk_of(team0 + team + 1)) - e0) : 0;
    // the pointers of the next entries to be copied, spread over the lanes: kind k (0: the
    // input, 1 + i: factor i) of team j in register k / K, lane k % K * EW + j
    constexpr int K = 32 / EW < D + 1 ? 32 / EW : D + 1, NPR = (D + K) / K;
    const int lteam = lane % EW, lkind = lane / EW;
    const long long l0 = entry_of(chunk_of(team0 + lteam));
    const int lcount = lteam < ew ? (int)(entry_of(chunk_of(team0 + lteam + 1)) - l0) : 0;
    const float *ptrs[NPR];
    auto load_ptrs = [&](int it) {
#pragma unroll
        for (int r = 0; r < NPR; ++r) {
            const int k = r * K + lkind;
            const bool has = it < lcount && lkind < K && k <= D;
            if constexpr (UNITS) {
                const unsigned u = (unsigned)(l0 + it), e = u / (unsigned)a.split_R;
                const float *const *src = k == 0 ? a.in + e : a.mats + ((size_t)e * a.d + (a.d - D) + (k - 1));
                ptrs[r] = has ? *src + (k == 0 ? (size_t)(u - e * a.split_R) * N : 0) : nullptr;
            } else {
                const float *const *src = k == 0 ? a.in + (l0 + it) : a.mats + ((l0 + it) * D + (k - 1));
                ptrs[r] = has ? *src : nullptr;
            }
        }
    };
    // pointer of kind `kind` (a constant) of team j
    auto ptr_of = [&](int kind, int j) {
        return reinterpret_cast<const float *>(
            __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(ptrs[kind / K]), kind % K * EW + j));
    };
    BlkFactorLanes<CF> fl(lane, a.stride);
    // a vector by GS lanes (small teams: several vectors at a time), or by the whole group
    constexpr int pieces = B::shifted || B::copy16 ? (N + 6) / 4 : N;
    constexpr int GS = EW == 1 ? 32 * W : pieces > 16 ? 32 : pieces > 8 ? 16 : pieces > 4 ? 8 : 4;
    // copies the entries of the loaded pointers; returns the shift of this thread's own vector
    auto copy_data = [&](int slot) {
        float *vdst = base + (size_t)slot * B::SLOT, *fdst = vdst + (EW * VS + 3) / 4 * 4;
        const float *own = ptr_of(0, EW == 1 || !mine ? 0 : team);
        if constexpr (EW == 1) {
            if (own) blk_copy_vec<B, GS>(vdst, own, grank);
        } else {
#pragma unroll 1
            for (int j0 = 0; j0 < ew; j0 += 32 * W / GS) {
                const int j = j0 + grank / GS;
                const float *src = ptr_of(0, j < ew ? j : 0);
                if (j < ew && src) blk_copy_vec<B, GS>(vdst + j * VS, src, lane % GS);
            }
        }
        fl.copy(fdst, gw, ew, [&](int i, int j) { return ptr_of(1 + i, j); });
        return B::shifted ? blk_shift(own) : 0;
    };

    auto out_of = [&](long long e) {
        if constexpr (UNITS) {
            const unsigned w = (unsigned)e / (unsigned)a.split_R;
            return a.ws[w] + (size_t)((unsigned)e - w * a.split_R) * N;
        } else {
            return a.out[e];
        }
    };
    TO *o = count > 0 ? out_of(e0) : nullptr;
    bool fresh = true;  // the current run starts with this entry
    int run = 0;        // entries in its sum (where chunk_len bounds them)
    bool whole = false;  // kTwo: the run has a sum of the second level
    long long chunk = c0 + 1;  // FP64 outputs: the next chunk and, as an entry of this team, its start
    int cut = kCuts && mine ? (int)(entry_of(chunk) - e0) : 0;
    load_ptrs(0);
    int sh_next = 0;  // shift of the entry staged ahead
    if (slots == 2) {
        sh_next = copy_data(0);
        cp_async_commit();
        if (iters > 1) load_ptrs(1);
    }
    for (int it = 0; it < iters; ++it) {
        const int slot = slots == 2 ? it & 1 : 0;
        const bool active = it < count;
        TO *o_next = it + 1 < count ? out_of(e0 + it + 1) : nullptr;
        int sh;
        if (slots == 2) {
            cp_async_wait_all();
            blk_sync<W, B::C>(group);  // entry it staged, the other slot free
            sh = sh_next;
            if (it + 1 < iters) {
                sh_next = copy_data(slot ^ 1);
                cp_async_commit();
                if (it + 2 < iters) load_ptrs(it + 2);
            }
        } else {
            blk_sync<W, B::C>(group);  // the slot's last reads are done
            sh = copy_data(0);
            cp_async_commit();
            if (it + 1 < iters) load_ptrs(it + 1);
            cp_async_wait_all();
            blk_sync<W, B::C>(group);
        }

        typename B::X x[V0];
        float *vec = base + (size_t)slot * B::SLOT;
        const int own = mine ? team : 0;
        blk_passes<CF, 0>(x, vec + own * VS + sh,
                             (unsigned)__cvta_generic_to_shared(vec + (EW * VS + 3) / 4 * 4 + own * FS), t, active, group);

        // into the run's sum; the run ends where the next entry's output differs
        using L = BlkPass<CF, B::passes - 1>;
        float y[V];
#pragma unroll
        for (int j = 0; j < V0; ++j) blk_split(x[j], y[j], y[V - V0 + j]);
        if constexpr (UNITS) {
            if (active) {
                TO *p = o + t;
#pragma unroll
                for (int i = 0; i < L::NG; ++i) {
                    if (L::has(t, i)) {
#pragma unroll
                        for (int m = 0; m < L::NB; ++m) p[T * i + m * L::Q] = y[(i % L::NH) * L::NB + m + (i / L::NH) * V0];
                    }
                }
            }
            o = o_next;
            continue;
        }
        bool last = active && (!sums || o_next != o || (!kCuts && !kTwo && run + 1 == a.chunk_len));
        bool edge = false;  // sums of runs that go on are added to the second level
        if constexpr (kTwo) edge = it % 8 == 7;
        if constexpr (kCuts) {
            if (active && it + 1 == cut) {
                last = true;
                ++chunk;
                cut = (int)(entry_of(chunk) - e0);
            }
        }
        if (__any_sync(0xffffffffu, active && !fresh)) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            const bool mixed = __any_sync(0xffffffffu, fresh);
            blk_tm_add<V>(tmem, y, fresh, mixed);
        }
        if constexpr (kTwo) {
            const bool add = active && whole && (last || edge);
            if (__any_sync(0xffffffffu, add)) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                blk_tm_add<V>(tmem + B::cols_used, y, !add, true);
            }
        }
        if constexpr (T >= 8) {
            if (last) {
                TO *p = o + t;
#pragma unroll
                for (int i = 0; i < L::NG; ++i) {
                    if (L::has(t, i)) {
#pragma unroll
                        for (int m = 0; m < L::NB; ++m)
                            atomic_add<TO>(p + T * i + m * L::Q, blk_out<TO>(y[(i % L::NH) * L::NB + m + (i / L::NH) * V0]));
                    }
                }
                o = o_next;
            }
        } else if (__any_sync(0xffffffffu, last)) {
            // small teams: back through the slot, so that an addition's lanes cover whole
            // sectors of the output; finished runs of consecutive teams into one FP32 output
            // are summed first
            float *const mine_at = vec + own * VS + sh;
            __syncwarp();  // the slot's last reads are done
            if (last) {
#pragma unroll
                for (int i = 0; i < L::NG; ++i) {
                    if (L::has(t, i)) {
                        float *const p = mine_at + L::base(t, i);
#pragma unroll
                        for (int m = 0; m < L::NB; ++m) p[m * L::step] = y[(i % L::NH) * L::NB + m + (i / L::NH) * V0];
                    }
                }
            }
            __syncwarp();
            const unsigned done = __ballot_sync(0xffffffffu, last && t == 0);
            const unsigned long long out = (unsigned long long)reinterpret_cast<uintptr_t>(o);
#pragma unroll 1
            for (int q0 = 0; q0 < N; q0 += 32) {
                const int q = q0 + lane;
                unsigned long long at = 0;
                float sum = 0.f, part = 0.f;
                auto add = [&]() {
                    if (at != 0 && q < N) atomic_add<TO>(reinterpret_cast<TO *>(at) + q, blk_out<TO>(EW > 8 ? part + sum : sum));
                };
#pragma unroll 1
                for (unsigned left = done; left != 0; left &= left - 1) {
                    const int l = __ffs(left) - 1;
                    const unsigned long long to = __shfl_sync(0xffffffffu, out, l);
                    const float v = vec[l / T * VS + __shfl_sync(0xffffffffu, sh, l) + (q < N ? B::phys(q) : 0)];
                    if (sizeof(TO) == 4 && to == at) {
                        // more than 8 teams: 8 at a time (one chain over 32 of them had more error
                        // than the kernels before: d = 2, n = 3, 27 entries per output 1.0e-7
                        // against 0.83e-7)
                        if (EW > 8 && l % (8 * T) == 0) {
                            part += sum;
                            sum = v;
                        } else {
                            sum += v;
                        }
                    } else {
                        add();
                        at = to;
                        sum = v;
                        part = 0.f;
                    }
                }
                add();
            }
            if (last) o = o_next;
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, active && !last)) blk_tm_st<V>(tmem + (kTwo && edge ? B::cols_used : 0), y);
        fresh = last || edge;
        run = last ? 0 : run + 1;
        if constexpr (kTwo) whole = !last && (whole || edge);
    }
    if (sums) {
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "n"(B::template cols<TO>) : "memory");
        }
    }
}

// What the planner needs of one instantiation: entries per group, threads per group, groups
// per CTA (at most), shared-memory bytes per group and slot, tensor-memory columns per CTA.
struct BlkInfo {
    const void *fn = nullptr;
    int n = 0, d = 0;  // of the instantiation
    int EW = 0, group = 0, groups = 0, slot_bytes = 0, cols = 0;
    bool guided = false;
};

template <typename TO, typename CF, bool UNITS = false> BlkInfo blk_info_of()
{
    using B = Blk<CF>;
    return BlkInfo{(const void *)fwd_block_kernel<TO, CF, UNITS>, CF::NN, CF::D, B::EW, 32 * B::W, B::C, B::SLOT * 4, B::template cols<TO>,
                   !UNITS && B::template guided<TO>};
}

// The instantiation for large batches (fn == nullptr where (n, d) has none) and, where
// there is one, for small batches.
struct BlkPair {
    BlkInfo large, small;
};
template <typename TO, int NN> BlkPair blk_lookup_n(int d);

template <typename TO, int NN, int D> BlkPair blk_pair_of()
{
    using L = BlkLarge<NN, D>;
    using S = BlkSmall<NN, D>;
    BlkPair p{blk_info_of<TO, L>(), BlkInfo{}};
    // one fibre per thread pays where a vector still has few threads and passes
    if constexpr (NN >= 4 && L::M > S::M && D > 1 && Blk<S>::T <= (NN == 4 ? 256 : 128)) p.small = blk_info_of<TO, S>();
    return p;
}

template <typename TO> BlkPair blk_lookup(int n, int d)
{
    if constexpr (sizeof(TO) == 4) {  // FP64 outputs, n = 2: fwd_pair_kernel is faster throughout
        if (n == 2) return blk_lookup_n<TO, 2>(d);
    }
    switch (n) {
    case 3: return blk_lookup_n<TO, 3>(d);
    case 4: return blk_lookup_n<TO, 4>(d);
    case 5: return blk_lookup_n<TO, 5>(d);
    case 6: return blk_lookup_n<TO, 6>(d);
    case 7: return blk_lookup_n<TO, 7>(d);
    case 8: return blk_lookup_n<TO, 8>(d);
    case 9: return blk_lookup_n<TO, 9>(d);
    case 10: return blk_lookup_n<TO, 10>(d);
    default: return BlkPair{};
    }
}

}  // namespace kgb

#define KGB_BLK_D(TO, NN, D) \
    case D: return blk_pair_of<TO, NN, D>();
#define KGB_BLK_N(TO, NN, ...)                                       \
    template <> BlkPair blk_lookup_n<TO, NN>(int d)                  \
    {                                                                \
        switch (d) {                                                 \
            __VA_ARGS__                                              \
        default: return BlkPair{};                                   \
        }                                                            \
    }
