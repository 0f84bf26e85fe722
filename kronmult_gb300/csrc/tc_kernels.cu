// Tensor-core (tcgen05) forward for n = 8: FP32 storage, TF32 or BF16 mode
// products with FP32 accumulation in tensor memory, FP64 output accumulation.
//
// For n = 8 every mode product of the backward sweep (kronmult_gpu/kronmult.cu:54-78)
//     Y[c + r*F] = sum_k A_i(r, k) X[k + 8c],   F = N/8 fibres
// is a dense GEMM D[c][r] = sum_k X^T[c][k] A_i^T[k][r] with M = F, N = 8, K = 8.
// It runs as tcgen05.mma.cta_group::1 with M = 128 fibres per instruction
// (N = 16, the smallest N for M = 128; K = 8 for TF32, K = 16 for BF16 with the
// upper 8 zero).  Operands live in shared memory in the canonical K-major,
// no-swizzle layout of 8-row x 16-byte core matrices; the accumulator lives in
// tensor memory, one 16-column block per PAIR of 128-fibre tiles: the even tile
// multiplies B = [A_i^T | 0] into columns 0..7, the odd tile B = [0 | A_i^T]
// accumulated into columns 8..15, so no accumulator column is padding and a CTA
// needs half the columns (more CTAs per SM).  After each mode the four warps read
// their 32 TMEM lanes (tcgen05.ld.32x32b), round to the operand type and write
// the mode output straight into the next mode's operand layout at the rotated
// positions, so the vector never leaves shared memory.
//
// BF16 (fwd_tc_bf16_kernel) keeps the vector operand MN-major (8 consecutive fibres =
// 16 contiguous bytes per K row of a core matrix) and applies the modes in the order
// 0, 1, ..., d-1: the contracted index is then always the most significant digit of the
// fibre index, and the 8 outputs a thread reads from its TMEM lane (one fibre, the 8
// values of the new index) are 8 consecutive fibres of the next mode's operand, written
// with ONE 16-byte store.  The first operand is the natural vector itself read as
// MN-major (fibre = the fastest d-1 indices, K = the slowest), converted 8 values per
// 16-byte store.  Two 128-fibre tiles share one MMA: K = 16 holds the even tile in K
// rows 0..7 and the odd one in rows 8..15, against the block-diagonal factor operand
// [A_i 0; 0 A_i], so the operand carries no zero padding.  TF32 (fwd_tc_kernel; K = 8
// per MMA) keeps the backward order and the K-major operand, written element by element.
//
// One CTA of up to four warps works on one entry at a time; several CTAs per SM overlap the
// input loads.  Consecutive entries with the same output pointer are summed in tensor memory
// and added with FP64 atomics.
//
// What bounds it: the chain of steps of an entry (copy, convert, then per mode MMA, wait,
// TMEM load, store, barrier) times the CTAs that shared memory admits (d = 4: 6 for TF32, 8
// for BF16).  Hence d at compile time, operands that stay in uniform registers for the MMAs,
// one barrier per mode, all TMEM loads of a mode before one wait, and exact integer
// conversion of the sums to FP64.  FP32 storage, FP64 outputs, 32768 entries of d = 4: TF32
// 224 -> 176 us (shared-memory pipe 63 % busy), BF16 140 -> 131 us, split BF16 225 -> 209 us;
// 100000 entries of d = 2: TF32 176 -> 51, BF16 153 -> 52, split 232 -> 92 us.
//
// Every wait on an mbarrier is bounded; on timeout the kernel records an error
// code in a device word (kronmult_device_error) and leaves after freeing its
// tensor memory.
#include <cuda_bf16.h>
#include <cstdint>
#include "fwd_launch.cuh"

namespace kgb {

__device__ unsigned int g_tc_error = 0;  // 0 = ok; otherwise the code of the first failure

namespace {

constexpr int kTileRows = 128;               // fibres per MMA (M)
constexpr int kTileBytes = kTileRows * 32;   // one K-major tile: 128 rows x 32 bytes
constexpr int kBBytes = 16 * 32;             // one factor operand: 16 rows x 32 bytes
constexpr unsigned kWaitLimit = 1u << 22;    // bounded mbarrier polling
// BF16 MN-major vector operand: per group of 8 fibres, K rows 0..7 (128 bytes), K rows
// 8..15 (128 bytes), then 16 bytes of padding, so that 8 consecutive groups start in 8
// different 16-byte bank slots
constexpr uint32_t kMnLbo = 128;                 // K-group stride
constexpr uint32_t kMnSbo = 272;                 // 8-fibre group stride

enum : int { KIND_TF32 = 0, KIND_BF16 = 1 };

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// byte offset of element (row, k) of a 32-byte-row K-major operand in core-matrix layout:
// core matrix = 8 rows x 16 bytes (128 B contiguous); K-adjacent core matrices are
// 128 B apart (leading byte offset), M-adjacent 8-row groups 256 B apart (stride byte offset)
__device__ __forceinline__ uint32_t core_offset(uint32_t row, uint32_t kbyte)
{
    return (row >> 3) * 256u + (kbyte >> 4) * 128u + (row & 7u) * 16u + (kbyte & 15u);
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo = 128u, uint32_t sbo = 256u)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);          // start address
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;      // leading byte offset (K direction)
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;      // stride byte offset (M/N direction)
    d |= (uint64_t)1u << 46;                          // descriptor version for sm_100 family
    return d;                                         // base offset 0, no swizzle
}

// The A operand (the vector: `tiles` tiles of 128 rows) uses the same core matrices
// with a different arrangement: the k-chunk-0 core matrices of all rows first (8-row
// groups 128 B apart, SBO = 128), the k-chunk-1 ones LBO = tiles*2048 + 64 bytes
// later.  The two 16-byte halves of a row then sit 64 bytes apart modulo the 128-byte
// bank row, so the epilogue's stores (consecutive lanes = consecutive rows, both
// halves) and the staging conversion hit distinct banks.
__device__ __forceinline__ uint32_t a_offset(uint32_t row, uint32_t kbyte, uint32_t lbo)
{
    return (row >> 3) * 128u + (kbyte >> 4) * lbo + (row & 7u) * 16u + (kbyte & 15u);
}

template <int KIND, bool A_MN_MAJOR = false> __device__ __forceinline__ constexpr uint32_t instr_desc()
{
    // D = F32; A, B = TF32 (2) or BF16 (1); A K-major, or MN-major (bit 15, "transpose A");
    // B K-major; N = 16; M = 128
    return (1u << 4) | ((KIND == KIND_TF32 ? 2u : 1u) << 7) | ((KIND == KIND_TF32 ? 2u : 1u) << 10) |
           ((A_MN_MAJOR ? 1u : 0u) << 15) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
}

// The lane that issues MMAs and their commits.  Whole warps run the issuing code with warp-
// uniform operands, predicated on that lane (in a branch of one thread the operands went
// through vector registers: 600 cycles per mode, now 100).
__device__ __forceinline__ uint32_t elect_lane()
{
    uint32_t leader;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}\n" : "=r"(leader));
    return leader;
}

// D (+)= A B where `leader`; BF16: A MN-major (the vector), B K-major (the factor)
template <int KIND>
__device__ __forceinline__ void mma(uint32_t leader, uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate)
{
    if constexpr (KIND == KIND_TF32) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
            "l"(adesc), "l"(bdesc), "r"(instr_desc<KIND>()), "r"(accumulate), "r"(leader));
    } else {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
            "l"(adesc), "l"(bdesc), "r"(instr_desc<KIND_BF16, true>()), "r"(accumulate), "r"(leader));
    }
}

// 8 FP32 values rounded to BF16 (nearest even), packed in order into 16 bytes
__device__ __forceinline__ uint4 pack_bf16x8(float a0, float a1, float a2, float a3, float a4, float a5, float a6,
                                             float a7)
{
    uint4 r;
    __nv_bfloat162 h;
    h = __floats2bfloat162_rn(a0, a1);
    r.x = *reinterpret_cast<uint32_t *>(&h);
    h = __floats2bfloat162_rn(a2, a3);
    r.y = *reinterpret_cast<uint32_t *>(&h);
    h = __floats2bfloat162_rn(a4, a5);
    r.z = *reinterpret_cast<uint32_t *>(&h);
    h = __floats2bfloat162_rn(a6, a7);
    r.w = *reinterpret_cast<uint32_t *>(&h);
    return r;
}

// BF16 K-stacked operand: the tiles of a pair (128 fibres each) share 8-fibre groups; K
// rows 0..7 of a group hold the even tile, K rows 8..15 (one K-group = 128 bytes later)
// the odd one, so one MMA with K = 16 and a block-diagonal factor operand computes both
// tiles and no operand byte is padding.  Byte offset of fibre group g, K row kk:
constexpr uint32_t kPairBytes = 16 * kMnSbo;  // 16 groups of 8 fibres
constexpr int kBf16B = 512;                   // factor operand: 16 rows x 16 K x 2 bytes
__device__ __forceinline__ uint32_t mn_offset(uint32_t g, uint32_t kk)
{
    const uint32_t t = g >> 4;  // tile of the group
    return (t >> 1) * kPairBytes + (g & 15u) * kMnSbo + (t & 1u) * kMnLbo + kk * 16u;
}

// FP64 addition into global memory without a returned value
__device__ __forceinline__ void red_add_f64(double *p, double v)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// 8x8 transpose across the 8 lanes of each aligned lane octet: afterwards lane l's v[j]
// is lane j's former v[l] (three butterfly stages of register-pair exchanges)
__device__ __forceinline__ void octet_transpose(float (&v)[8], int lane)
{
#pragma unroll
    for (int s = 4; s >= 1; s >>= 1) {
        const bool upper = (lane & s) != 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j & s) continue;
            const float send = upper ? v[j] : v[j | s];
            const float recv = __shfl_xor_sync(0xffffffffu, send, s);
            if (upper)
                v[j] = recv;
            else
                v[j | s] = recv;
        }
    }
}

__device__ __forceinline__ void mma_commit(uint32_t leader, uint32_t mbar)
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(mbar), "r"(leader)
        : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase, unsigned limit = kWaitLimit)
{
    for (unsigned it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// 16 consecutive columns of this warp's 32 lanes: the two tiles of one block
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v0)[8], float (&v1)[8])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(v0[0]), "=f"(v0[1]), "=f"(v0[2]), "=f"(v0[3]), "=f"(v0[4]), "=f"(v0[5]), "=f"(v0[6]), "=f"(v0[7]),
          "=f"(v1[0]), "=f"(v1[1]), "=f"(v1[2]), "=f"(v1[3]), "=f"(v1[4]), "=f"(v1[5]), "=f"(v1[6]), "=f"(v1[7])
        : "r"(taddr));
}
// no use of loaded values before the wait
template <int NT> __device__ __forceinline__ void tmem_wait_ld(float (&v)[NT][8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int j = 0; j < 8; ++j) asm volatile("" : "+f"(v[t][j]));
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ float to_tf32(float x)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// 8 FP32 values split into BF16 pairs v = hi + lo: hi rounded to nearest, lo the rounded
// remainder (v - hi is exact in FP32), each set packed in order into 16 bytes
__device__ __forceinline__ void split_bf16x8(const float (&v)[8], uint4 &hi, uint4 &lo)
{
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 hb = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        h[i] = *reinterpret_cast<const uint32_t *>(&hb);
        // hi back in FP32 (a BF16 value is the upper half of its FP32 bits), both lanes at
        // once; the remainders with one packed subtraction
        const f2 hf = ((unsigned long long)(h[i] & 0xFFFF0000u) << 32) | ((unsigned long long)(h[i] & 0xFFFFu) << 16);
        float r0, r1;
        f2_unpack(f2_sub(f2_pack(v[2 * i], v[2 * i + 1]), hf), r0, r1);
        const __nv_bfloat162 lb = __floats2bfloat162_rn(r0, r1);
        l[i] = *reinterpret_cast<const uint32_t *>(&lb);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// store one value of the operand element (row, k) in the operand type of KIND: B
// operands (factors) in the plain core-matrix layout, A (lbo != 0) in the split one
template <int KIND>
__device__ __forceinline__ void put(unsigned char *base, uint32_t row, uint32_t k, float v, uint32_t lbo = 0)
{
    constexpr uint32_t es = KIND == KIND_TF32 ? 4u : 2u;
    const uint32_t off = lbo ? a_offset(row, k * es, lbo) : core_offset(row, k * es);
    if constexpr (KIND == KIND_TF32) {
        *reinterpret_cast<float *>(base + off) = to_tf32(v);
    } else {
        *reinterpret_cast<__nv_bfloat16 *>(base + off) = __float2bfloat16_rn(v);
    }
}

}  // namespace

struct TcArgs {
    const float *const *mats;
    const float *const *in;
    double *const *out;
    long long nb;
    int stride, entries_per_chunk;
};

// d modes: sizes known at compile time.  A CTA has no more warps than the vector has fibres
// in tensor-memory lanes (the others' instructions are wasted: d = 2, 200000 entries, TF32,
// 198 us with four warps, 110 with one; d = 3, 60000 entries, 89 with four, 65 with two).  Two
// warpgroups for d = 4 were slower (TF32, 32768 entries: 220 against 170 us).
template <int D> struct TcShape {
    static constexpr int d = D, N = 1 << (3 * D), F = N / 8;
    static constexpr int threads = F >= 128 ? 128 : F > 32 ? F : 32;
    static constexpr int copier = threads > 32 ? 32 : 0;  // issues bulk copies (warp 0 issues MMAs)
    static constexpr int tiles = (F + kTileRows - 1) / kTileRows, pairs = (tiles + 1) / 2;
    static constexpr int cols = 32 * pairs;  // tensor-memory columns: mode output + run sums
    static constexpr int fac_slots = (D * 64 + threads - 1) / threads;  // factor elements per thread
};

// A CTA's entries: chunks of entries_per_chunk consecutive ones, gridDim.x chunks apart (a grid
// of all chunks: one each).
// Run sums end with their chunk.  (One chunk per CTA: a CTA of a kernel that allocates tensor
// memory starts on an SM only when the one before has given up its right to, which left the
// small vectors waiting for CTA starts.)
struct TcWalk {
    long long e;  // the current entry (a.nb or beyond: none)
    int left;     // entries left in its chunk, itself included
    __device__ __forceinline__ TcWalk next(const TcArgs &a) const
    {
        if (left > 1) return TcWalk{e + 1, left - 1};
        return TcWalk{e + 1 + (long long)(gridDim.x - 1) * a.entries_per_chunk, a.entries_per_chunk};
    }
};

// per-thread pointers of one entry, loaded one entry ahead of the copies that use them
template <int D> struct TcPtrs {
    const float *src;
    const float *mat[TcShape<D>::fac_slots];
};

template <int D> __device__ __forceinline__ void tc_load_ptrs(TcPtrs<D> &p, const TcArgs &a, long long e, int tid)
{
    p.src = a.in[e];
#pragma unroll
    for (int s = 0; s < TcShape<D>::fac_slots; ++s) {
        const int idx = tid + s * TcShape<D>::threads;
        p.mat[s] = idx < D * 64 ? a.mats[e * D + (idx >> 6)] : nullptr;
    }
}

// asynchronous copy of one entry's vector into the raw staging slot (natural order)
// and of its factor elements into registers: thread tid holds fv[s] = A_i(r, k) for
// idx = tid + 128 s, i = idx / 64, r = idx % 8, k = (idx / 8) % 8.  The vector is one TMA
// bulk copy (cp.async.bulk) issued by thread 0 and completed on the staging barrier
// `sbar` when its source is 16-byte aligned; otherwise every thread copies 4-byte
// elements with cp.async and thread 0 completes the barrier's phase without bytes.
// Either way the staging barrier completes exactly one phase per entry.  The factor
// loads are plain loads consumed one entry later, so their latency is hidden too.
// Returns whether it was the bulk copy.
template <int D>
__device__ __forceinline__ bool tc_stage_async(float *raw, float (&fv)[TcShape<D>::fac_slots], const TcPtrs<D> &p,
                                               const TcArgs &a, int tid, uint32_t sbar)
{
    constexpr int N = TcShape<D>::N;
    constexpr unsigned bytes = (unsigned)N * 4u;
    const bool bulk = (reinterpret_cast<uintptr_t>(p.src) & 15u) == 0;
    if (bulk) {
        if (tid == TcShape<D>::copier) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sbar), "r"(bytes)
                         : "memory");
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    smem_u32(raw)),
                "l"(p.src), "r"(bytes), "r"(sbar)
                : "memory");
        }
    } else {
        for (int q = tid; q < N; q += TcShape<D>::threads) cp_async<4>(raw + q, p.src + q);
        if (tid == TcShape<D>::copier) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sbar) : "memory");
    }
    cp_async_commit();
#pragma unroll
    for (int s = 0; s < TcShape<D>::fac_slots; ++s) {
        const int idx = tid + s * TcShape<D>::threads;
        if (idx < D * 64) {
            const int r = idx & 7, k = (idx >> 3) & 7;
            fv[s] = __ldg(p.mat[s] + r + (size_t)k * a.stride);
        }
    }
    return bulk;
}

template <int D> __global__ void __launch_bounds__(TcShape<D>::threads, D == 4 ? 6 : 16) fwd_tc_kernel(const TcArgs a)
{
    constexpr int KIND = KIND_TF32;
    using S = TcShape<D>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int N = S::N, F = S::F, d = D, tiles = S::tiles, blocks = S::pairs;  // 16-column accumulator blocks, two tiles each
    // shared memory: one raw staging slot for the vector, operand A, operands B, barriers.
    // The slot is refilled with the next entry as soon as this entry's operands are built.
    float *raw = reinterpret_cast<float *>(smem_raw);
    unsigned char *xs = reinterpret_cast<unsigned char *>(raw + N);  // tiles x 4 KB
    unsigned char *bs = xs + (size_t)tiles * kTileBytes + 64;            // d x 512 B: [A_i^T | 0]
    unsigned char *bs2 = bs + (size_t)d * kBBytes;                         // d x 512 B: [0 | A_i^T]
    uint64_t *mbar = reinterpret_cast<uint64_t *>(bs2 + (size_t)d * kBBytes);  // MMA completion
    uint64_t *sbar = mbar + 1;                                                  // staging completion
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbar + 2);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

    const long long nb = a.nb;
    TcWalk w{(long long)blockIdx.x * a.entries_per_chunk, a.entries_per_chunk};  // the entry being computed
    if (w.e >= nb) return;
    TcWalk w1 = w.next(a);  // the entry staged after it

    // first of all: the SM's next CTA starts only when this one has given up its right to allocate
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "n"(S::cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const uint32_t sbar_a = smem_u32(sbar);
    if (tid == S::copier) {  // the thread that uses the staging barrier before the others see it
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    TcPtrs<D> nxt;
    float fv[S::fac_slots] = {};  // factor elements of the entry staged last
    tc_load_ptrs<D>(nxt, a, w.e, tid);
    const bool bulk0 = tc_stage_async<D>(raw, fv, nxt, a, tid, sbar_a);
    if (w1.e < nb) tc_load_ptrs<D>(nxt, a, w1.e, tid);
    // while the first vector is on its way: operands zeroed once, that is the zero half of each
    // B (rows 8..15 of [A^T | 0], rows 0..7 of [0 | A^T]) and the rows beyond F
    for (int v = tid + (F % kTileRows == 0 ? (tiles * kTileBytes + 64) / 16 : 0);
         v < (tiles * kTileBytes + 64 + 2 * d * kBBytes) / 16; v += S::threads)
        reinterpret_cast<int4 *>(xs)[v] = make_int4(0, 0, 0, 0);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tacc = tmem + 16u * blocks;   // run accumulator after the mode output
    const uint32_t mbar_a = smem_u32(mbar);
    const uint32_t xs_a = smem_u32(xs), bs_a = smem_u32(bs), bs2_a = smem_u32(bs2);
    constexpr uint32_t lboa = (uint32_t)tiles * 2048u + 64u;  // A operand: k-chunk-1 core matrices this far after chunk 0
    const uint32_t leader = elect_lane();  // of each warp; warp 0's issues the MMAs
    uint32_t phase = 0, sphase = 0;
    bool failed = false;
    bool staging = true;  // a staging copy is in flight whose phase has not been waited for
    double *cur = nullptr;

    // run sum (TMEM accumulator) -> FP64 atomics into `dst`
    auto flush = [&](double *dst) {
        auto add_tile = [&](int t, const float (&v)[8]) {
            const int c = t * kTileRows + warp * 32 + lane;
            if (c < F)
#pragma unroll
                for (int r = 0; r < 8; ++r) red_add_f64(dst + c + r * F, blk_out<double>(v[r]));
        };
#pragma unroll
        for (int j = 0; j < blocks; ++j) {
            float v[2][8];
            tmem_ld16(tacc + ((uint32_t)(warp * 32) << 16) + 16u * j, v[0], v[1]);
            tmem_wait_ld(v);
            add_tile(2 * j, v[0]);
            add_tile(2 * j + 1, v[1]);
        }
    };

    bool ok = true;      // this warp's waits so far; the CTA agrees on it at the next barrier
    bool bulk = bulk0;   // how the entry being computed was staged
    for (; w.e < nb; w = w1, w1 = w.next(a)) {
        double *o = a.out[w.e];
        cp_async_wait_all();
        ok = ok && mbar_wait(sbar_a, sphase);  // the slot's bulk copy (or its empty phase)
        ok = __all_sync(0xffffffffu, ok);
        // a bulk copy is complete for whoever waited for it, copies by threads need a barrier;
        // the MMAs that read the operands are done for every thread (each waited for them)
        if (!bulk) __syncthreads();
        if (ok) {
            sphase ^= 1u;
            staging = false;
        }
        // operands: B_i[row r][k] = A_i(r, k) (and row r + 8 of the second copy); input
        // natural index p = k + 8c -> A row c, column k
#pragma unroll
        for (int s = 0; s < S::fac_slots; ++s) {
            const int v = tid + s * S::threads;
            if (v < d * 64) {
                const int i = v >> 6, r = v & 7, k = (v >> 3) & 7;
                put<KIND>(bs + (size_t)i * kBBytes, r, k, fv[s]);
                put<KIND>(bs2 + (size_t)i * kBBytes, r + 8, k, fv[s]);
            }
        }
        // natural position p = k + 8c -> operand row c, column k: the 4 values of a float4
        // are one 16-byte half of a core-matrix row
#pragma unroll
        for (int q = tid; q < N / 4; q += S::threads) {
            const float4 v4 = *reinterpret_cast<const float4 *>(raw + 4 * q);
            const uint32_t c = q >> 1, kbyte = (q & 1) * 16;
            *reinterpret_cast<float4 *>(xs + a_offset(c, kbyte, lboa)) =
                make_float4(to_tf32(v4.x), to_tf32(v4.y), to_tf32(v4.z), to_tf32(v4.w));
        }
        // the run continues when this entry adds into the same output as the previous one;
        // otherwise the previous run's sum leaves TMEM before the last mode overwrites it
        const bool cont = o == cur && w.left < a.entries_per_chunk;
        if (!cont && cur != nullptr && ok) flush(cur);
        cur = o;
        fence_async_smem();  // the staging slot has been read (generic proxy) before the bulk copy refills it
        tc_fence_before();
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        if (w1.e < nb) {
            bulk = tc_stage_async<D>(raw, fv, nxt, a, tid, sbar_a);
            staging = true;
            const TcWalk w2 = w1.next(a);
            if (w2.e < nb) tc_load_ptrs<D>(nxt, a, w2.e, tid);
        }

        for (int i = d - 1; i >= 0; --i) {
            if (warp == 0) {
                tc_fence_after();
                const uint32_t dst = i > 0 ? tmem : tacc;
                const uint32_t accumulate = (i == 0 && cont) ? 1u : 0u;
                // even tile: columns 0..7 of its block (overwriting, or adding to the run);
                // odd tile: columns 8..15, always added (the even tile's B zeroed them)
#pragma unroll
                for (int t = 0; t < tiles; ++t)
                    mma<KIND>(leader, dst + 16u * (uint32_t)(t >> 1), smem_desc(xs_a + t * 2048u, lboa, 128u),
                              smem_desc(((t & 1) ? bs2_a : bs_a) + i * kBBytes), (t & 1) ? 1u : accumulate);
                mma_commit(leader, mbar_a);
            }
            // uniform over the warp (the TMEM loads below are warp-collective), over the CTA at
            // the next barrier
            ok = __all_sync(0xffffffffu, mbar_wait(mbar_a, phase));
            phase ^= 1u;
            tc_fence_after();
            if (i > 0) {
                // mode output element (row c, r) goes to natural position p = c + r*F,
                // which is operand row p/8, column p%8 of the next mode; one block (two
                // tiles) at a time keeps 16 values per thread live
                auto store_tile = [&](int t, const float (&v)[8]) {
                    const int c = t * kTileRows + warp * 32 + lane;
                    if (c < F) {
                        if (F >= 64) {
                            // F/8 a multiple of 8: row p/8 = c/8 + r*F/8 keeps its position in
                            // the 8-row group and moves r*F/64 groups, 2F bytes per r
                            const uint32_t base = a_offset((uint32_t)c >> 3, 4u * ((uint32_t)c & 7u), lboa);
#pragma unroll
                            for (int r = 0; r < 8; ++r)
                                *reinterpret_cast<float *>(xs + base + (uint32_t)r * 2u * (uint32_t)F) = to_tf32(v[r]);
                        } else {
#pragma unroll
                            for (int r = 0; r < 8; ++r) {
                                const uint32_t p = c + r * F;
                                put<KIND>(xs, p >> 3, p & 7, v[r], lboa);
                            }
                        }
                    }
                };
                float v[2 * blocks][8];
#pragma unroll
                for (int j = 0; j < blocks; ++j)
                    tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + 16u * j, v[2 * j], v[2 * j + 1]);
                tmem_wait_ld(v);
#pragma unroll
                for (int t = 0; t < 2 * blocks; ++t) store_tile(t, v[t]);
                fence_async_smem();
                tc_fence_before();
                if (__syncthreads_or(!ok)) {
                    failed = true;
                    break;
                }
            }
        }
        if (failed) break;
    }
    if (!ok || failed) {
        failed = true;
        if (lane == 0) atomicCAS(&g_tc_error, 0u, 1u);
    }
    cp_async_wait_all();
    // leaving early with a bulk copy still in flight: one more bounded wait for it, so
    // that it does not land in shared memory after this CTA is gone
    if (failed && staging) mbar_wait(sbar_a, sphase);
    if (cur != nullptr && !failed) flush(cur);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(S::cols) : "memory");
}

// BF16 forward (layout and mode order in the file comment).  Same pipeline as
// fwd_tc_kernel: one staging slot refilled by a bulk copy while the current entry's
// modes run, factors one entry ahead in registers, runs of entries with one output
// summed in TMEM, bounded mbarrier waits.
// SPLIT (KRONMULT_COMPUTE_BF16X3): every operand value v is held as two BF16 values,
// hi = bf16(v) and lo = bf16(v - hi), and each tile pair runs three MMAs into one FP32
// accumulator, x_hi.A_hi + x_lo.A_hi + x_hi.A_lo (the lo.lo term, 2^-16 relative, is
// dropped): about 16 significand bits per product instead of 8.  The hi and lo vector
// operands and factor operands sit side by side in the same layouts.
template <bool SPLIT, int D>
__global__ void __launch_bounds__(TcShape<D>::threads, D < 4 ? 16 : SPLIT ? 5 : 8) fwd_tc_bf16_kernel(const TcArgs a)
{
    using S = TcShape<D>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int N = S::N, F = S::F, d = D, tiles = S::tiles, pairs = S::pairs;
    constexpr int kParts = SPLIT ? 2 : 1;
    float *raw = reinterpret_cast<float *>(smem_raw);                          // staging slot, N floats
    unsigned char *xs = reinterpret_cast<unsigned char *>(raw + N);           // pairs x kPairBytes (hi)
    unsigned char *xl = xs + (size_t)pairs * kPairBytes;                      // the lo parts (SPLIT)
    unsigned char *bs = xs + (size_t)kParts * pairs * kPairBytes + 64;        // d x [A_i 0; 0 A_i] (hi)
    unsigned char *bl = bs + (size_t)d * kBf16B;                              // the lo parts (SPLIT)
    uint64_t *mbar = reinterpret_cast<uint64_t *>(bs + (size_t)kParts * d * kBf16B);  // MMA completion
    uint64_t *sbar = mbar + 1;                                                // staging completion
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbar + 2);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

    const long long nb = a.nb;
    TcWalk w{(long long)blockIdx.x * a.entries_per_chunk, a.entries_per_chunk};  // the entry being computed
    if (w.e >= nb) return;
    TcWalk w1 = w.next(a);  // the entry staged after it

    // first of all: the SM's next CTA starts only when this one has given up its right to allocate
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "n"(S::cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const uint32_t sbar_a = smem_u32(sbar);
    if (tid == S::copier) {  // the thread that uses the staging barrier before the others see it
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    TcPtrs<D> nxt;
    float fv[S::fac_slots] = {};  // factor elements of the entry staged last
    tc_load_ptrs<D>(nxt, a, w.e, tid);
    const bool bulk0 = tc_stage_async<D>(raw, fv, nxt, a, tid, sbar_a);
    if (w1.e < nb) tc_load_ptrs<D>(nxt, a, w1.e, tid);
    // while the first vector is on its way: operands zeroed once; fibres beyond F, the odd K
    // half of an unpaired tile and the off-diagonal blocks of the factor operands stay zero
    for (int v = tid + (F % (2 * kTileRows) == 0 ? (int)(kParts * pairs * kPairBytes + 64) / 16 : 0);
         v < (int)(kParts * pairs * kPairBytes + 64 + kParts * d * kBf16B) / 16; v += S::threads)
        reinterpret_cast<int4 *>(xs)[v] = make_int4(0, 0, 0, 0);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tacc = tmem + 16u * pairs;  // run accumulator after the mode output
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    const uint32_t mbar_a = smem_u32(mbar);
    const uint32_t xs_a = smem_u32(xs), bs_a = smem_u32(bs), xl_a = smem_u32(xl), bl_a = smem_u32(bl);
    const uint32_t leader = elect_lane();  // of each warp; warp 0's issues the MMAs
    uint32_t phase = 0, sphase = 0;
    bool failed = false;
    bool staging = true;  // a staging copy is in flight whose phase has not been waited for
    double *cur = nullptr;

    // run sum (TMEM accumulator) -> FP64 reductions into `dst`.  Fibre c of the last mode
    // holds output positions 8c + r; after an octet transpose lane l of octet o holds
    // positions 64o + 8j + l (o = c / 8), so every reduction instruction of a warp covers
    // 4 runs of 8 consecutive doubles.
    auto flush = [&](double *dst) {
        if (F < 8) {  // d = 1: one fibre, its 8 values are the whole output vector
            if (warp == 0) {
                float v[2][8];
                tmem_ld16(tacc, v[0], v[1]);  // warp-collective: the whole warp loads
                tmem_wait_ld(v);
                if (lane == 0)
#pragma unroll
                    for (int r = 0; r < 8; ++r) red_add_f64(dst + r, blk_out<double>(v[0][r]));
            }
            return;
        }
#pragma unroll
        for (int j = 0; j < pairs; ++j) {
            {
                float v[2][8];
                tmem_ld16(tacc + lane_base + 16u * j, v[0], v[1]);
                tmem_wait_ld(v);
                octet_transpose(v[0], lane);
                octet_transpose(v[1], lane);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int t = 2 * j + h;
                    const int c0 = t * kTileRows + warp * 32 + (lane & ~7);  // first fibre of the octet
                    if (c0 < F) {
                        double *p = dst + 8 * c0 + (lane & 7);
#pragma unroll
                        for (int r = 0; r < 8; ++r) red_add_f64(p + 8 * r, blk_out<double>(v[h][r]));
                    }
                }
            }
        }
    };

    bool ok = true;      // this warp's waits so far; the CTA agrees on it at the next barrier
    bool bulk = bulk0;   // how the entry being computed was staged
    for (; w.e < nb; w = w1, w1 = w.next(a)) {
        double *o = a.out[w.e];
        cp_async_wait_all();
        ok = ok && mbar_wait(sbar_a, sphase);  // the slot's bulk copy (or its empty phase)
        ok = __all_sync(0xffffffffu, ok);
        // a bulk copy is complete for whoever waited for it, copies by threads need a barrier;
        // the MMAs that read the operands are done for every thread (each waited for them)
        if (!bulk) __syncthreads();
        if (ok) {
            sphase ^= 1u;
            staging = false;
        }
        // factor operands: B_i[n][k] = A_i(n, k) in the upper-left and lower-right blocks
#pragma unroll
        for (int s = 0; s < S::fac_slots; ++s) {
            const int v = tid + s * S::threads;
            if (v < d * 64) {
                const int i = v >> 6, r = v & 7, k = (v >> 3) & 7;
                put<KIND_BF16>(bs + (size_t)i * kBf16B, r, k, fv[s]);
                put<KIND_BF16>(bs + (size_t)i * kBf16B, r + 8, k + 8, fv[s]);
                if constexpr (SPLIT) {
                    const float rem = fv[s] - __bfloat162float(__float2bfloat16_rn(fv[s]));
                    put<KIND_BF16>(bl + (size_t)i * kBf16B, r, k, rem);
                    put<KIND_BF16>(bl + (size_t)i * kBf16B, r + 8, k + 8, rem);
                }
            }
        }
        // vector operand: natural position p = fibre + F*K (K = the slowest index, mode 0,
        // contracted first), so 8 consecutive positions are 8 consecutive fibres of one K row
        if (d == 1) {
            if (tid < 8) {
                const __nv_bfloat16 h = __float2bfloat16_rn(raw[tid]);
                *reinterpret_cast<__nv_bfloat16 *>(xs + tid * 16) = h;
                if constexpr (SPLIT)
                    *reinterpret_cast<__nv_bfloat16 *>(xl + tid * 16) =
                        __float2bfloat16_rn(raw[tid] - __bfloat162float(h));
            }
        } else {
            const uint32_t fsh = 3u * (uint32_t)(d - 1);
#pragma unroll
            for (int q = tid; q < N / 8; q += S::threads) {
                // the two 16-byte halves in an order that keeps each 8-lane phase of the
                // 16-byte loads on 8 distinct bank slots
                const int h = (q >> 2) & 1;
                const float4 first = *reinterpret_cast<const float4 *>(raw + 8 * q + 4 * h);
                const float4 second = *reinterpret_cast<const float4 *>(raw + 8 * q + 4 * (h ^ 1));
                const float4 u = h ? second : first, w = h ? first : second;
                const uint32_t p0 = 8u * (uint32_t)q;
                const uint32_t off = mn_offset((p0 & (uint32_t)(F - 1)) >> 3, p0 >> fsh);
                if constexpr (SPLIT) {
                    const float v8[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
                    uint4 hi, lo;
                    split_bf16x8(v8, hi, lo);
                    *reinterpret_cast<uint4 *>(xs + off) = hi;
                    *reinterpret_cast<uint4 *>(xl + off) = lo;
                } else {
                    *reinterpret_cast<uint4 *>(xs + off) = pack_bf16x8(u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w);
                }
            }
        }
        // the run continues when this entry adds into the same output as the previous one;
        // otherwise the previous run's sum leaves TMEM before the last mode overwrites it
        const bool cont = o == cur && w.left < a.entries_per_chunk;
        if (!cont && cur != nullptr && ok) flush(cur);
        cur = o;
        fence_async_smem();  // the staging slot has been read (generic proxy) before the bulk copy refills it
        tc_fence_before();
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        if (w1.e < nb) {
            bulk = tc_stage_async<D>(raw, fv, nxt, a, tid, sbar_a);
            staging = true;
            const TcWalk w2 = w1.next(a);
            if (w2.e < nb) tc_load_ptrs<D>(nxt, a, w2.e, tid);
        }

        for (int i = 0; i < d; ++i) {  // modes 0, 1, ..., d-1
            const bool last = i == d - 1;
            if (warp == 0) {
                tc_fence_after();
                const uint32_t dst = last ? tacc : tmem;
                const uint32_t accumulate = (last && cont) ? 1u : 0u;
#pragma unroll
                for (int j = 0; j < pairs; ++j) {
                    const uint32_t dj = dst + 16u * (uint32_t)j;
                    const uint64_t xh = smem_desc(xs_a + j * kPairBytes, kMnLbo, kMnSbo), bh = smem_desc(bs_a + i * kBf16B);
                    mma<KIND_BF16>(leader, dj, xh, bh, accumulate);
                    if constexpr (SPLIT) {
                        mma<KIND_BF16>(leader, dj, smem_desc(xl_a + j * kPairBytes, kMnLbo, kMnSbo), bh, 1u);
                        mma<KIND_BF16>(leader, dj, xh, smem_desc(bl_a + i * kBf16B), 1u);
                    }
                }
                mma_commit(leader, mbar_a);
            }
            // uniform over the warp (the TMEM loads below are warp-collective), over the CTA at
            // the next barrier
            ok = __all_sync(0xffffffffu, mbar_wait(mbar_a, phase));
            phase ^= 1u;
            tc_fence_after();
            if (!last) {
                // fibre c = g + F/8 * kk with kk the next mode's index (c's top digit): the 8
                // new values become the 8 consecutive fibres 8g..8g+7 of the next operand
                const uint32_t sh = 3u * (uint32_t)(d - 2);
                float v[2 * pairs][8];
#pragma unroll
                for (int j = 0; j < pairs; ++j) tmem_ld16(tmem + lane_base + 16u * j, v[2 * j], v[2 * j + 1]);
                tmem_wait_ld(v);
#pragma unroll
                for (int t = 0; t < tiles; ++t) {
                    const int c = t * kTileRows + warp * 32 + lane;
                    if (c < F) {
                        const uint32_t kk = (uint32_t)c >> sh, g = (uint32_t)c & ((1u << sh) - 1u);
                        if constexpr (SPLIT) {
                            uint4 hi, lo;
                            split_bf16x8(v[t], hi, lo);
                            *reinterpret_cast<uint4 *>(xs + mn_offset(g, kk)) = hi;
                            *reinterpret_cast<uint4 *>(xl + mn_offset(g, kk)) = lo;
                        } else {
                            *reinterpret_cast<uint4 *>(xs + mn_offset(g, kk)) =
                                pack_bf16x8(v[t][0], v[t][1], v[t][2], v[t][3], v[t][4], v[t][5], v[t][6], v[t][7]);
                        }
                    }
                }
                fence_async_smem();
                tc_fence_before();
                if (__syncthreads_or(!ok)) {
                    failed = true;
                    break;
                }
            }
        }
        if (failed) break;
    }
    if (!ok || failed) {
        failed = true;
        if (lane == 0) atomicCAS(&g_tc_error, 0u, 1u);
    }
    cp_async_wait_all();
    // leaving early with a bulk copy still in flight: one more bounded wait for it, so
    // that it does not land in shared memory after this CTA is gone
    if (failed && staging) mbar_wait(sbar_a, sphase);
    if (cur != nullptr && !failed) flush(cur);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(S::cols) : "memory");
}

struct TcKernel {
    void (*fn)(const TcArgs);
    int threads, cols;
    size_t need;  // bytes of shared memory; 32 of them for two mbarriers and the TMEM address
};
template <int D> static TcKernel tc_kernel(int kind)
{
    using S = TcShape<D>;
    const size_t bf16 = (size_t)S::N * 4 + 64 + 32, part = S::pairs * kPairBytes + D * kBf16B;
    if (kind == KRONMULT_COMPUTE_BF16X3) return {fwd_tc_bf16_kernel<true, D>, S::threads, S::cols, bf16 + 2 * part};
    if (kind == KRONMULT_COMPUTE_BF16) return {fwd_tc_bf16_kernel<false, D>, S::threads, S::cols, bf16 + part};
    return {fwd_tc_kernel<D>, S::threads, S::cols, bf16 + (size_t)S::tiles * kTileBytes + 2 * D * kBBytes};
}

// Plans and enqueues the tensor-core forward.  Returns cudaErrorNotSupported for
// shapes it does not cover (n != 8, n^d > 4096), so that the caller can fall back.
int launch_tc_forward(int kind, int d, int n, const float *const *mats, int stride, const float *const *in,
                      double *const *out, long long nb, cudaStream_t st, const kronmult_tuning *tune)
{
    if (n != 8 || d < 1 || d > 4) return cudaErrorNotSupported;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return cudaErrorInvalidDevice;
    const DeviceInfo &di = device_info(dev);
    const TcKernel k = d == 1 ? tc_kernel<1>(kind) : d == 2 ? tc_kernel<2>(kind) : d == 3 ? tc_kernel<3>(kind) : tc_kernel<4>(kind);
    TcArgs a{};
    a.mats = mats;
    a.in = in;
    a.out = out;
    a.nb = nb;
    a.stride = stride;
    // resident CTAs per SM are limited so that their tensor-memory columns fit in 512
    // (or to tuning.ctas_per_sm when that is fewer): each CTA reserves 1/max_ctas of the
    // SM's shared memory (less the per-CTA system reservation), so at most max_ctas fit
    int max_ctas = 512 / k.cols;
    if (tune && tune->ctas_per_sm > 0 && tune->ctas_per_sm < max_ctas) max_ctas = tune->ctas_per_sm;
    size_t smem = (size_t)di.smem_per_sm / max_ctas - (size_t)di.smem_reserved_cta;
    smem &= ~(size_t)15;
    if (smem < k.need) smem = k.need;
    if (smem > (size_t)di.max_smem_optin) return cudaErrorNotSupported;
    const void *fn = (const void *)k.fn;
    if (!ensure_smem_attr(fn, smem) || !ensure_max_carveout(fn)) return cudaErrorInvalidValue;
    // run sums over chunks of 8 consecutive entries (the fan-in of a typical output group);
    // one wave of CTAs walks the chunks
    long long ept = (tune && tune->entries_per_team > 0) ? tune->entries_per_team : 8;
    if (ept > INT_MAX) ept = INT_MAX;
    a.entries_per_chunk = (int)ept;
    long long grid = (nb + ept - 1) / ept;
    const long long wave = (long long)di.sms * tmem_occupancy(fn, k.threads, smem, k.cols, di);
    // d = 4, more than two waves: a CTA per chunk.  CTAs that walk chunks leave the order of the
    // batch, and outputs with few entries then cost more in memory (56000 entries, TF32: 774 us
    // in one wave, 699 with a CTA per chunk for outputs of one entry, 377 and 356 for three,
    // 289.5 either way for eight; 8192 entries: 131 and 135, 73 and 75, 59 and 61)
    if (grid > wave && !(d == 4 && grid > 2 * wave)) grid = wave;
    k.fn<<<(unsigned)grid, k.threads, smem, st>>>(a);
    return (int)cudaGetLastError();
}

// Self-test of the bounded wait: an mbarrier that nothing ever arrives on is waited
// for with the kernels' own bounded wait (a short limit); the wait runs out, the
// kernel records code 1 in the device error word and returns, and the context stays
// usable.  No tensor memory, no copies in flight.
__global__ void wait_selftest_kernel()
{
    __shared__ uint64_t mbar;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const bool ok = mbar_wait(smem_u32(&mbar), 0, 1u << 12);
    if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicCAS(&g_tc_error, 0u, 1u);
}

}  // namespace kgb

extern "C" int kronmult_diag_wait_selftest(int *code)
{
    if (!code) return cudaErrorInvalidValue;
    *code = 0;
    const unsigned z = 0;
    cudaError_t e = cudaMemcpyToSymbol(kgb::g_tc_error, &z, sizeof z);
    if (e != cudaSuccess) return e;
    kgb::wait_selftest_kernel<<<1, 32>>>();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return e;
    unsigned v = 0;
    if ((e = cudaMemcpyFromSymbol(&v, kgb::g_tc_error, sizeof v)) != cudaSuccess) return e;
    *code = (int)v;
    return cudaMemcpyToSymbol(kgb::g_tc_error, &z, sizeof z);
}

extern "C" int kronmult_device_error(int *code, int clear)
{
    if (!code) return cudaErrorInvalidValue;
    unsigned v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, kgb::g_tc_error, sizeof v);
    if (e != cudaSuccess) return e;
    *code = (int)v;
    if (clear && v) {
        const unsigned z = 0;
        e = cudaMemcpyToSymbol(kgb::g_tc_error, &z, sizeof z);
    }
    return e;
}
