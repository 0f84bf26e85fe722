// FP32 adjoint in register blocks, n and d known at compile time (adj_kernels.cuh has the
// definitions of p_i, q_i and the gradients).
//
// The layouts are fwd_block_kernel's: vectors in natural order in shared memory, the axes in
// passes of M, whole blocks of n^M values per thread, E entries per group of warps.  The
// p-sweep goes down the passes (axes d-1 .. 1 on x), every pass writing its result to a
// buffer of its own; the q-sweep goes back up (axes 0 .. d-1, transposed factors, on the
// output gradient, in place).  On the way up a thread holds a block of q and rebuilds the
// block's p_i from the pass's input, so that for every axis i of the pass it adds
//     sum over its fibres f of  q_i[f, r] * p_i[f, k]
// to its own n x n partial of grad_A_i and then applies A_i^T to its q block.  The partials
// (d n^2 values per thread) live in tensor memory, over all consecutive entries whose
// factor gradients go to the same place; only at the end of such a run are they summed over
// the team's threads and added to the gradients.  Shared-memory traffic per entry: 2 reads
// and 1 write per pass on the way down and up, against 3 reads and 2 writes per mode with a
// reduction through shared memory per mode and entry in the fibre-mapped kernel.
//
// Measured against that kernel, 8 entries per factor set: d = 3, n = 6, 16384 entries 60 -> 31 us
// (shared-memory pipe 50 %, issue 47 %, FMA 26 %: two rounds of entries per CTA and their chain of
// passes); d = 4, n = 8, 3904 entries 532 -> 179 us; d = 2, n = 2, 100000 entries 31.5 -> 11.6;
// d = 3, n = 4, 100000 entries 84 -> 46.
#pragma once
#include "adj_kernels.cuh"
#include "block_kernels.cuh"

namespace kgb {

// y[k] = sum_r A(r, k) q[r] on the axis of stride ST of a thread's values, in place
template <int NN, int NX, int ST, int GB> __device__ __forceinline__ void blk_mode_t(float (&x)[NX], unsigned fac)
{
    constexpr int NF = NX / NN, P4 = (NN * NN + 3) / 4 * 4;
#pragma unroll
    for (int f0 = 0; f0 < NF; f0 += GB) {
        float y[GB][NN];
        float m[P4];
#pragma unroll
        for (int k = 0; k < NN; ++k) {
#pragma unroll
            for (int r = 0; r < NN; ++r) {
                const int j = k * NN + r;
                if (j % 4 == 0) blk_ld_factor(fac + 4u * j, m + j);
#pragma unroll
                for (int g = 0; g < GB; ++g) {
                    const int f = f0 + g;
                    if (f < NF) {
                        const float q = x[f / ST * ST * NN + f % ST + r * ST];
                        y[g][k] = r == 0 ? fmaf(m[j], q, 0.f) : fmaf(m[j], q, y[g][k]);
                    }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < GB; ++g) {
            const int f = f0 + g;
            if (f < NF) {
#pragma unroll
                for (int k = 0; k < NN; ++k) x[f / ST * ST * NN + f % ST + k * ST] = y[g][k];
            }
        }
    }
}

// part(r, k) += sum over the thread's fibres of q[f, r] c[f, k], on the axis of stride ST;
// part at tensor-memory columns col + r * NN + k, at most RB rows in registers at a time;
// from zero where `fresh`
template <int NN, int NX, int ST, int R0 = 0>
__device__ __forceinline__ void adj_contract(const float (&q)[NX], const float (&c)[NX], unsigned col, bool fresh,
                                             bool any_old)
{
    if constexpr (R0 < NN) {
        constexpr int NF = NX / NN, RB = NN <= 4 ? NN : (24 / NN > 0 ? 24 / NN : 1), RC = NN - R0 < RB ? NN - R0 : RB;
        float s[RC * NN];
        // this entry's part first, then the earlier ones': shorter chains of additions (d = 4,
        // n = 8, fan-in 8: error of the factor gradients 2.0e-7 -> 1.4e-7; d = 3, n = 6: 1.3e-7
        // -> 1.1e-7, 48.5 -> 50.1 us)
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const int b = f / ST * ST * NN + f % ST;
#pragma unroll
            for (int r = 0; r < RC; ++r)
#pragma unroll
                for (int k = 0; k < NN; ++k) {
                    const float qv = q[b + (R0 + r) * ST], cv = c[b + k * ST];
                    s[r * NN + k] = f == 0 ? qv * cv : fmaf(qv, cv, s[r * NN + k]);
                }
        }
        if (any_old) {
            float o[RC * NN];
            blk_tm_ld<RC * NN>(col + R0 * NN, o);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < RC * NN; ++j) asm volatile("" : "+f"(o[j]));  // no use before the wait
#pragma unroll
            for (int j = 0; j < RC * NN; ++j) s[j] += fresh ? 0.f : o[j];
        }
        blk_tm_st<RC * NN>(col + R0 * NN, s);
        adj_contract<NN, NX, ST, R0 + RC>(q, c, col, fresh, any_old);
    }
}

template <typename CF> struct AdjBlk {
    using B = Blk<CF>;
    static constexpr int P = CF::NN * CF::NN;
    static constexpr int VE = (B::EW * B::VS + 3) / 4 * 4;  // one vector of every team
    static constexpr int SLOT = 2 * VE + B::EW * B::FS;     // staged: x, output gradient, factors
    static constexpr int SCR = (B::passes - 1) * VE;        // inputs of the passes after the first
    static constexpr int RBF = P <= B::V0 ? CF::NN : B::V0 / CF::NN;  // rows of a partial reduced at a time
    static constexpr int per_thread = CF::D * P;  // a thread's partials
    static constexpr int cols_used = per_thread * ((B::threads + 127) / 128);
    static constexpr int cols = tmem_cols(cols_used);
    static_assert(CF::G == 1 && cols_used <= 512 && (B::EW == 1 || B::W == 1 || B::C == 1), "adjoint blocks");
};

template <typename CF> struct AdjSpot {  // where one thread's entry lies
    const float *x;
    float *q, *scr;  // scr: buffer k at scr + k * VE
    unsigned fac, tmem;
    int t, group;
    bool active, fresh, any_old, want_gA, want_gin;
};

template <typename CF, int P> __device__ __forceinline__ void adj_down(const AdjSpot<CF> &s)
{
    using B = Blk<CF>;
    using W = BlkPass<CF, P>;
    if constexpr (P + 1 < B::passes) {
        float x[B::V0];
        blk_load_pass<CF, P>(x, P == 0 ? s.x : s.scr + (P - 1) * AdjBlk<CF>::VE, s.t);
        blk_modes<CF, W::axes>(x, s.fac + 4u * B::P4 * (CF::D - 1 - W::first));
        if (s.active) blk_store_pass<CF, P>(x, s.scr + P * AdjBlk<CF>::VE, s.t);
        blk_sync<B::W, B::C>(s.group);
        adj_down<CF, P + 1>(s);
    }
}

// axes A, A - 1, .. 0 of pass P (stride n^A within a block) on the q block
template <typename CF, int P, int A> __device__ __forceinline__ void adj_axes(const AdjSpot<CF> &s, float (&q)[Blk<CF>::V0])
{
    using B = Blk<CF>;
    constexpr int NN = CF::NN, V0 = B::V0, ST = blk_pow(NN, A), top = CF::D - 1 - BlkPass<CF, P>::first;
    if (s.want_gA) {
        float c[V0];
        blk_load_pass<CF, P>(c, P == 0 ? s.x : s.scr + (P - 1) * AdjBlk<CF>::VE, s.t);
        if constexpr (A > 0) blk_modes<CF, A>(c, s.fac + 4u * B::P4 * top);
        adj_contract<NN, V0, ST>(q, c, s.tmem + (top - A) * NN * NN, s.fresh, s.any_old);
    }
    if (P > 0 || A > 0 || s.want_gin) blk_mode_t<NN, V0, ST, CF::GB>(q, s.fac + 4u * B::P4 * (top - A));
    if constexpr (A > 0) adj_axes<CF, P, A - 1>(s, q);
}

template <typename CF, int P> __device__ __forceinline__ void adj_up(const AdjSpot<CF> &s)
{
    using B = Blk<CF>;
    float q[B::V0];
    blk_load_pass<CF, P>(q, s.q, s.t);
    adj_axes<CF, P, BlkPass<CF, P>::axes - 1>(s, q);
    if (s.active) blk_store_pass<CF, P>(q, s.q, s.t);
    blk_sync<B::W, B::C>(s.group);
    if constexpr (P > 0) adj_up<CF, P - 1>(s);
}

// a.team_size teams per group, a.entries_per_team entries per team or one more,
// a.slices staging slots.
template <typename CF>
__global__ void __launch_bounds__(Blk<CF>::threads, Blk<CF>::ctas) adj_block_kernel(const AdjArgs<float> a)
{
    using B = Blk<CF>;
    using AB = AdjBlk<CF>;
    constexpr int NN = CF::NN, D = CF::D, P = NN * NN;
    constexpr int V0 = B::V0, T = B::T, N = B::N, VS = B::VS, FS = B::FS, EW = B::EW, W = B::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_tmem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = warp / W, gw = warp - group * W, grank = gw * 32 + lane;
    const int slots = a.slices;
    float *base = reinterpret_cast<float *>(smem_raw) + (size_t)group * (slots * AB::SLOT + AB::SCR);
    float *scr = base + slots * AB::SLOT;

    const int ew = a.team_size, share = a.entries_per_team;
    const long long teams = (long long)gridDim.x * (blockDim.x / (32 * W)) * ew;
    const long long team0 = ((long long)blockIdx.x * (blockDim.x / (32 * W)) + group) * ew;
    const long long more = a.nb - share * teams;
    auto first_of = [&](long long g) { return g * share + (g < more ? g : more); };
    auto count_of = [&](long long g) { return share + (g < more ? 1 : 0); };
    const int iters = share + (more > 0 ? 1 : 0);
    const bool want_gA = a.gmats != nullptr, want_gin = a.gin != nullptr;
    if (warp == 0) {
        if (want_gA) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(&s_tmem)),
                         "n"(AB::cols)
                         : "memory");
        }
        // the next CTA starts on this SM only now
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = want_gA ? s_tmem + ((unsigned)(warp & 3) << 21) + (unsigned)(warp >> 2) * AB::per_thread : 0u;

    const int team = grank / T, t = grank - team * T;
    const bool mine = team < ew;
    const int own = mine ? team : 0;
    const long long e0 = mine ? first_of(team0 + team) : 0;
    const int count = mine ? count_of(team0 + team) : 0;
    // pointers of the next entries to be copied, spread over the lanes: kind 0 x, 1 output
    // gradient, 2 + i factor i
    constexpr int KINDS = D + 2, K = 32 / EW < KINDS ? 32 / EW : KINDS, NPR = (KINDS + K - 1) / K;
    const int lteam = lane % EW, lkind = lane / EW;
    const long long l0 = first_of(team0 + lteam);
    const int lcount = lteam < ew ? count_of(team0 + lteam) : 0;
    const float *ptrs[NPR];
    auto load_ptrs = [&](int it) {
#pragma unroll
        for (int r = 0; r < NPR; ++r) {
            const int k = r * K + lkind;
            const bool has = it < lcount && lkind < K && k < KINDS;
            const float *const *src = k == 0   ? a.in + (l0 + it)
                                      : k == 1 ? a.gout + (l0 + it)
                                               : a.mats + ((l0 + it) * D + (k - 2));
            ptrs[r] = has ? *src : nullptr;
        }
    };
    auto ptr_of = [&](int kind, int j) {
        return reinterpret_cast<const float *>(
            __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(ptrs[kind / K]), kind % K * EW + j));
    };
    BlkFactorLanes<CF> fl(lane, a.stride);
    constexpr int pieces = B::shifted || B::copy16 ? (N + 6) / 4 : N;
    constexpr int GS = EW == 1 ? 32 * W : pieces > 16 ? 32 : pieces > 8 ? 16 : pieces > 4 ? 8 : 4;
    int shx = 0, shq = 0, nshx = 0, nshq = 0;  // shifts of this thread's own vectors, now and staged ahead
    auto copy_data = [&](int slot) {
        float *dst = base + (size_t)slot * AB::SLOT;
        const float *ox = ptr_of(0, EW == 1 || !mine ? 0 : team), *oq = ptr_of(1, EW == 1 || !mine ? 0 : team);
        if constexpr (EW == 1) {
            if (ox) {
                blk_copy_vec<B, GS>(dst, ox, grank);
                blk_copy_vec<B, GS>(dst + AB::VE, oq, grank);
            }
        } else {
#pragma unroll 1
            for (int j0 = 0; j0 < ew; j0 += 32 * W / GS) {
                const int j = j0 + grank / GS;
                const float *sx = ptr_of(0, j < ew ? j : 0), *sq = ptr_of(1, j < ew ? j : 0);
                if (j < ew && sx) {
                    blk_copy_vec<B, GS>(dst + j * VS, sx, lane % GS);
                    blk_copy_vec<B, GS>(dst + AB::VE + j * VS, sq, lane % GS);
                }
            }
        }
        fl.copy(dst + 2 * AB::VE, gw, ew, [&](int i, int j) { return ptr_of(2 + i, j); });
        nshx = B::shifted ? blk_shift(ox) : 0;
        nshq = B::shifted ? blk_shift(oq) : 0;
    };
    // where this entry's factor gradients go
    float *gm[D];
#pragma unroll
    for (int i = 0; i < D; ++i) gm[i] = want_gA && count > 0 ? a.gmats[e0 * D + i] : nullptr;

    bool fresh = true;
    load_ptrs(0);
    if (slots == 2) {
        copy_data(0);
        cp_async_commit();
        if (iters > 1) load_ptrs(1);
    }
    for (int it = 0; it < iters; ++it) {
        const int slot = slots == 2 ? it & 1 : 0;
        const bool active = it < count;
        float *const gi = want_gin && active ? a.gin[e0 + it] : nullptr;
        float *gm_next[D];
        bool last = false;  // the run of entries with these factor gradients ends here
        if (want_gA) {
            last = active && it + 1 >= count;
#pragma unroll
            for (int i = 0; i < D; ++i) {
                gm_next[i] = it + 1 < count ? a.gmats[(e0 + it + 1) * D + i] : nullptr;
                if (active && gm_next[i] != gm[i]) last = true;
            }
            // at most 32 entries in one chain of FP32 additions
            if (it % 32 == 31) last = active;
        }
        if (slots == 2) {
            cp_async_wait_all();
            blk_sync<W, B::C>(group);  // entry `it` staged, the other slot and the buffers free
            shx = nshx, shq = nshq;
            if (it + 1 < iters) {
                copy_data(slot ^ 1);
                cp_async_commit();
                if (it + 2 < iters) load_ptrs(it + 2);
            }
        } else {
            blk_sync<W, B::C>(group);
            copy_data(0);
            shx = nshx, shq = nshq;
            cp_async_commit();
            if (it + 1 < iters) load_ptrs(it + 1);
            cp_async_wait_all();
            blk_sync<W, B::C>(group);
        }
        float *xs = base + (size_t)slot * AB::SLOT, *qs = xs + AB::VE;
        AdjSpot<CF> s;
        s.x = xs + own * VS + shx;
        s.q = qs + own * VS + shq;
        s.scr = scr + own * VS;
        s.fac = (unsigned)__cvta_generic_to_shared(qs + AB::VE + own * FS);
        s.tmem = tmem;
        s.t = t;
        s.group = group;
        s.active = active;
        s.fresh = fresh;
        s.any_old = want_gA && __any_sync(0xffffffffu, active && !fresh);
        s.want_gA = want_gA;
        s.want_gin = want_gin;
        if (s.any_old) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        if (want_gA) adj_down<CF, 0>(s);
        adj_up<CF, B::passes - 1>(s);

        // q is K^T g: into the input gradient, lanes on consecutive values
        if (want_gin) {
            if constexpr (W == 1) {
                const unsigned long long to = (unsigned long long)reinterpret_cast<uintptr_t>(gi);
#pragma unroll 1
                for (int j = 0; j < ew; ++j) {
                    float *const dst = reinterpret_cast<float *>(__shfl_sync(0xffffffffu, to, j * T));
                    const float *const src = qs + j * VS + (B::shifted ? __shfl_sync(0xffffffffu, shq, j * T) : 0);
                    if (dst != nullptr) {
#pragma unroll
                        for (int p = lane; p < N; p += 32) atomic_add<float>(dst + p, src[B::phys(p)]);
                    }
                }
            } else if (gi != nullptr) {
#pragma unroll 4
                for (int p = t; p < N; p += T) atomic_add<float>(gi + p, s.q[B::phys(p)]);
            }
        }
        if (want_gA) {
            // the end of a run: sum the partials over the team's threads, through the q buffer
            bool flush;  // uniform over the group
            if constexpr (W > 1 && EW > 1)
                flush = __syncthreads_or(last);
            else
                flush = __any_sync(0xffffffffu, last);
            if (flush) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                blk_sync<W, B::C>(group);  // the q buffer's last reads are done
                // many teams of a warp whose runs end together and go to the same places: summed over
                // the teams, as a tree, before one addition (with one each the sums in memory had
                // 1.65 times the error at d = 2, n = 2, 100 entries per factor set, 50000 entries, and
                // took 14.4 us, now 8.9).  Up to 8 teams add by themselves: 10 % faster at 8 entries
                // per factor set.
                constexpr int kSteps = W > 1 || EW < 8 ? 0 : EW > 16 ? 5 : EW > 8 ? 4 : 3;
                bool head = true, with[kSteps + 1], merge = false;
                if constexpr (kSteps > 0) {
                    const int before = __shfl_up_sync(0xffffffffu, (int)last, T);  // all lanes take part
                    head = team == 0 || !last || !before;
#pragma unroll
                    for (int i = 0; i < D; ++i) {
                        const unsigned long long at = (unsigned long long)reinterpret_cast<uintptr_t>(gm[i]);
                        const unsigned long long prev = __shfl_up_sync(0xffffffffu, at, T);
                        head = head || prev != at;
                    }
                    const unsigned rest = __ballot_sync(0xffffffffu, head) >> (lane - t) >> T;  // heads of later teams
                    const int end = rest == 0 ? EW : team + 1 + (__ffs(rest) - 1) / T;
                    merge = __any_sync(0xffffffffu, mine && end - team >= (EW < 9 ? EW : 9));
#pragma unroll
                    for (int s = 0; s < kSteps; ++s) with[s] = mine && team + (1 << s) < end;
                }
#pragma unroll 1
                for (int i = 0; i < D; ++i) {
                    float *dst = nullptr;  // gm[i], selected without indexing registers
#pragma unroll
                    for (int m = 0; m < D; ++m) dst = m == i ? gm[m] : dst;
#pragma unroll 1
                    for (int r0 = 0; r0 < NN; r0 += AB::RBF) {
                        constexpr int NV = AB::RBF * NN;
                        float v[NV];
                        blk_tm_ld<NV>(tmem + i * P + r0 * NN, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = 0; j < NV; ++j) asm volatile("" : "+f"(v[j]));
                        float *const buf = qs + own * VS;
                        if (last) {
#pragma unroll
                            for (int j = 0; j < NV; ++j) buf[j * T + t] = v[j];
                        }
                        blk_sync<W, B::C>(group);
                        auto team_sum = [&](int j) {
                            constexpr int L = T >= 32 ? 8 : T >= 8 ? 4 : 1;  // independent partial sums
                            float sum[L];
#pragma unroll
                            for (int l = 0; l < L; ++l) sum[l] = buf[j * T + l];
#pragma unroll 1
                            for (int h = L; h + L <= T; h += L) {
#pragma unroll
                                for (int l = 0; l < L; ++l) sum[l] += buf[j * T + h + l];
                            }
#pragma unroll
                            for (int l = 0; l < L; ++l)
                                if (l < T % L) sum[l] += buf[j * T + T / L * L + l];
#pragma unroll
                            for (int w = L / 2; w > 0; w /= 2)
#pragma unroll
                                for (int l = 0; l < w; ++l) sum[l] += sum[l + w];
                            return sum[0];
                        };
                        auto place = [&](int j) { return dst + (r0 + j / NN) + (size_t)(j % NN) * a.gstride; };
                        if (!merge) {
                            if (last && dst != nullptr) {  // null: no gradient of this factor wanted
                                for (int j = t; j < NV; j += T) atomic_add<float>(place(j), team_sum(j));
                            }
                        } else {
#pragma unroll 1
                            for (int j0 = 0; j0 < NV; j0 += T) {
                                const int j = j0 + t;
                                const bool valid = last && dst != nullptr && j < NV;
                                float sum = valid ? team_sum(j) : 0.f;
#pragma unroll
                                for (int s = 0; s < kSteps; ++s) {
                                    const float other = __shfl_down_sync(0xffffffffu, sum, T << s);
                                    if (with[s]) sum += other;
                                }
                                if (valid && head) atomic_add<float>(place(j), sum);
                            }
                        }
                        blk_sync<W, B::C>(group);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < D; ++i) gm[i] = gm_next[i];
            fresh = last || (fresh && !active);
        }
    }
    if (want_gA) {
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "n"(AB::cols) : "memory");
        }
    }
}

struct AdjBlkInfo {
    const void *fn = nullptr;
    int n = 0, d = 0;  // of the instantiation
    int EW = 0, group = 0, groups = 0, slot_bytes = 0, scratch_bytes = 0, cols = 0;
};
template <typename CF> AdjBlkInfo adj_info_of()
{
    using B = Blk<CF>;
    using AB = AdjBlk<CF>;
    return AdjBlkInfo{(const void *)adj_block_kernel<CF>, CF::NN, CF::D, B::EW, 32 * B::W, B::C, AB::SLOT * 4, AB::SCR * 4, AB::cols};
}

// Axes per pass, fibres at once, warps per group, groups per CTA and CTAs per SM, by (n, d):
// the fastest of those that fit 255 registers and the 512 tensor-memory columns (d n^2 per
// thread and four warps).  n = 6, 7, d = 4: 7 and 5 entries share 8 warps (36 and 49 threads
// per entry leave 44 and 23 % of whole warps idle: 190 -> 120 us and 190 -> 135 us on 64 MB).
template <int NN, int D> struct AdjTune;
#define KGB_ADJ_TUNE(NN, M, GB, W, C, CTAS) \
    template <int D> struct AdjTune<NN, D> : BlkCfg<NN, D, M, 1, GB, W, C, CTAS> {};
KGB_ADJ_TUNE(2, (D >= 5 ? 3 : D >= 3 ? 2 : 1), (D >= 5 ? 4 : 2), 1, 4, 6)
KGB_ADJ_TUNE(3, (D >= 5 ? 3 : D >= 3 ? 2 : 1), (D >= 5 ? 9 : 3), 1, 4, (D >= 5 ? 4 : 6))
KGB_ADJ_TUNE(4, (D >= 5 ? 3 : D >= 3 ? 2 : 1), 4, 1, 4, (D >= 5 ? 2 : D >= 3 ? 4 : 6))
KGB_ADJ_TUNE(5, (D >= 3 ? 2 : 1), 5, 1, 4, (D >= 3 ? 3 : 5))
KGB_ADJ_TUNE(6, (D >= 3 ? 2 : 1), 3, (D >= 4 ? 8 : 1), (D >= 4 ? 1 : 4), (D >= 4 ? 1 : D == 3 ? 3 : 4))
KGB_ADJ_TUNE(7, (D >= 3 ? 2 : 1), 4, (D >= 4 ? 8 : 1), (D >= 4 ? 1 : D == 3 ? 8 : 4), (D >= 3 ? 1 : 4))
KGB_ADJ_TUNE(8, (D >= 3 ? 2 : 1), 4, 1, (D >= 4 ? 8 : 4), (D >= 4 ? 1 : D == 3 ? 2 : 3))
#undef KGB_ADJ_TUNE

// fn == nullptr where (n, d) has no instantiation
AdjBlkInfo adj_block_lookup(int n, int d);

// A launch's teams per group, groups per CTA and, from these, threads and shared memory:
// as in the forward's plan_block, with fewer groups where their shared memory (`max_smem`
// bytes at most) asks for it.
struct AdjBlkShape {
    long long ew = 0;
    int groups = 0;
    bool fits = false;
    int threads(const AdjBlkInfo &b) const { return groups * b.group; }
    size_t smem(const AdjBlkInfo &b, int slots) const { return (size_t)groups * (slots * b.slot_bytes + b.scratch_bytes); }
};
inline AdjBlkShape adj_block_shape(const AdjBlkInfo &b, long long nb, int sms, size_t max_smem)
{
    AdjBlkShape s;
    const long long spread = (long long)sms * 8 * 32 / b.group + 1;
    s.ew = (nb + spread - 1) / spread;
    if (s.ew > b.EW) s.ew = b.EW;
    s.groups = b.groups;
    while (s.groups > 1 && (long long)(s.groups / 2) * s.ew * sms >= nb) s.groups /= 2;
    while (s.groups > 1 && s.smem(b, 1) > max_smem) s.groups /= 2;
    s.fits = s.smem(b, 1) <= max_smem;
    return s;
}

}  // namespace kgb
