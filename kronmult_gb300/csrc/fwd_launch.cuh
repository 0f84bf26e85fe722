// Host-side launch planning for the forward kernels.
#pragma once
#include <climits>
#include <cstdint>
#include <mutex>
#include "block_kernels.cuh"
#include "column_kernels.cuh"
#include "dmma_kernels.cuh"
#include "f64_kernels.cuh"
#include "fwd_kernels.cuh"
#include "pair_kernels.cuh"
#include "kronmult_gb300.h"
#include "tuning.cuh"

namespace kgb {

// per-device properties, queried once
struct DeviceInfo {
    int sms = 0;
    int max_smem_optin = 0;      // bytes of dynamic shared memory one CTA may opt into
    int smem_per_sm = 0;         // bytes of shared memory per SM
    int smem_reserved_cta = 0;   // bytes the system reserves per resident CTA
};

const DeviceInfo &device_info(int dev);

// remembers which kernels have had their dynamic shared-memory limit raised
bool ensure_smem_attr(const void *fn, size_t smem);

// resident CTAs per SM for a kernel/launch shape (cached)
int occupancy(const void *fn, int block, size_t smem);

inline long long pow_ll(int b, int e)
{
    long long r = 1;
    for (int i = 0; i < e; ++i) {
        r *= b;
        if (r > (long long)INT_MAX) return (long long)INT_MAX + 1;
    }
    return r;
}

inline int round_up(int v, int m) { return (v + m - 1) / m * m; }

// host twin of FactorInSmem: an n x n factor of T does not fit the register path
template <typename T> inline bool FactorInSmemHost(int n) { return (size_t)n * n * sizeof(T) > 128; }

// Team size (power of two, 8..max_ts) for an element-mapped kernel over N outputs:
// the best lane utilisation N / (ts * ceil(N / ts)) with at most max_per outputs per
// thread; among teams within 2 % of the best, the one closest to 8 outputs per thread.
// `forced` > 0 fixes the size (grown until max_per holds).  Returns 0 if none fits.
inline int elem_team_size(int N, int max_per, int forced, int max_ts)
{
    if (forced > 0) {
        int ts = forced;
        while (ts < max_ts && (N + ts - 1) / ts > max_per) ts *= 2;
        return (N + ts - 1) / ts <= max_per ? ts : 0;
    }
    double best = -1.0;
    for (int c = 8; c <= max_ts; c *= 2) {
        const int per = (N + c - 1) / c;
        if (per <= max_per) {
            const double u = (double)N / ((double)per * c);
            if (u > best) best = u;
        }
    }
    int ts = 0, dist = 1 << 30;
    for (int c = 8; c <= max_ts; c *= 2) {
        const int per = (N + c - 1) / c;
        if (per > max_per) continue;
        const double u = (double)N / ((double)per * c);
        const int dd = per > 8 ? per - 8 : 8 - per;
        if (u >= best - 0.02 && dd < dist) {
            dist = dd;
            ts = c;
        }
    }
    return ts;
}

// Lane use of a mapping in which a team of ts threads covers `items` work items in
// rounds of ts (item = rank + j * ts), when the FP64 pipe is charged per warp
// instruction issued: in teams of a warp or more, a warp whose lanes all fall beyond
// `items` skips the round, so ceil(items / 32) warp rounds issue; sub-warp teams share
// a warp and each issues ceil(items / ts) rounds.
inline double lane_use(int items, int ts)
{
    if (ts >= 32) return (double)items / (32.0 * ((items + 31) / 32));
    return (double)items / ((double)ts * ((items + ts - 1) / ts));
}

// Margin by which the element mapping's lane use must beat the fibre mapping's before
// the FP64 planners take it (measured: equal lane use left the fibre kernels as fast or
// up to 16 % faster; d = 6, n = 3, 99 % against 95 %, is the closest case taken).
constexpr double kElemMargin = 0.03;

// FP64 mapping forced by kronmult_tuning::fp64_path: 3 = whole fibres per thread,
// 4 = one output element per thread (both on the FMA pipe); 0 otherwise.
inline int fp64_mapping(const kronmult_tuning *tune)
{
    const int p = tune ? tune->fp64_path : 0;
    return (p == 3 || p == 4) ? p : 0;
}

// largest power of two <= v (v >= 1)
inline int pow2_floor(long long v)
{
    int p = 1;
    while ((long long)p * 2 <= v) p *= 2;
    return p;
}

// A resolved forward launch.
template <typename T, typename TO> struct FwdPlan {
    FwdArgs<T, TO> args{};
    const void *fn = nullptr;
    bool smem_path = false;  // register in-place shared-memory kernel
    int use_smem = 0;        // generic kernel: shared-memory ping-pong
    dim3 grid, block;
    size_t smem = 0;
    const void *fn2 = nullptr;  // second launch (pass 2 of the two-pass path), same arguments
    dim3 grid2, block2;
    size_t smem2 = 0;
    bool columns = false;  // both passes in register blocks (launch_columns)
};

// Fibres per thread the two-pass path's pass-1 kernel is instantiated for, by n.
inline int split_qmax(int n) { return n <= 3 ? 8 : (n <= 7 ? 4 : 2); }

// Two-pass plan for vectors beyond shared memory (split_pass1/2_kernel): the
// largest fast part n^d1 one 256-thread team sweeps in registers, then tiles of
// L fast positions for pass 2.  Returns false where no split fits.
template <typename T, typename TO>
bool plan_split(FwdPlan<T, TO> &pl, const DeviceInfo &di)
{
    FwdArgs<T, TO> &a = pl.args;
    const int n = a.n, d = a.d;
    // FP64 stays on the one-vector global sweep: it is bound by the FP64 pipe, which
    // the two passes do not relieve (measured slower on n = 8, d = 6)
    if (sizeof(T) == 8 || n < 2 || n > 8 || d < 2 || !a.ws) return false;
    const int qm = split_qmax(n);
    constexpr int kAlign = 16 / (int)sizeof(T);
    for (int d1 = d - 1; d1 >= 1; --d1) {
        const long long C = pow_ll(n, d1), F1 = C / n, R = pow_ll(n, d - d1);
        if (F1 > 256LL * qm || R > 4096) continue;
        int ts = 8;
        while (ts < 256 && (long long)ts * qm < F1) ts *= 2;
        const int vpad = round_up((int)C, kAlign), fpad = round_up(d1 * n * n, kAlign);
        const int teams = 256 / ts;
        const size_t smem1 = (size_t)teams * 2 * (vpad + fpad) * sizeof(T);  // two staging slots
        auto f1 = split_pass1_lookup<T, TO>(n, qm);
        auto f2 = split_pass2_lookup<T, TO>(n);
        if (!f1 || !f2 || smem1 > (size_t)di.max_smem_optin) continue;
        // pass-2 tile: rows of at least 128 bytes and at least 256 (fibre, position)
        // tasks per mode, where two tiles fit in half the SM; else narrower (32 bytes
        // at least)
        const int fpad2 = round_up((d - d1) * n * n, kAlign);
        int L = 128 / (int)sizeof(T);
        while ((long long)L * (R / n) < 512 && L < 512) L *= 2;
        while (L > 32 / (int)sizeof(T) &&
               (4 * R * L + 2 * fpad2) * (long long)sizeof(T) > (long long)di.max_smem_optin / 2)
            L /= 2;
        const size_t smem2 = (size_t)(4 * R * L + 2 * fpad2) * sizeof(T);
        if (smem2 > (size_t)di.max_smem_optin) return false;
        const long long tiles = (C + L - 1) / L;
        // pass 2 sums runs of up to 64 consecutive entries per CTA while leaving ~16
        // CTAs per SM
        long long ept2 = a.nb * tiles / (16LL * di.sms);
        if (ept2 > 64) ept2 = 64;
        if (ept2 < 1) ept2 = 1;
        // pass 1: up to 8 chunks per team while leaving ~8 CTAs per SM
        long long ept1 = a.nb * R / ((long long)teams * di.sms * 8);
        if (ept1 > 8) ept1 = 8;
        if (ept1 < 1) ept1 = 1;
        const long long per_cta1 = (long long)teams * ept1;
        const long long grid1 = (a.nb * R + per_cta1 - 1) / per_cta1, grid2 = (a.nb + ept2 - 1) / ept2 * tiles;
        if (grid1 > INT_MAX || grid2 > INT_MAX) return false;
        if (!ensure_smem_attr((const void *)f1, smem1) || !ensure_smem_attr((const void *)f2, smem2)) return false;
        a.team_size = ts;
        a.teams_per_cta = teams;
        a.entries_per_team = (int)ept2;  // pass 2 only; pass 1 runs one chunk per team
        a.team_elems = 2 * (vpad + fpad);
        a.vec_pad = vpad;
        a.fac_pad = fpad;
        a.prefetch = 1;
        a.split_ept1 = (int)ept1;
        a.split_d1 = d1;
        a.split_C = (int)C;
        a.split_R = (int)R;
        a.split_L = L;
        pl.fn = (const void *)f1;
        pl.smem_path = true;
        pl.grid = dim3((unsigned)grid1);
        pl.block = dim3((unsigned)(teams * ts));
        pl.smem = smem1;
        pl.fn2 = (const void *)f2;
        pl.grid2 = dim3((unsigned)grid2);
        pl.block2 = dim3(256);
        pl.smem2 = smem2;
        return true;
    }
    return false;
}

// Gives a kernel that allocates tensor memory the SM's whole shared memory.  The runtime
// sizes the shared-memory carve-out for the occupancy it computes, and that is one CTA per
// SM for such kernels: left alone, they run one CTA at a time unless an earlier kernel left
// a larger carve-out behind (d = 4, n = 4, 5000 entries: 3.8 instead of 14.3 warps per SM).
bool ensure_max_carveout(const void *fn);

// Resident CTAs per SM of a kernel that holds `cols` tensor-memory columns per CTA: the
// occupancy call answers 1 for every kernel that allocates tensor memory.
int tmem_occupancy(const void *fn, int block, size_t smem, int cols, const DeviceInfo &di);

// Both passes in register blocks (column_kernels.cuh), for the vectors plan_split takes and
// pl holds its plan of.  Faster at every shape and batch measured (us, plan_split's kernels /
// these): n = 8, d = 6 19.9 / 14.0 at 8 entries, 4954 / 2746 at 3905; n = 7, d = 6 2646 / 1507
// at 3000; n = 8, d = 5 18.0 / 13.9 at 60; n = 2, d = 16 2237 / 725 at 3500.
template <typename T, typename TO> bool plan_columns(FwdPlan<T, TO> &pl, const DeviceInfo &di)
{
    if constexpr (sizeof(T) != 4) {
        return false;
    } else {
        FwdArgs<T, TO> &a = pl.args;
        const int d1 = a.d - col_axes(a.n);
        const BlkInfo u = d1 > 0 ? units_lookup(a.n, d1) : BlkInfo{};
        const ColInfo c = col_lookup<TO>(a.n);
        if (!u.fn || !c.fn) return false;
        const long long C = pow_ll(a.n, d1), R = a.N / C, tiles = (C + 31) / 32;
        const size_t smem1 = (size_t)u.groups * 2 * u.slot_bytes;
        if (a.nb > INT_MAX / (R > tiles ? R : tiles) || smem1 > (size_t)di.max_smem_optin ||
            c.smem > di.max_smem_optin || !ensure_smem_attr(u.fn, smem1) || !ensure_smem_attr(c.fn, c.smem) ||
            !ensure_max_carveout(c.fn))
            return false;
        const int block1 = u.groups * u.group, occ1 = occupancy(u.fn, block1, smem1);
        const int occ2 = tmem_occupancy(c.fn, c.block, c.smem, c.cols, di);
        if (occ1 < 1) return false;
        // FP64 outputs: the run sums (in FP32) that plan_split's pass 2 forms
        a.chunk_len = sizeof(TO) == 8 ? a.entries_per_team : 1;
        a.chunks = tiles * ((a.nb + a.chunk_len - 1) / a.chunk_len);
        const long long units = a.nb * R, per = (long long)u.groups * u.EW, warps = c.block / 32;
        const long long grid1 = (units + per - 1) / per, grid2 = (a.chunks + warps - 1) / warps;
        a.split_d1 = d1;
        a.split_C = (int)C;
        a.split_R = (int)R;
        a.team_size = u.EW;
        a.teams_per_cta = (int)per;
        pl.columns = true;
        pl.fn = u.fn;
        pl.grid = dim3((unsigned)(grid1 < (long long)di.sms * occ1 ? grid1 : di.sms * occ1));
        pl.block = dim3((unsigned)block1);
        pl.smem = smem1;
        pl.fn2 = c.fn;
        pl.grid2 = dim3((unsigned)(grid2 < (long long)di.sms * occ2 ? grid2 : di.sms * occ2));
        pl.block2 = dim3((unsigned)c.block);
        pl.smem2 = (size_t)c.smem;
        a.entries_per_team = (int)(a.chunks / (pl.grid2.x * warps));
        return true;
    }
}

// Whether an FP64 forward of factor size n runs on the FP64 tensor path: forced by
// tuning->fp64_path == 2, automatic (0) for n = 16 only, where the FMA pipe has only the
// generic run-time-n kernel (n <= 8 has compile-time-n FMA kernels, and n = 9..15 fill
// the 8 x 8 MMA tile too poorly: both measured faster on the FMA pipe).
inline bool dmma_wanted(int n, const kronmult_tuning *tune)
{
    const int path = tune ? tune->fp64_path : 0;
    if (!dmma_has_n(n)) return false;
    return path == 2 || (path == 0 && n == 16);
}

// FP64 tensor-path plan (fwd_dmma_kernel): one entry per team of W warps, each warp
// QT tiles of 8 fibres (W * QT * 8 >= F, at most 8 tiles per warp), the vector and the
// factors in shared memory.  False where no instantiation or shared-memory size fits.
template <typename T, typename TO>
bool plan_dmma(FwdPlan<T, TO> &pl, const DeviceInfo &di, const kronmult_tuning *tune)
{
    if constexpr (sizeof(T) != 8 || sizeof(TO) != 8) {
        return false;
    } else {
        FwdArgs<T, TO> &a = pl.args;
        const int n = a.n, d = a.d, N = a.N;
        if (d < 1 || !dmma_wanted(n, tune)) return false;
        const int F = N / n, tiles = (F + 7) / 8;
        int W = 1;
        while (W < 8 && W * 8 < tiles) W *= 2;
        const int per = (tiles + W - 1) / W;
        int qt = 1;
        while (qt < per) qt *= 2;
        const bool full = F % 8 == 0 && tiles == W * qt;
        DmmaFn fn = fwd_dmma_lookup(n, qt, full);
        if (!fn) return false;
        const int vpad = round_up(N, 2), fpad = round_up(d * n * n, 2);
        const int team_elems = vpad + fpad, ts = 32 * W;
        int teams = 256 / ts;
        while (teams > 1 && (size_t)teams * team_elems * sizeof(T) > (size_t)di.max_smem_optin) teams /= 2;
        const size_t smem = (size_t)teams * team_elems * sizeof(T);
        if (smem > (size_t)di.max_smem_optin || !ensure_smem_attr((const void *)fn, smem)) return false;
        const long long grid = (a.nb + teams - 1) / teams;
        if (grid > INT_MAX) return false;
        a.team_size = ts;
        a.teams_per_cta = teams;
        a.entries_per_team = 1;
        a.team_elems = team_elems;
        a.vec_pad = vpad;
        a.fac_pad = fpad;
        a.prefetch = 0;
        pl.fn = (const void *)fn;
        pl.smem_path = true;
        pl.grid = dim3((unsigned)grid);
        pl.block = dim3((unsigned)(teams * ts));
        pl.smem = smem;
        return true;
    }
}

// Whole fibres per thread, a team's consecutive entries summed in registers
// (fwd_smem_kernel): ts threads per team, at most qmax fibres per thread.
template <typename T, typename TO>
bool plan_runs(FwdPlan<T, TO> &pl, const DeviceInfo &di, const kronmult_tuning *tune, int ts, int qmax)
{
    FwdArgs<T, TO> &a = pl.args;
    const int n = a.n, d = a.d, N = a.N;
    const int vpad = round_up(N, 16 / (int)sizeof(T));
    const int fpad = round_up(d * n * n, 16 / (int)sizeof(T));
    // two staging slots (asynchronous prefetch of the next entry) unless disabled
    // or too large for half of the SM's shared memory; FP32 with factors in
    // shared memory (n >= 6) ping-pongs between vector buffers instead (three
    // vector buffers, two factor slots)
    int prefetch = (tune && tune->prefetch == 1) ? 0 : 1;
    if ((size_t)2 * (vpad + fpad) * sizeof(T) > (size_t)di.max_smem_optin / 2) prefetch = 0;
    const bool pp_ok = FactorInSmemHost<T>(n) && (size_t)(3 * vpad + 2 * fpad) * sizeof(T) <=
                                                     (size_t)di.max_smem_optin / 2;
    // default for FP32 into FP32 outputs (measured 1.5-4.5 % faster on n = 6, 8);
    // with FP64 outputs the in-place slots measured faster
    if (pp_ok && ((tune && tune->prefetch == 3) ||
                  (sizeof(T) == 4 && sizeof(TO) == 4 && (!tune || tune->prefetch == 0))))
        prefetch = 3;
    const int team_elems = prefetch == 3 ? 3 * vpad + 2 * fpad : (prefetch ? 2 : 1) * (vpad + fpad);
    const size_t team_bytes = (size_t)team_elems * sizeof(T);
    int block = ts >= 256 ? ts : 256;
    int teams = block / ts;
    // named barriers 1..15 limit the number of multi-warp teams per CTA
    while (ts >= 64 && ts < block && teams > 15) {
        block /= 2;
        teams = block / ts;
    }
    while (teams > 1 && (size_t)teams * team_bytes > (size_t)di.max_smem_optin) {
        block /= 2;
        teams = block / ts;
    }
    if (block < 32) block = 32, teams = block / ts;
    const size_t smem = (size_t)teams * team_bytes;
    if (smem <= (size_t)di.max_smem_optin) {
        auto fn = fwd_smem_lookup<T, TO>(n, qmax);
        if (fn && ensure_smem_attr((const void *)fn, smem)) {
            int per_sm = (tune && tune->ctas_per_sm > 0) ? tune->ctas_per_sm
                                                         : occupancy((const void *)fn, block, smem);
            if (per_sm < 1) per_sm = 1;
            const long long total_teams = (long long)di.sms * per_sm * teams;
            long long ept = (tune && tune->entries_per_team > 0) ? tune->entries_per_team : 8;
            if (ept * total_teams > a.nb * 2) ept = (a.nb + total_teams - 1) / total_teams;  // small batches
            if (ept < 1) ept = 1;
            if (ept > INT_MAX) ept = INT_MAX;
            const long long per_cta = ept * teams;
            const long long grid = (a.nb + per_cta - 1) / per_cta;
            if (grid <= INT_MAX) {
                a.team_size = ts;
                a.teams_per_cta = teams;
                a.entries_per_team = (int)ept;
                a.team_elems = team_elems;
                a.vec_pad = vpad;
                a.fac_pad = fpad;
                a.prefetch = prefetch;
                pl.fn = (const void *)fn;
                pl.smem_path = true;
                pl.grid = dim3((unsigned)grid);
                pl.block = dim3((unsigned)block);
                pl.smem = smem;
                return true;
            }
        }
    }
    return false;
}

// Team size (threads per entry) of the fibre kernels over F fibres: the smallest team that
// leaves every thread at most ~2-4 fibres (4 for FP64 n = 6 too: smaller teams keep more
// entries in flight, measured 5-34 % faster on d = 2..4).
template <typename T> inline int fibre_team(int n, int F)
{
    const int qtarget = (n <= 4 || (n == 6 && sizeof(T) == 8)) ? 4 : 2;
    int ts = 8;
    while (ts < 512 && (long long)ts * qtarget < F) ts *= 2;
    return ts;
}

// Chunks of the register-block path with FP64 outputs: run sums are kept in FP32 over at
// most 8 consecutive entries (fewer in small batches; none for n > 8) and added in FP64, so
// the chunks, and with them the FP32 sums, are fixed by (n, d, batch) alone.  R: teams per
// SM that the chunk length of a small batch spreads over.
template <typename TO> bool block_chunks(FwdArgs<float, TO> &a, const DeviceInfo &di, const kronmult_tuning *tune)
{
    const int n = a.n, d = a.d;
    const int forced = tune && tune->entries_per_team > 1 ? tune->entries_per_team : 0;
    const int ctas = tune && tune->ctas_per_sm > 0 ? tune->ctas_per_sm : 0;
    long long len = 1;
    if (n <= 8) {
        int teams = 0, per_sm = 0;  // per CTA, CTAs per SM
        if (n == 8 && (d == 3 || d == 4)) {
            teams = d == 3 ? 8 : 1;
            per_sm = 3;
        } else if (n == 4 && d >= 2 && d <= 5) {
            int ts = 8;
            while (ts < 256 && ts < a.N / (n * n)) ts *= 2;
            teams = 256 / ts;
            per_sm = 3;
        }
        if (teams > 0) {
            const long long R = (long long)di.sms * (ctas ? ctas : per_sm) * teams;
            len = forced ? forced : 8;
            if (len * R > a.nb * 2) len = (a.nb + R - 1) / R;
        } else {
            FwdPlan<float, TO> p;
            p.args = a;
            const int F = a.N / n, ts = fibre_team<float>(n, F), q = (F + ts - 1) / ts;
            int qmax = 1;
            while (qmax < q) qmax *= 2;
            if (qmax > (n <= 4 ? 8 : 4) || !plan_runs<float, TO>(p, di, tune, ts, qmax)) return false;
            len = p.args.entries_per_team;
        }
    }
    if (len > INT_MAX) return false;
    a.chunk_len = (int)len;
    a.chunks = (a.nb + len - 1) / len;
    return true;
}

// Where the other FP32 kernels measured faster than the register blocks: [from, to) entries.
// Most lie where a batch is a few waves of small teams and their uneven last one costs what
// the blocks save, or just beyond a whole number of waves.  Figures: us there / in register
// blocks at the entries named, one output per entry and (after the semicolon) one per 8
// entries.  Left as they are: batches where one entry per output loses what more gain (FP64
// outputs, d = 3, n = 7, 60000 entries 129 / 172 at one, 1.23 times as fast at eight): the host
// cannot tell them apart.
struct BlkSlower {
    int n, d;
    long long from, to;
};
constexpr BlkSlower kBlkSlowerF32[] = {
    {2, 1, 0, 400000},     // 9.7 / 11.7 at 150000, 16.9 / 17.9; 16.0 / 15.6 at 300000
    {2, 2, 0, 120000},     // 7.4 / 8.7; 6.8 / 7.2 at 70000, 12.8 / 12.4; 11.9 / 10.7 at 150000
    {2, 3, 0, 50000},      // 5.9 / 6.9; 5.6 / 6.0 at 30000, 9.6 / 8.9 at 70000
    {3, 1, 0, 50000},      // 3.5 / 4.5; 4.1 / 4.2 at 12000, 8.5 / 8.5; 8.3 / 7.6 at 70000
    {4, 1, 0, 120000},     // 7.3 / 9.1; 7.2 / 8.1 at 70000, 12.8 / 12.8; 11.8 / 11.1 at 150000
    {5, 1, 0, 200000},     // 9.8 / 11.2; 9.5 / 10.1 at 70000, 30.6 / 28.8; 28.9 / 22.3 at 300000
    {6, 1, 0, 50000},      // 7.5 / 8.5; 7.4 / 7.6 at 30000, 13.2 / 11.9 at 70000
    {3, 2, 2000, 20000},   // 4.7 / 5.2; 4.5 / 4.7 at 12000
    {7, 2, 2000, 50000},   // 6.9 / 8.0; 6.9 / 7.8 at 12000, just beyond two waves 9.1 / 11.3; 8.9 / 10.4 at 40000
    {2, 5, 38900, 45000},  // just beyond one wave: 7.9 / 9.9; 7.4 / 9.4 at 40000
    {2, 6, 0, 25000},      // 6.9 / 8.2; 6.6 / 7.7 at 20000
    {3, 3, 2000, 20000},   // 5.1 / 6.0; 5.3 / 5.5 at 12000
    {5, 3, 3000, 25000},   // 6.4 / 7.9; 6.4 / 7.6 at 5000
    {6, 3, 1000, 8000},    // 6.0 / 7.6; 6.0 / 7.2 at 3000
    {7, 3, 2500, 4000},    // 8.9 / 10.6; 8.9 / 10.2 at 3000
    {7, 3, 9700, 10800},   // just beyond one wave: 0.89 of the speed there at 10000
    {7, 4, 0, 500},        // few threads per entry: 5.4 / 6.4 at 48
    {8, 4, 0, 1100},       // 14.5 / 15.1 at 1000, 31.8 / 22.1 at 2500
    {4, 3, 7800, 9800},    // 5.8 / 6.4; 5.8 / 6.1 at 9000
    {4, 4, 5900, 14500},   // 10.3 / 10.8; 9.3 / 10.8 at 12000, 13.5 / 11.3 at 15000
    {4, 4, 19500, 21500},  // just beyond two waves: 13.7 / 15.4; 12.3 / 14.3 at 20000
    {4, 6, 0, 2500},       // 10.5 / 13.8 at 1000, 40.5 / 38.4 at 6000
};
// FP64 outputs: chunks of 6-8 entries leave a wave's last teams uneven as well
constexpr BlkSlower kBlkSlowerF64[] = {
    {3, 2, 0, 200000},     // 4.6 / 5.3; 4.5 / 5.2 at 12000, 48.7 / 54.9; 45.9 / 33.5 at 300000
    {5, 3, 3000, 40000},   // 7.3 / 8.3; 7.4 / 8.4 at 5000
    {5, 3, 116000, 140000},  // just beyond one wave: 0.81 of the speed; 1.03 at 120000
    {6, 3, 2000, 25000},   // 11.8 / 13.0; 9.4 / 10.7 at 5000
    {7, 3, 2500, 6000},    // 9.9 / 10.8; 10.1 / 11.0 at 3000
    {8, 3, 2500, 18000},   // 17.9 / 20.3; 15.0 / 15.9 at 5000
    {6, 4, 0, 200},        // 5.6 / 5.9; 5.4 / 5.8 at 100
    {7, 4, 0, 500},        // few threads per entry
    {8, 4, 0, 4000},       // 33.4 / 37.1 at 2500, 56.3 / 53.6 at 6000
    {8, 4, 7300, 9500},    // just beyond one wave: 0.84 of the speed; 0.86 at 8000
    {4, 4, 77900, 90000},  // just beyond one wave: 0.91 of the speed; 0.85 at 80000
    {4, 5, 4000, 9500},    // two entries per output, 5000: 20.8 / 24.8
};
// No instantiation, for the same reason: n = 6, d = 2 (39.5 / 41.7 at 200000) and, of FP64
// outputs, d = 1 with n <= 7 (n = 7: 52.3 / 58.5; 44.4 / 39.6 at 300000, 9.0 / 9.7; 8.5 / 8.8
// at 30000), d = 3, n = 3 (9.8 / 10.9; 9.2 / 10.0 at 30000, 86 / 104; 76 / 85 at 400000),
// d = 6, n = 4 (183 / 193 at 30000) and n = 2.
template <typename TO> inline bool block_slower(int n, int d, long long nb)
{
    auto in = [&](const auto &list) {
        for (const BlkSlower &s : list)
            if (s.n == n && s.d == d && nb >= s.from && nb < s.to) return true;
        return false;
    };
    if (n == 2 && nb < 20000) return true;  // d = 6: 3.9 / 4.9 at 6000, 10.5 / 8.9 at 30000
    return sizeof(TO) == 4 ? in(kBlkSlowerF32) : in(kBlkSlowerF64);
}

// FP32 register-block plan (fwd_block_kernel) where (n, d) has an instantiation.
template <typename T, typename TO>
bool plan_block(FwdPlan<T, TO> &pl, const DeviceInfo &di, const kronmult_tuning *tune)
{
    if constexpr (sizeof(T) != 4) {
        return false;
    } else {
        FwdArgs<T, TO> &a = pl.args;
        // a forced team size or one entry per team selects the one-mode-per-step kernels
        if (tune && (tune->team_size > 0 || tune->entries_per_team == 1 || tune->prefetch == 3)) return false;
        const BlkPair both = blk_lookup<TO>(a.n, a.d);
        if (!both.large.fn) return false;
        if (block_slower<TO>(a.n, a.d, a.nb)) return false;
        BlkInfo b = both.large;
        if (both.small.fn) {
            // one fibre per thread while its groups fill at most one wave of CTAs (n = 8,
            // d = 3: 3.2 against 5.2 us at 200 entries, 13.1 against 10.8 us at 5000)
            const BlkInfo &s = both.small;
            const int occ = tmem_occupancy(s.fn, s.groups * s.group, (size_t)s.groups * s.slot_bytes, s.cols, di);
            if (a.nb <= (long long)di.sms * occ * s.groups * s.EW) b = s;
        }
        if (!ensure_max_carveout(b.fn)) return false;
        if constexpr (sizeof(TO) == 8) {
            if (!block_chunks<TO>(a, di, tune)) return false;
        } else {
            a.chunks = a.nb;
            // FP32 run sums as long as the kernels below form them
            a.chunk_len = tune && tune->entries_per_team > 1 ? tune->entries_per_team : a.n == 4 && a.d == 6 ? 6 : 8;
        }
        // about 8 warps per SM before groups get more than one team (a group copies and adds for
        // its teams one after another; more warps cost more than they save at 5000 entries),
        // and CTAs of fewer groups where that leaves SMs without one
        const long long spread = (long long)di.sms * 8 * 32 / b.group + 1;
        long long ew = (a.chunks + spread - 1) / spread;
        if (ew > b.EW) ew = b.EW;
        int groups = b.groups;
        while (groups > 1 && (long long)(groups / 2) * ew * di.sms >= a.chunks) groups /= 2;
        const int block = groups * b.group;
        auto smem_of = [&](int slots) { return (size_t)groups * slots * b.slot_bytes; };
        if (smem_of(1) > (size_t)di.max_smem_optin || !ensure_smem_attr(b.fn, smem_of(1))) return false;
        int slots = 1, occ = tmem_occupancy(b.fn, block, smem_of(1), b.cols, di);
        if (a.nb > (long long)di.sms * occ * groups * b.EW || (sizeof(TO) == 8 && a.chunk_len > 1)) {
            // a second slot (the next entries copied while the current ones are computed)
            // unless it halves the resident warps
            if (smem_of(2) <= (size_t)di.max_smem_optin && ensure_smem_attr(b.fn, smem_of(2))) {
                const int occ2 = tmem_occupancy(b.fn, block, smem_of(2), b.cols, di);
                if (tune && tune->prefetch > 0 ? tune->prefetch == 2 : 2 * occ2 > occ) slots = 2;
                if (slots == 2) occ = occ2;
            }
        }
        if (tune && tune->ctas_per_sm > 0 && tune->ctas_per_sm < occ) occ = tune->ctas_per_sm;
        // one wave of CTAs with equal shares of the chunks
        const long long per_cta = groups * ew, wave = (long long)di.sms * occ;
        long long grid = (a.chunks + per_cta - 1) / per_cta;
        if (tune && tune->entries_per_team > 1 && sizeof(TO) == 4) {
            grid = (grid + tune->entries_per_team - 1) / tune->entries_per_team;
        } else if (grid > wave) {
            // or, large vectors, of at most nine tenths of them (FP32 outputs: eight); the rest goes in
            // small shares to CTAs that follow as SMs come free.  (One entry per output is bound by DRAM, which serves
            // SMs unequally: d = 6, n = 4, 60000 entries 493 -> 437 us, and 311 -> 314 at eight per
            // output, 36864 entries 306 -> 275 and 196 -> 200; FP64 outputs, d = 4, n = 8, 36864 543
            // -> 473 and 268 -> 248.  FP32 outputs, d = 4, n = 8: from 32 entries per team on; below,
            // 15000 entries at eight per output 59 / 63.)  Shares
            // of whole chunks, FP32 outputs as well: their run sums are then cut where the kernels
            // below cut them.
            const long long teams = wave * per_cta, len = sizeof(TO) == 8 ? 1 : a.chunk_len;
            const long long share = a.chunks * (sizeof(TO) == 8 ? 9 : 8) / (10 * teams) / len * len, rest = a.chunks - share * teams;
            const long long least = sizeof(TO) == 4 && a.n == 8 ? 3 * len : len;
            grid = wave;
            if (b.guided && a.chunk_len > 1 && share >= least && !(tune && tune->ctas_per_sm > 0)) {
                const long long rounds = (rest + teams * len - 1) / (teams * len);
                const long long later = sizeof(TO) == 8 ? 1 : (rest + teams * rounds - 1) / (teams * rounds);
                a.first_ctas = (int)wave;
                a.entries_per_team = (int)share;
                a.later_share = (int)later;
                grid += (rest + later * per_cta - 1) / (later * per_cta);
            }
        }
        const long long teams = grid * per_cta, most = a.first_ctas > 0 ? a.entries_per_team : a.chunks / teams + 1;
        if (grid > INT_MAX || most > INT_MAX / (sizeof(TO) == 8 ? a.chunk_len : 1)) return false;
        if (a.first_ctas == 0) a.entries_per_team = (int)(a.chunks / teams);
        a.team_size = (int)ew;
        a.teams_per_cta = (int)(groups * ew);
        a.prefetch = slots == 2;
        pl.fn = b.fn;
        pl.smem_path = true;
        pl.grid = dim3((unsigned)grid);
        pl.block = dim3((unsigned)block);
        pl.smem = smem_of(slots);
        return true;
    }
}

// FP64 short-vector plan (fwd_f64_kernel; n^d <= 2048).  Against the kernels below it at the
// same shapes (us there / here): d = 3, n = 4 8.6 / 3.3 at 16 entries, 11.0 / 4.1 at 1000,
// 275 / 270 at 200000; d = 4, n = 6 38.5 / 11.2 at 16, 461 / 437 at 8192; d = 3, n = 10 468 /
// 419 at 8192; d = 1, n = 10 426 / 94 at 200000.  (With 1024 threads for n^d up to 4096 it was
// slower: d = 6, n = 4, 3000 entries 512 / 595.)
template <typename T, typename TO>
bool plan_f64(FwdPlan<T, TO> &pl, const DeviceInfo &di, const kronmult_tuning *tune)
{
    if constexpr (sizeof(T) != 8 || sizeof(TO) != 8) {
        return false;
    } else {
        FwdArgs<T, TO> &a = pl.args;
        const F64Info f = f64_lookup(a.n, a.d);
        if (!f.fn[2]) return false;
        // any tuning field selects the kernels below, but for this kernel's own threads as the
        // team size (how the autotuner names this launch) and fp64_path = 1 (the FMA pipe)
        if (tune && ((tune->team_size > 0 && (tune->team_size != f.threads || tune->fp64_path > 0)) ||
                     tune->ctas_per_sm > 0 || tune->entries_per_team > 0 || tune->prefetch > 0 || tune->fp64_path > 1))
            return false;
        // 1 % slower: 202.9 / 204.6 us at 60000 entries, 270 / 274 at 8192
        if (!(tune && tune->team_size > 0) && ((a.n == 5 && a.d == 3 && a.nb > 15000) || (a.n == 9 && a.d == 3 && a.nb > 2000)))
            return false;
        // entries per CTA: one element per thread while one wave of CTAs holds the batch, else
        // two, else four; equally many CTAs on every SM
        long long cap = 1;
        const void *fn = nullptr;
        for (int r = 0; r < 3; ++r) {
            fn = f.fn[r];
            if (!fn) continue;
            cap = ((long long)f.threads << r) / a.N;
            const size_t smem_r = (size_t)cap * f.entry_bytes;
            if (smem_r > (size_t)di.max_smem_optin || !ensure_smem_attr(fn, smem_r)) return false;
            if (a.nb <= (long long)di.sms * occupancy(fn, f.threads, smem_r) * cap) break;
        }
        const long long k = (a.nb + di.sms * cap - 1) / (di.sms * cap);
        const long long E = (a.nb + di.sms * k - 1) / (di.sms * k);
        const size_t smem = (size_t)E * f.entry_bytes;
        const long long grid = (a.nb + E - 1) / E;
        if (grid > INT_MAX || smem > (size_t)di.max_smem_optin || !ensure_smem_attr(fn, smem)) return false;
        long long threads = (E * a.N + 31) / 32 * 32;
        if (threads > f.threads) threads = f.threads;
        a.teams_per_cta = (int)E;
        a.team_size = (int)threads;
        a.entries_per_team = 1;
        pl.fn = fn;
        pl.smem_path = true;
        pl.grid = dim3((unsigned)grid);
        pl.block = dim3((unsigned)threads);
        pl.smem = smem;
        return true;
    }
}

// Checks arguments and fills a plan.  Returns cudaSuccess, cudaErrorInvalidValue,
// or cudaErrorNotSupported (vector too long for any path without a workspace).
template <typename T, typename TO>
int plan_forward(FwdPlan<T, TO> &pl, int d, int n, const T *const *mats, int stride, const T *const *in,
                 TO *const *out, T *const *ws, long long nb, const kronmult_tuning *tune)
{
    if (d < 0 || n < 0 || nb < 0) return cudaErrorInvalidValue;
    if (stride < (n > 0 ? n : 1)) return cudaErrorInvalidValue;
    const long long Nl = pow_ll(n, d);
    if (Nl > (long long)INT_MAX) return cudaErrorInvalidValue;
    pl.args = FwdArgs<T, TO>{};
    pl.fn = nullptr;
    pl.fn2 = nullptr;
    pl.columns = false;
    kronmult_tuning cached{};
    if (!tune) {
        const int code = sizeof(T) == 8 ? KRONMULT_DTYPE_F64
                                        : (sizeof(TO) == 8 ? KRONMULT_DTYPE_F32_F64OUT : KRONMULT_DTYPE_F32);
        if (tuning_cache_lookup(d, n, code, cached)) tune = &cached;
    }
    if (nb == 0 || n == 0) return cudaSuccess;  // nothing to add
    if (!in || !out || (d > 0 && !mats)) return cudaErrorInvalidValue;

    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return cudaErrorInvalidDevice;
    const DeviceInfo &di = device_info(dev);
    const int N = (int)Nl;

    FwdArgs<T, TO> &a = pl.args;
    a.mats = mats;
    a.in = in;
    a.out = out;
    a.ws = ws;
    a.nb = nb;
    a.d = d;
    a.n = n;
    a.stride = stride;
    a.N = N;

    // ---- FP64 on the tensor path (n = 7, 8, 16 unless tuned otherwise)
    if (plan_dmma<T, TO>(pl, di, tune)) return cudaSuccess;

    // ---- FP32, n and d known at compile time: register blocks
    if (plan_block<T, TO>(pl, di, tune)) return cudaSuccess;

    // ---- FP64, short vectors
    if (plan_f64<T, TO>(pl, di, tune)) return cudaSuccess;

    // ---- register in-place shared-memory path: 2 <= n <= 8, d >= 1
    if (n >= 2 && n <= 8 && d >= 1) {
        const int F = N / n;
        const int qcap = (n <= 4) ? 8 : 4;
        int ts = 8;
        if (tune && tune->team_size > 0) {
            // a forced team size grows until every thread holds at most qcap fibres
            ts = tune->team_size;
            while (ts < 512 && (F + ts - 1) / ts > qcap) ts *= 2;
        } else {
            ts = fibre_team<T>(n, F);
        }
        // One entry per team (fwd_single_kernel) unless runs are requested: measured
        // fastest for FP64, where the FP64 pipe is the bound and more resident CTAs
        // hide the staging; FP32 sums runs of 8 entries by default.
        bool single = tune && tune->entries_per_team > 0 ? tune->entries_per_team == 1 : sizeof(T) == 8;
        const int ts_runs = ts;
        if (single && ts > 256) {
            ts = 256;  // the single-entry kernel runs teams of at most 256 threads
            if ((F + ts - 1) / ts > qcap) {
                single = false;
                ts = ts_runs;
            }
        }
        const int q = (F + ts - 1) / ts;
        int qmax = 1;
        while (qmax < q) qmax *= 2;
        const bool ts_ok = (ts == 8 || ts == 16 || ts == 32 || ts == 64 || ts == 128 || ts == 256 || ts == 512);
        if (single && ts_ok && qmax <= qcap) {
            const int vpad = round_up(N, 16 / (int)sizeof(T));
            const int fpad = round_up(d * n * n, 16 / (int)sizeof(T));
            const int team_elems = vpad + fpad;
            int teams = 256 / ts;
            auto fn = fwd_single_lookup<T, TO>(n, qmax);
            // Whole fibres per thread leave (ts*q - F) of ts*q lanes idle, and the FP64 pipe
            // is charged per warp instruction whatever the number of active lanes.  FP64
            // maps output elements to threads instead (fwd_single_elem_kernel) when that
            // uses the lanes clearly better: teams are the smallest power of two that gives
            // every thread at most 4 elements (2-4 elements per thread measured 5-25 %
            // faster than 6-16 on d = 3..6, n = 3..7: shorter chains per mode), and the
            // element mapping is taken when its lane use beats the fibre mapping's by more
            // than 5 points.  Measured on 128 MB batches: d = 3, n = 6 -22 %; d = 3, n = 5
            // -24 %; d = 2, n = 4 -27 %; d = 3, n = 3 / 7 and d = 5, n = 3 -14..-17 %
            // (for odd n the baseline was an element kernel taking n at run time); where
            // the lane use is equal (d = 2, n = 6..8; d = 4, n = 4..6) the fibre kernels were
            // as fast or up to 16 % faster.
            const double fibre_util = lane_use(F, ts);
            const int fmap = fp64_mapping(tune);
            if (sizeof(T) == 8 && fmap != 3 && (fmap == 4 || !(tune && tune->team_size > 0))) {
                int tse = 8;
                if (fmap == 4 && tune->team_size > 0) {
                    tse = tune->team_size;
                    while (tse < 256 && (N + tse - 1) / tse > 8) tse *= 2;
                } else {
                    while (tse < 256 && (N + tse - 1) / tse > 4) tse *= 2;
                }
                const int per = (N + tse - 1) / tse;
                const double util_e = lane_use(N, tse);
                // at most 8 elements per thread: no spills
                if (tse <= 256 && per <= 8 && (fmap == 4 || util_e > fibre_util + kElemMargin)) {
                    int emax = 1;
                    while (emax < per) emax *= 2;
                    auto fe = fwd_single_elem_lookup<T, TO>(n, emax);
                    if (fe) {
                        fn = fe;
                        ts = tse;
                        teams = 256 / ts;
                    }
                }
            }
            size_t smem = (size_t)teams * team_elems * sizeof(T);
            if (fn && smem <= (size_t)di.max_smem_optin && ensure_smem_attr((const void *)fn, smem)) {
                long long grid = (nb + teams - 1) / teams;
                // FP64 batches of one wave or less: fewer teams per CTA so that every SM holds
                // the same number of CTAs (256 CTAs on 152 SMs would give some SMs twice the
                // entries of others: d = 3, n = 4, 8192 entries)
                if (sizeof(T) == 8 && !(tune && tune->ctas_per_sm > 0) && grid > di.sms) {
                    const int occ = occupancy((const void *)fn, teams * ts, smem);
                    if (grid <= (long long)occ * di.sms) {
                        const long long k = (grid + di.sms - 1) / di.sms;  // CTAs per SM
                        const long long t2 = (nb + k * di.sms - 1) / (k * di.sms);
                        if (t2 >= 1 && t2 < teams) {
                            teams = (int)t2;
                            smem = (size_t)teams * team_elems * sizeof(T);
                            grid = (nb + teams - 1) / teams;
                        }
                    }
                }
                if (grid <= INT_MAX) {
                    a.team_size = ts;
                    a.teams_per_cta = teams;
                    a.entries_per_team = 1;
                    a.team_elems = team_elems;
                    a.vec_pad = vpad;
                    a.fac_pad = fpad;
                    a.prefetch = 0;
                    pl.fn = (const void *)fn;
                    pl.smem_path = true;
                    pl.grid = dim3((unsigned)grid);
                    pl.block = dim3((unsigned)(teams * ts));
                    pl.smem = smem;
                    return cudaSuccess;
                }
            }
        }
        // FP32, n = 4, d = 6: three modes per shared-memory pass, a lane pair per 64-value
        // tri-fibre (fwd_tri4_kernel), one team of 128 threads per CTA, a grid of about
        // 6 entries per CTA (36864 entries: 0.207 ms; 8: 0.209 ms; one wave of CTAs with
        // equal shares of all entries: 3-6 % slower), the entries spread evenly
        if constexpr (sizeof(T) == 4) {
            const bool want_tri4 = !single && n == 4 && d == 6 && !(tune && tune->prefetch == 1) &&
                                   !(tune && tune->team_size > 0);
            if (want_tri4) {
                auto fn = fwd_pair_lookup<TO>(4, 3);
                // two staging slots and the middle buffer: 55.5 KB, 4 CTAs per SM
                const size_t smem = (size_t)(3 * kTri4Elems + 2 * kTri4Fac) * sizeof(T);
                if (fn && smem <= (size_t)di.max_smem_optin && ensure_smem_attr((const void *)fn, smem)) {
                    int per_sm = (tune && tune->ctas_per_sm > 0) ? tune->ctas_per_sm
                                                                 : occupancy((const void *)fn, 128, smem);
                    if (per_sm < 1) per_sm = 1;
                    long long ept = (tune && tune->entries_per_team > 0) ? tune->entries_per_team : 6;
                    if (ept * di.sms * per_sm > nb * 2) ept = (nb + (long long)di.sms * per_sm - 1) / ((long long)di.sms * per_sm);
                    if (ept < 1) ept = 1;
                    const long long grid = (nb + ept - 1) / ept;
                    if (grid <= INT_MAX) {
                        a.team_size = 128;
                        a.teams_per_cta = 1;
                        a.entries_per_team = (int)((nb + grid - 1) / grid);  // the largest share
                        a.team_elems = 3 * kTri4Elems + 2 * kTri4Fac;
                        a.vec_pad = kTri4Elems;  // padded layouts (t4_in, t4_phys)
                        a.fac_pad = kTri4Fac;    // factors duplicated
                        a.prefetch = 1;
                        pl.fn = (const void *)fn;
                        pl.smem_path = true;
                        pl.grid = dim3((unsigned)grid);
                        pl.block = dim3(128);
                        pl.smem = smem;
                        return cudaSuccess;
                    }
                }
            }
        }
        // FP32, n = 8, d = 3 or 4: two modes per shared-memory pass, a lane pair per
        // 64-value bi-fibre (fwd_pair8_kernel), CTAs of 128 threads
        if constexpr (sizeof(T) == 4) {
            const bool want_pair8 = !single && n == 8 && (d == 3 || d == 4) && !(tune && tune->prefetch == 1) &&
                                    !(tune && tune->team_size > 0);
            if (want_pair8) {
                const int tsp = N / 32;  // two lanes per bi-fibre: 128 (d = 4) or 16 (d = 3)
                auto fn = fwd_pair_lookup<TO>(8, 1);
                const int vpad = p8_elems(N);  // padded layout (p8_phys)
                const int fpad = round_up(d * 64, 4);
                const int team_elems = 2 * (vpad + fpad);
                const int teams = 128 / tsp;
                const size_t smem = (size_t)teams * team_elems * sizeof(T);
                if (fn && smem <= (size_t)di.max_smem_optin && ensure_smem_attr((const void *)fn, smem)) {
                    int per_sm = (tune && tune->ctas_per_sm > 0) ? tune->ctas_per_sm
                                                                 : occupancy((const void *)fn, 128, smem);
                    if (per_sm < 1) per_sm = 1;
                    const long long total_teams = (long long)di.sms * per_sm * teams;
                    long long ept = (tune && tune->entries_per_team > 0) ? tune->entries_per_team : 8;
                    if (ept * total_teams > nb * 2) ept = (nb + total_teams - 1) / total_teams;
                    if (ept < 1) ept = 1;
                    const long long grid = (nb + ept * teams - 1) / (ept * teams);
                    if (grid <= INT_MAX && ept <= INT_MAX) {
                        a.team_size = tsp;
                        a.teams_per_cta = teams;
                        a.entries_per_team = (int)ept;
                        a.team_elems = team_elems;
                        a.vec_pad = vpad;
                        a.fac_pad = fpad;
                        a.prefetch = 1;
                        pl.fn = (const void *)fn;
                        pl.smem_path = true;
                        pl.grid = dim3((unsigned)grid);
                        pl.block = dim3(128);
                        pl.smem = smem;
                        return cudaSuccess;
                    }
                }
            }
        }
        // FP32, n = 2 and 4, d >= 2: two modes per shared-memory pass (fwd_pair_kernel)
        if constexpr (sizeof(T) == 4) {
            const bool want_pair = !single && (n == 2 || n == 4) && d >= 2 && !(tune && tune->prefetch == 1) &&
                                   !(tune && tune->team_size > 0);
            if (want_pair) {
                const int F2 = N / (n * n);
                int tsp = 8;
                while (tsp < 256 && tsp < F2) tsp *= 2;  // one bi-fibre per thread up to 256 threads
                const int qp = (F2 + tsp - 1) / tsp;
                auto fn = qp <= 2 ? fwd_pair_lookup<TO>(n, qp <= 1 ? 1 : 2) : nullptr;
                const int vpad = round_up(N, 4);
                const int fpad = round_up(d * n * n, 4);
                const int team_elems = 2 * (vpad + fpad);
                const int teams = 256 / tsp;
                const size_t smem = (size_t)teams * team_elems * sizeof(T);
                if (fn && smem <= (size_t)di.max_smem_optin && ensure_smem_attr((const void *)fn, smem)) {
                    int per_sm = (tune && tune->ctas_per_sm > 0) ? tune->ctas_per_sm
                                                                 : occupancy((const void *)fn, teams * tsp, smem);
                    if (per_sm < 1) per_sm = 1;
                    const long long total_teams = (long long)di.sms * per_sm * teams;
                    long long ept = (tune && tune->entries_per_team > 0) ? tune->entries_per_team : 8;
                    if (ept * total_teams > nb * 2) ept = (nb + total_teams - 1) / total_teams;
                    if (ept < 1) ept = 1;
                    const long long grid = (nb + ept * teams - 1) / (ept * teams);
                    if (grid <= INT_MAX && ept <= INT_MAX) {
                        a.team_size = tsp;
                        a.teams_per_cta = teams;
                        a.entries_per_team = (int)ept;
                        a.team_elems = team_elems;
                        a.vec_pad = vpad;
                        a.fac_pad = fpad;
                        a.prefetch = 1;
                        pl.fn = (const void *)fn;
                        pl.smem_path = true;
                        pl.grid = dim3((unsigned)grid);
                        pl.block = dim3((unsigned)(teams * tsp));
                        pl.smem = smem;
                        return cudaSuccess;
                    }
                }
            }
        }
        if (ts_ok && qmax <= qcap && plan_runs<T, TO>(pl, di, tune, ts, qmax)) return cudaSuccess;
    }

    // ---- large vectors: two passes through the workspace (input left intact)
    if (plan_split<T, TO>(pl, di)) {
        plan_columns<T, TO>(pl, di);  // where it can; pl stays as it is otherwise
        return cudaSuccess;
    }

    // ---- larger still: every mode through input/workspace in global memory, FP64
    // on the tensor path where it is wanted
    if constexpr (sizeof(T) == 8 && sizeof(TO) == 8) {
        if (d >= 1 && ws && dmma_wanted(n, tune)) {
            const size_t smem_s = ((size_t)round_up(n * n, 2) + 2 * (size_t)round_up(N, 2)) * sizeof(T);
            auto fn = fwd_dmma_global_lookup(n);
            if (fn && smem_s > (size_t)di.max_smem_optin) {
                const long long grid = nb < INT_MAX ? nb : INT_MAX;  // one CTA per entry
                pl.fn = (const void *)fn;
                pl.smem_path = true;
                pl.grid = dim3((unsigned)grid);
                pl.block = dim3(512);
                pl.smem = 0;
                return cudaSuccess;
            }
        }
    }
    if (n >= 2 && n <= 8 && d >= 1 && ws) {
        const size_t smem_s = ((size_t)round_up(n * n, 2) + 2 * (size_t)round_up(N, 2)) * sizeof(T);
        if (smem_s > (size_t)di.max_smem_optin) {
            auto fn = fwd_global_lookup<T, TO>(n);
            if (fn) {
                const long long grid = nb < INT_MAX ? nb : INT_MAX;  // one CTA per entry
                pl.fn = (const void *)fn;
                pl.smem_path = true;  // same launch signature as the shared-memory kernels
                pl.grid = dim3((unsigned)grid);
                pl.block = dim3(512);
                pl.smem = 0;
                return cudaSuccess;
            }
        }
    }

    // ---- generic path
    const void *fn = fwd_generic_ptr<T, TO>();
    const size_t smem_s = ((size_t)round_up(n * n, 2) + 2 * (size_t)round_up(N, 2)) * sizeof(T);
    if (smem_s <= (size_t)di.max_smem_optin && ensure_smem_attr(fn, smem_s)) {
        pl.use_smem = 1;
        pl.smem = smem_s;
    } else {
        if (!ws) return cudaErrorNotSupported;
        pl.use_smem = 0;
        pl.smem = (size_t)round_up(n * n, 2) * sizeof(T);
        if (!ensure_smem_attr(fn, pl.smem)) return cudaErrorInvalidValue;
    }
    const int block = 256;
    int per_sm = occupancy(fn, block, pl.smem);
    if (per_sm < 1) per_sm = 1;
    long long grid = (long long)di.sms * per_sm * 4;
    if (grid > nb) grid = nb;
    pl.fn = fn;
    pl.smem_path = false;
    pl.grid = dim3((unsigned)grid);
    pl.block = dim3(block);
    return cudaSuccess;
}

// The two passes of plan_columns.  (Waves of entries whose workspace stays in L2 are slower:
// n = 8, d = 6, 3905 entries 3340 us with 96 MB at a time, 3571 us with 64 MB, 2770 us at
// once; every launch ends with a partly empty GPU.)
template <typename TO> int launch_columns(const FwdPlan<float, TO> &pl, cudaStream_t st)
{
    const FwdArgs<float, TO> &a = pl.args;
    FwdArgs<float, float> u{};
    u.mats = a.mats;
    u.in = a.in;
    u.ws = a.ws;
    u.d = a.d;
    u.n = a.n;
    u.stride = a.stride;
    u.N = a.N;
    u.split_R = a.split_R;
    u.team_size = a.team_size;
    u.prefetch = 1;
    u.chunk_len = 1;
    u.nb = u.chunks = a.nb * a.split_R;
    u.entries_per_team = (int)(u.chunks / ((long long)pl.grid.x * a.teams_per_cta));
    reinterpret_cast<void (*)(const FwdArgs<float, float>)>(const_cast<void *>(pl.fn))<<<pl.grid, pl.block, pl.smem, st>>>(u);
    reinterpret_cast<void (*)(const FwdArgs<float, TO>)>(const_cast<void *>(pl.fn2))<<<pl.grid2, pl.block2, pl.smem2, st>>>(a);
    return (int)cudaGetLastError();
}

template <typename T, typename TO> int launch_plan(const FwdPlan<T, TO> &pl, cudaStream_t st)
{
    if (!pl.fn) return cudaSuccess;
    if constexpr (sizeof(T) == 4) {
        if (pl.columns) return launch_columns<TO>(pl, st);
    }
    if (pl.smem_path) {
        auto fn = reinterpret_cast<void (*)(const FwdArgs<T, TO>)>(const_cast<void *>(pl.fn));
        fn<<<pl.grid, pl.block, pl.smem, st>>>(pl.args);
        if (pl.fn2) {
            auto fn2 = reinterpret_cast<void (*)(const FwdArgs<T, TO>)>(const_cast<void *>(pl.fn2));
            fn2<<<pl.grid2, pl.block2, pl.smem2, st>>>(pl.args);
        }
    } else {
        auto fn = reinterpret_cast<void (*)(const FwdArgs<T, TO>, int)>(const_cast<void *>(pl.fn));
        fn<<<pl.grid, pl.block, pl.smem, st>>>(pl.args, pl.use_smem);
    }
    return (int)cudaGetLastError();
}

}  // namespace kgb
