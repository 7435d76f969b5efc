// The contact search shared by the FP64 and FP32 contact kernels: each
// particle's 27 cells scanned with an FP32 test that never misses a contact,
// the partners that pass collected per particle in search order, and the
// exact contact law then run on them one per lane.
//
// What it is for: a thread per particle that evaluates the law where it finds
// a contact runs the law for a lane or two at a time (a packed bed has four
// contacts among some 65 candidates), and GB300 issues an FP64 instruction of
// a warp in about 16 cycles whatever its lanes do.  Collected first, a warp's
// contacts fill its lanes.  The order of every particle's sums stays the
// reference's search order.
#pragma once

#include "xd_internal.cuh"

namespace xd {

constexpr unsigned kFullWarp = 0xffffffffu;

// An FP64 value rounded towards zero to FP32 in integer instructions (the
// conversion instruction runs on the FP64 pipe): relative error below 2^-23;
// below the FP32 range it becomes 0 or a wrong value below 2^-126, beyond it
// (or not finite) infinity.
__device__ __forceinline__ float f32_of(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int t = (int)(hi & 0x7fffffffu) - 0x38000000;   // exponent from bias 1023 to bias 127
    unsigned b = __funnelshift_l(lo, (unsigned)t, 3);
    if (t < 0) b = 0u;
    if (t >= 0x0ff00000) b = 0x7f800000u;
    return __uint_as_float(b | (hi & 0x80000000u));
}

// grid_pos (the reference's floor((x - wo) / cs) in FP64) from an FP32
// estimate: where the estimate is farther from a cell face than its error
// bound it has the same integer part, and elsewhere (about one coordinate in
// 4,000 on a 128-cell axis, or a value that is not finite) the FP64 division
// decides.  Bound: x is cut by 2^-23 of itself, wo rounded by 2^-24, and the
// difference, the product and the reciprocal round by 2^-24 each.  (Without an
// estimate, inv_csf 0, both sides of the first comparison are zero: divided.)
__device__ __forceinline__ int cell_of(const Params& P, double x, int a)
{
    const float xf = f32_of(x), q = (xf - P.wof[a]) * P.inv_csf, f = floorf(q);
    const float e = (fabsf(xf) + fabsf(P.wof[a])) * P.inv_csf * 5e-7f;
    if (q - f > e && f + 1.0f - q > e && fabsf(q) < 1e6f) return (int)f;
    return (int)floor((x - P.wo[a]) / P.cs);
}
__device__ __forceinline__ int3 grid_pos_fast(const Params& P, double x, double y, double z)
{
    return make_int3(cell_of(P, x, 0), cell_of(P, y, 1), cell_of(P, z, 2));
}

// The buffer of a block of NW warps, NP = 32 / LP particles a warp: the runs of sorted slots
// that their cells cover, the partners found (k-th of a warp's particle o at
// [k * NP + o] of the warp's kEach), where each comes in the pooled order and
// that order, and NR values of result per lane.
template <int LP, int NW, typename Real, int NR>
struct ScanBuf {
    static constexpr unsigned kWarps = NW, kParticles = 32 / LP, kSlots = LP == 1 ? 16 : 24;
    static constexpr unsigned kEach = kSlots * kParticles, kLanes = 32 * kWarps;
    uint2 run[kWarps][27][kParticles];
    Real res[NR][kLanes];
    unsigned cand[kWarps * kEach];
    unsigned short slot[kWarps * kEach];
    unsigned short pos[kWarps * kEach];
    unsigned total[kWarps];
};

// The cells of lane group o's particle (cell gp, when valid) into run[][o]:
// the sorted slots of its 27 cells in search order (x fastest), empty cells
// left out and cells whose slots follow on from the one before joined to it.
// hash(x, y, z): a cell's number.  Returns the number of runs.
template <int LP, typename Buf, typename Hash>
__device__ __forceinline__ unsigned stage_runs(Buf& B, bool valid, int3 gp, const unsigned* __restrict__ cstart,
                                               const unsigned* __restrict__ cend, Hash hash)
{
    const unsigned lane = threadIdx.x & 31u, o = lane / LP, sub = lane % LP;
    auto& run = B.run[threadIdx.x / 32u];
    constexpr int kEach = (27 + LP - 1) / LP;
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        const int c = q * LP + (int)sub;
        if (valid && c < 27) {
            const unsigned h = hash(gp.x + c % 3 - 1, gp.y + (c / 3) % 3 - 1, gp.z + c / 9 - 1);
            const unsigned st = __ldg(cstart + h);
            run[c][o] = make_uint2(st, st == 0xffffffffu ? st : __ldg(cend + h));
        }
    }
    __syncwarp();
    unsigned n = 0;
    if (valid && sub == 0) {
        uint2 cur = make_uint2(0u, 0u);
        for (int c = 0; c < 27; ++c) {
            const uint2 b = run[c][o];
            if (b.x >= b.y) continue;
            if (b.x == cur.y && cur.x != cur.y) {
                cur.y = b.y;
            } else {
                if (cur.x != cur.y) run[n++][o] = cur;
                cur = b;
            }
        }
        if (cur.x != cur.y) run[n++][o] = cur;
    }
    n = __shfl_sync(kFullWarp, n, (int)(o * LP));
    __syncwarp();
    return n;
}

// The block's contacts (every thread of it calls).  near(k, o): whether entry
// k of the sorted list may touch particle o of the warp (never false for one
// that does).  eval(o, k, l): the law of that pair, o counted through the
// block's warps, its result into B.res[][l]; returns a code, 0 for no contact.
// add(code, l): the result in B.res[][l] to the sums of the calling lane's
// particle; lane o of a warp adds its particle o's, in search order.
//
// Each round collects partners until a particle's slots could overflow, then
// takes a warp's level by level (every particle's first, then every
// particle's second, ...), 32 a warp at a time: a group of 32 then holds one
// or two of most particles and the adding runs on most lanes.  The groups run
// on across the block's warps: the FP64 pipe takes as long for a group of
// three contacts as for one of 32, and a warp's own last group was half empty
// (pairs, us a call, a warp's own groups and a block's: 8,000 spheres 50 and
// 40.5, 120,989 343 and 327, FP32 100,003 80 and 70; on a mesh's wide cells,
// which the search bounds, 17,159 212 and 215).
template <int LP, typename Buf, typename Near, typename Eval, typename Add>
__device__ __forceinline__ void scan_contacts(Buf& B, unsigned nruns, const unsigned* __restrict__ sorted, Near near,
                                              Eval eval, Add add)
{
    constexpr unsigned P = 32 / LP, U = LP == 1 ? 4u : (LP == 4 ? 2u : 1u), S = Buf::kSlots, E = Buf::kEach;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x / 32u, o = lane / LP, sub = lane % LP;
    const unsigned group = LP == 32 ? kFullWarp : ((1u << LP) - 1u) << (o * LP);
    unsigned* const cand = B.cand + warp * E;
    unsigned short* const pos = B.pos + warp * E;
    const auto& run = B.run[warp];
    unsigned r = 0, j = 0, e = 0;
    bool more = nruns != 0u;
    if (more) {
        const uint2 b = run[0][o];
        j = b.x;
        e = b.y;
    }
    while (true) {
        unsigned cnt = 0;
        while (true) {
            const bool act = more && cnt + LP * U <= S;
            if (!__any_sync(kFullWarp, act)) break;
            unsigned k[U];
            bool in[U];
#pragma unroll
            for (unsigned u = 0; u < U; ++u) {
                const unsigned jj = j + u * LP + sub;
                in[u] = act && jj < e;
                k[u] = in[u] ? __ldg(sorted + jj) : 0u;
            }
#pragma unroll
            for (unsigned u = 0; u < U; ++u) in[u] = in[u] && near(k[u], o);
#pragma unroll
            for (unsigned u = 0; u < U; ++u) {
                if (LP == 1) {
                    if (in[u]) cand[cnt++ * P + o] = k[u];
                } else {
                    const unsigned b = __ballot_sync(kFullWarp, in[u]) & group;
                    if (in[u]) cand[(cnt + __popc(b & ((1u << lane) - 1u))) * P + o] = k[u];
                    cnt += __popc(b);
                }
            }
            if (act) {
                j += LP * U;
                if (j >= e) {
                    more = ++r < nruns;
                    if (more) {
                        const uint2 b = run[r][o];
                        j = b.x;
                        e = b.y;
                    }
                }
            }
        }
        // lane o < P owns particle o
        const unsigned mine = LP == 1 ? cnt : __shfl_sync(kFullWarp, cnt, (int)((lane * LP) & 31u));
        const unsigned own = lane < P ? mine : 0u;
        const unsigned levels = __reduce_max_sync(kFullWarp, own), found = __reduce_add_sync(kFullWarp, own);
        if (lane == 0) B.total[warp] = found;
        __syncthreads();
        unsigned at = 0, total = 0;
#pragma unroll
        for (unsigned w = 0; w < Buf::kWarps; ++w) {
            const unsigned t = B.total[w];
            at += w < warp ? t : 0u;
            total += t;
        }
        for (unsigned l = 0; l < levels; ++l) {
            const unsigned b = __ballot_sync(kFullWarp, own > l);
            if (own > l) {
                const unsigned p = at + __popc(b & ((1u << lane) - 1u));
                B.slot[p] = (unsigned short)(warp * E + l * P + lane);
                pos[l * P + lane] = (unsigned short)p;
            }
            at += __popc(b);
        }
        __syncthreads();
        unsigned done = 0;
        for (unsigned base = 0; base < total; base += Buf::kLanes) {
            if (base + threadIdx.x < total) {
                const unsigned s = B.slot[base + threadIdx.x];
                B.cand[s] = eval(s / E * P + s % P, B.cand[s], threadIdx.x);
            }
            __syncthreads();
            for (; done < own; ++done) {
                const unsigned p = pos[done * P + lane];
                if (p >= base + Buf::kLanes) break;
                const unsigned code = cand[done * P + lane];
                if (code) add(code, p - base);
            }
            if (base + Buf::kLanes < total) __syncthreads();
        }
        if (!__syncthreads_or(more)) return;
    }
}

// Lanes per particle of a scan over np particles.  A warp of 32 particles
// fills its lanes best (131 contacts of a bed in five groups); with few
// particles the chip is not full and more lanes shorten the chain of loads
// and contacts that one warp goes through.  FP64 pairs, us with 1 / 4 / 8
// lanes: a bed of 2,000 spheres 70 / 37 / 25, 8,000 78 / 46 / 42, 17,000
// 99 / 73 / 85, 40,000 144 / 139 / 163, 60,000 184 / 210 / 226, 120,989
// 339 / 400 / 426; on a mesh's wide cells 17,159 583 / 220 / 254 and 60,000
// 2,032 / 1,860 / 2,301.
//
// Warps whose contacts a block pools: for the FP64 law 2, 4 or 8 by lanes per
// particle, about 32 to 64 particles a block, but with fewer than 152 blocks of
// 8 warps half as many (2,000 spheres: 8 warps 31 us, 4 25, 2 27; 8,000, before
// every SM got as many blocks: 46, 48 and 54).  The FP32 law gains from full
// groups only where there are many: 2 warps (8,000 spheres: 8 warps 20.8 us, 2
// 18.8), and 1 lane a particle from 28,000 on (30,000: 36.6 us, with 4 lanes
// 37.3; 100,003: 72 and 94).
//
// f(lanes, warps), each as a type's value, for np particles.
template <int V>
struct IntC {
    static constexpr int value = V;
};
template <bool FP64 = true, typename F>
inline void scan_shape(unsigned np, F f)
{
    if (np >= (FP64 ? 48000u : 28000u)) f(IntC<1>(), IntC<2>());
    else if (np >= 10000u) f(IntC<4>(), IntC<FP64 ? 4 : 2>());
    else if (FP64 && np >= 152u * 32u) f(IntC<8>(), IntC<8>());
    else f(IntC<8>(), IntC<FP64 ? 4 : 2>());
}

// Blocks for it, and how many particles each takes at a time: at most one wave
// (16 warps an SM), whose blocks then take several groups of particles and
// form the contact property's constants once.  Pools of 8 warps come one or
// two to an SM, and the SMs with one wait for those with two: every SM gets as
// many blocks there, with fewer particles in each (8,000 spheres 40.5 -> 37.5
// us).  With 4 lanes that gains a bed of 17,000 spheres 2 us of 73 and costs
// a hopper, whose search leaves lanes idle then, 3 of 220.
constexpr unsigned kSms = 152u, kScanWarps = kSms * 8u * 2u;
struct ScanGrid {
    unsigned blocks, each;
};
inline ScanGrid scan_grid(unsigned np, unsigned lp, unsigned nw)
{
    const unsigned full = 32u / lp * nw, blocks = div_up(np, full), most = kScanWarps / nw;
    if (blocks > most) return { most, full };
    if (nw < 8u) return { blocks, full };
    const unsigned each = div_up(np, div_up(blocks, kSms) * kSms);
    return { div_up(np, each), each };
}

}  // namespace xd
