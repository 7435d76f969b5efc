// Stable LSD radix sort of 32-bit (key, value) pairs on sm_103a.
//
// Replaces thrust::sort_by_key in cu_reorderDataAndFindCellStart
// (source/mphysics_cuda_def.cu:92-94).  The cell grid's keys only span
// ceil(log2(ncell)) bits (21 for the reference's 128^3 grid), and the sort is
// bound by its launches and by latency, so it takes as few passes as it can:
// digits of up to 11 bits, two passes for 21 bits.  Each pass is three
// launches with no inter-block waiting:
//   1. k_tile_hist   per-tile digit counts, [tile][digit];
//   2. k_tile_scan   each digit's exclusive prefix over the tiles, and its total;
//   3. k_scatter     the totals' prefix, stable in-tile ranking by ballots,
//                    and the scatter.
// A tile's keys are visited in index order, warp by warp, so equal digits
// keep their input order and the sort is stable.  Up to 8,192 pairs are
// ranked by comparing all of them in one launch (k_rank).
//
// 21-bit keys, us a sort in a graph (five launches in each of three 8-bit
// passes before): 8,000 pairs 13.5 (33), 100,000 19.5 (35), 1,000,000 46 (63).
#include <cuda_runtime.h>

#include "xd_internal.cuh"

namespace xd {
namespace {

constexpr unsigned kMaxBits = 11;
constexpr unsigned kMaxRadix = 1u << kMaxBits;
constexpr unsigned kRankMax = 8192;   // 8,192 pairs: 13.1 us ranked, 18.2 by digits; its cost grows with the square
static_assert(kRankMax <= 152 * 64, "a block ranks 64 keys at most");

__device__ __forceinline__ unsigned lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The valid lanes of the warp whose digit is this lane's, by a ballot per bit
// (1,000,000 keys: 46 us a sort, 49 with __match_any_sync).
__device__ __forceinline__ unsigned same_digit(unsigned d, bool valid)
{
    unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (unsigned b = 0; b < kMaxBits; ++b) {
        const bool one = (d >> b) & 1u;
        const unsigned v = __ballot_sync(0xffffffffu, one);
        peers &= one ? v : ~v;
    }
    return peers;
}

// A tile is R keys for each thread of W warps.
template <int W, int R>
__global__ void __launch_bounds__(W * 32) k_tile_hist(const unsigned* __restrict__ keys, unsigned n, unsigned shift,
                                                        unsigned bits, unsigned* __restrict__ hist)
{
    __shared__ unsigned cnt[kMaxRadix];
    constexpr unsigned kT = W * 32;
    const unsigned radix = 1u << bits, mask = radix - 1u;
    for (unsigned i = threadIdx.x; i < radix; i += kT) cnt[i] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kT * R;
    constexpr int kAtOnce = R < 8 ? R : 8;
    for (int r = 0; r < R; r += kAtOnce) {
        unsigned k[kAtOnce];
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            const size_t idx = base + (size_t)(r + q) * kT + threadIdx.x;
            k[q] = idx < n ? __ldg(keys + idx) : 0u;
        }
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q)
            if (base + (size_t)(r + q) * kT + threadIdx.x < n) atomicAdd(&cnt[(k[q] >> shift) & mask], 1u);
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < radix; i += kT) hist[(size_t)blockIdx.x * radix + i] = cnt[i];
}

// Each digit's counts over the tiles become their exclusive prefix, and
// total[digit] their sum.  A block takes 32 digits (x) and splits the tiles
// into 32 runs (y), so that the loads are rows of 32 digits and a digit's
// chain is a 32nd of the tiles.
__global__ void __launch_bounds__(1024) k_tile_scan(unsigned* __restrict__ hist, unsigned ntiles, unsigned radix,
                                                    unsigned* __restrict__ total)
{
    __shared__ unsigned sums[32][33];
    const unsigned x = threadIdx.x & 31u, y = threadIdx.x >> 5;
    const unsigned d = blockIdx.x * 32u + x;
    const unsigned run = (ntiles + 31u) / 32u, t0 = y * run, t1 = min(ntiles, t0 + run);
    unsigned s = 0;
    if (d < radix)
#pragma unroll 4
        for (unsigned t = t0; t < t1; ++t) s += hist[(size_t)t * radix + d];
    sums[x][y] = s;
    __syncthreads();
    // warp y scans digit y's 32 run sums
    const unsigned v = sums[y][x];
    unsigned inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (x >= (unsigned)o) inc += u;
    }
    sums[y][x] = inc - v;
    if (x == 31u && blockIdx.x * 32u + y < radix) total[blockIdx.x * 32u + y] = inc;
    __syncthreads();
    if (d >= radix) return;
    unsigned off = sums[x][y];
#pragma unroll 4
    for (unsigned t = t0; t < t1; ++t) {
        const unsigned c = hist[(size_t)t * radix + d];
        hist[(size_t)t * radix + d] = off;
        off += c;
    }
}

// Dynamic shared memory: the warps' digit counts (16 bits: a tile holds at
// most 8,192 keys), then the digits' first slots.
constexpr unsigned scatter_smem(unsigned warps, unsigned radix) { return warps * radix * 2u + radix * 4u; }

template <int W, int R>
__global__ void __launch_bounds__(W * 32) k_scatter(const unsigned* __restrict__ kin, const unsigned* __restrict__ vin,
                                                      unsigned* __restrict__ kout, unsigned* __restrict__ vout,
                                                      unsigned n, unsigned shift, unsigned bits,
                                                      const unsigned* __restrict__ offsets,
                                                      const unsigned* __restrict__ total)
{
    extern __shared__ __align__(16) unsigned char sort_smem[];
    __shared__ unsigned warp_sum[W];
    constexpr unsigned kT = W * 32;
    const unsigned radix = 1u << bits, mask = radix - 1u;
    unsigned short* const wcnt = reinterpret_cast<unsigned short*>(sort_smem);   // [W][radix]
    unsigned* const gbase = reinterpret_cast<unsigned*>(sort_smem + W * radix * 2u);
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (unsigned i = threadIdx.x; i < W * radix / 2u; i += kT) reinterpret_cast<unsigned*>(wcnt)[i] = 0;
    // the digits' first slots: the totals' exclusive prefix, a run of digits per thread
    const unsigned per = (radix + kT - 1u) / kT, d0 = threadIdx.x * per;
    unsigned s = 0;
    for (unsigned q = 0; q < per; ++q) s += d0 + q < radix ? __ldg(total + d0 + q) : 0u;
    unsigned inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (unsigned)o) inc += u;
    }
    if (lane == 31u) warp_sum[warp] = inc;
    __syncthreads();
    unsigned off = inc - s;
    for (unsigned w = 0; w < warp; ++w) off += warp_sum[w];
    for (unsigned q = 0; q < per && d0 + q < radix; ++q) {
        gbase[d0 + q] = off + __ldg(offsets + (size_t)blockIdx.x * radix + d0 + q);
        off += __ldg(total + d0 + q);
    }
    __syncthreads();

    const size_t wbase = ((size_t)blockIdx.x * W + warp) * (R * 32);
    const unsigned ltmask = lanemask_lt();
    unsigned short* const mine = wcnt + warp * radix;
    unsigned short rank[R];
    constexpr int kAtOnce = R < 8 ? R : 8;
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += kAtOnce) {
        unsigned key[kAtOnce];
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            const size_t idx = wbase + (size_t)(r0 + q) * 32 + lane;
            key[q] = idx < n ? __ldg(kin + idx) : 0u;
        }
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            const bool valid = wbase + (size_t)(r0 + q) * 32 + lane < n;
            const unsigned d = valid ? ((key[q] >> shift) & mask) : 0xffffffffu;
            const unsigned peers = same_digit(d, valid);
            unsigned before = 0;
            if (valid) before = mine[d];
            rank[r0 + q] = (unsigned short)(before + __popc(peers & ltmask));
            __syncwarp();
            if (valid && (__ffs(peers) - 1) == (int)lane) mine[d] = (unsigned short)(before + __popc(peers));
            __syncwarp();
        }
    }
    __syncthreads();
    for (unsigned d = threadIdx.x; d < radix; d += kT) {
        unsigned run = 0;
#pragma unroll 8
        for (unsigned w = 0; w < W; ++w) {
            const unsigned c = wcnt[w * radix + d];
            wcnt[w * radix + d] = (unsigned short)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += kAtOnce) {
        unsigned key[kAtOnce], val[kAtOnce];
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            const size_t idx = wbase + (size_t)(r0 + q) * 32 + lane;
            key[q] = idx < n ? __ldg(kin + idx) : 0u;
            val[q] = idx < n ? __ldg(vin + idx) : 0u;
        }
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            if (wbase + (size_t)(r0 + q) * 32 + lane >= n) continue;
            const unsigned d = (key[q] >> shift) & mask;
            const unsigned dst = gbase[d] + mine[d] + rank[r0 + q];
            kout[dst] = key[q];
            vout[dst] = val[q];
        }
    }
}

// Up to kRankMax pairs: each key's rank is the number of keys below it, and of
// equal keys before it.  A block ranks up to 64 keys (two a lane) against all
// of them in shared memory, its 32 warps a 32nd each; the keys before the
// block's own count when <=, those after when <.  Blocks are as many as SMs.
constexpr unsigned kRankThreads = 1024, kRankWarps = kRankThreads / 32;

__global__ void __launch_bounds__(kRankThreads) k_rank(const unsigned* __restrict__ kin,
                                                       const unsigned* __restrict__ vin, unsigned* __restrict__ kout,
                                                       unsigned* __restrict__ vout, unsigned n, unsigned mask,
                                                       unsigned each)
{
    __shared__ uint4 keys4[kRankMax / 4];
    __shared__ unsigned part[kRankWarps][64];
    unsigned* const keys = reinterpret_cast<unsigned*>(keys4);
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned n4 = (n + 3u) / 4u;
#pragma unroll 8
    for (unsigned j = threadIdx.x; j < 4u * n4; j += kRankThreads)
        keys[j] = j < n ? __ldg(kin + j) & mask : 0xffffffffu;
    __syncthreads();
    const unsigned b0 = blockIdx.x * each, b1 = min(n, b0 + each);
    const unsigned i0 = b0 + lane, i1 = i0 + 32u;
    const unsigned k0 = keys[min(i0, n - 1u)], k1 = keys[min(i1, n - 1u)];
    // groups of four keys: before the block's own, around them, after
    const unsigned per = (n4 + kRankWarps - 1u) / kRankWarps, g0 = warp * per, g1 = min(n4, g0 + per);
    const unsigned own0 = b0 / 4u, own1 = min(n4, (b1 + 3u) / 4u);
    unsigned c0 = 0, c1 = 0;
#pragma unroll 4
    for (unsigned g = g0; g < min(g1, own0); ++g) {
        const uint4 v = keys4[g];
        c0 += (v.x <= k0) + (v.y <= k0) + (v.z <= k0) + (v.w <= k0);
        c1 += (v.x <= k1) + (v.y <= k1) + (v.z <= k1) + (v.w <= k1);
    }
    for (unsigned j = 4u * max(g0, own0); j < 4u * min(g1, own1); ++j) {
        const unsigned v = keys[j];
        c0 += v < k0 || (v == k0 && j < i0);
        c1 += v < k1 || (v == k1 && j < i1);
    }
#pragma unroll 4
    for (unsigned g = max(g0, own1); g < g1; ++g) {
        const uint4 v = keys4[g];   // the last group's filling is the largest key: never below one
        c0 += (v.x < k0) + (v.y < k0) + (v.z < k0) + (v.w < k0);
        c1 += (v.x < k1) + (v.y < k1) + (v.z < k1) + (v.w < k1);
    }
    part[warp][lane] = c0;
    part[warp][lane + 32u] = c1;
    __syncthreads();
    const unsigned i = b0 + threadIdx.x;
    if (threadIdx.x < each && i < b1) {
        unsigned rank = 0;
#pragma unroll 8
        for (unsigned w = 0; w < kRankWarps; ++w) rank += part[w][threadIdx.x];
        kout[rank] = __ldg(kin + i);
        vout[rank] = __ldg(vin + i);
    }
}

// Every part is at least as large as for any smaller n, and so is the whole:
// a sort of fewer keys fits the scratch of a sort of more.
struct SortLayout {
    size_t keys_alt, vals_alt, hist, total, bytes;
};

SortLayout layout(unsigned n)
{
    SortLayout L;
    const size_t ntiles = n ? sort_tiles_within(n) : 1u;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    L.keys_alt = 0;
    L.vals_alt = L.keys_alt + al(sizeof(unsigned) * (size_t)n);
    L.hist = L.vals_alt + al(sizeof(unsigned) * (size_t)n);
    L.total = L.hist + al(sizeof(unsigned) * kMaxRadix * ntiles);
    L.bytes = L.total + al(sizeof(unsigned) * kMaxRadix);
    return L;
}

}  // namespace

size_t radix_sort_scratch_bytes(unsigned n) { return layout(n).bytes; }

unsigned radix_sort_launches(unsigned n, unsigned key_bits)
{
    if (n <= 1 || key_bits == 0) return 0;
    return n <= kRankMax ? 1u : 3u * div_up(key_bits < 32u ? key_bits : 32u, kMaxBits);
}

// Sorts (keys, vals) by the low key_bits bits.  The result is left either in
// the input arrays or in the scratch's alternate buffers; *out_keys/*out_vals
// point at it.
int radix_sort_pairs(unsigned* keys, unsigned* vals, unsigned n, unsigned key_bits, void* scratch,
                     cudaStream_t s, unsigned** out_keys, unsigned** out_vals)
{
    *out_keys = keys;
    *out_vals = vals;
    if (n <= 1 || key_bits == 0) return XD_OK;
    if (key_bits > 32) key_bits = 32;
    const SortLayout L = layout(n);
    char* base = static_cast<char*>(scratch);
    unsigned* kalt = reinterpret_cast<unsigned*>(base + L.keys_alt);
    unsigned* valt = reinterpret_cast<unsigned*>(base + L.vals_alt);
    if (n <= kRankMax) {
        const unsigned each = div_up(n, 152);   // at most 54 keys a block
        k_rank<<<div_up(n, each), kRankThreads, 0, s>>>(keys, vals, kalt, valt, n,
                                                        key_bits == 32 ? 0xffffffffu : (1u << key_bits) - 1u, each);
        *out_keys = kalt;
        *out_vals = valt;
        return launch_status("radix_sort_pairs");
    }
    unsigned* hist = reinterpret_cast<unsigned*>(base + L.hist);
    unsigned* total = reinterpret_cast<unsigned*>(base + L.total);
    const unsigned passes = div_up(key_bits, kMaxBits), most = div_up(key_bits, passes);
    const unsigned tile = sort_tile(n), ntiles = div_up(n, tile);
    unsigned *ks = keys, *vs = vals, *kd = kalt, *vd = valt;
    for (unsigned p = 0; p < passes; ++p) {
        const unsigned shift = p * most, bits = key_bits - shift < most ? key_bits - shift : most;
        const unsigned radix = 1u << bits;
#define XD_SORT_PASS(W, R)                                                                                        \
    do {                                                                                                          \
        const unsigned smem = scatter_smem(W, radix);                                                             \
        if (smem > 48u * 1024u) {                                                                                 \
            const int st = cuda_status(cudaFuncSetAttribute(k_scatter<W, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                            (int)smem), "radix_sort_pairs");                      \
            if (st != XD_OK) return st;                                                                           \
        }                                                                                                         \
        k_tile_hist<W, R><<<ntiles, W * 32, 0, s>>>(ks, n, shift, bits, hist);                                    \
        k_tile_scan<<<div_up(radix, 32), 1024, 0, s>>>(hist, ntiles, radix, total);                               \
        k_scatter<W, R><<<ntiles, W * 32, smem, s>>>(ks, vs, kd, vd, n, shift, bits, hist, total);                \
    } while (0)
        if (tile == 1024u) XD_SORT_PASS(8, 4);
        else if (tile == 2048u) XD_SORT_PASS(8, 8);
        else if (tile == 4096u) XD_SORT_PASS(16, 8);
        else XD_SORT_PASS(32, 8);
#undef XD_SORT_PASS
        unsigned* t;
        t = ks; ks = kd; kd = t;
        t = vs; vs = vd; vd = t;
    }
    *out_keys = ks;
    *out_vals = vs;
    return launch_status("radix_sort_pairs");
}

}  // namespace xd
