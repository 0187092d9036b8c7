// galn_device.cuh -- device side of the `bwa aln` search for sm_100a.
//
// Two occurrence layouts, both one 32-byte sector (one DRAM sector) per block; the kernels take the stride
// as a template parameter and an index holds both.
//   occ64: blocks of 64 symbols of the $-free BWT: four uint32 counts of each base before the block,
//          relative to the block's 2^32-symbol superblock, then the 64 symbols as two 64-bit bit planes
//          (bit j of p0 = low bit of symbol j, of p1 = high bit).
//   occ80: blocks of 80 symbols: three uint32 counts (A, C, G) before the block relative to its superblock
//          of 2^25 blocks, a word holding bits 64-79 of both planes (p0 in the low half, p1 in the high),
//          then bits 0-63 of p0 and p1. The count of T is the position's rank minus the other three.
//          20% smaller (80 MB for a 100 Mbp genome, inside the device's persisting-L2 limit), and a pair
//          (k-1, l) falls in one block more often.
// One LF step for one position is one 32-byte fetch; the reference's layout (src/bwtsearch.h:22-34, 128
// symbols in 64 bytes) needs two sectors. The superblock counts are kernel parameters. Counts and intervals
// are the same integers as bwt_occ / bwt_2occ / bwt_occ4 / bwt_2occ4 (src/bwtsearch.h:46-108,
// src/bwtgap_hd.h:135-192).
#pragma once

#include <stdint.h>

namespace galn {

constexpr int kMaxSuper = 16;          // superblocks: 2^36 symbols for occ64, 2^29 x 80 for occ80
constexpr int kMaxSuper32 = 2;         // texts below 2^32: one occ64 superblock, two occ80 ones
constexpr int kOcc64 = 64, kOcc80 = 80;   // the layouts' strides
constexpr int kOcc80SuperShift = 25;   // occ80 blocks per superblock: 2^25
constexpr int kModeGape = 0x01, kModeLoggap = 0x04, kModeNonstop = 0x10;
constexpr int kStM = 0, kStI = 1, kStD = 2;
constexpr int kErrStack = -1, kErrAln = -2, kErrScore = -3;
constexpr uint64_t kTraceInit = 1469598103934665603ULL;
constexpr uint64_t kTracePrime = 1099511628211ULL;

// The index as kernels see it. P is the type of BWT positions and counts: uint32_t for texts shorter than
// kNarrowText (nearly all: up to about 2.1 Gbp of reference), uint64_t otherwise. The search's step is integer
// work on interval ends with a chain of dependent instructions behind each fetch; 64-bit positions make most of them
// two or three. With 32-bit positions (and width_word, galn_search.cuh) the first tier of 2 M aDNA reads on 100 Mbp
// went from 78.6 to 72.3 ms, a warp-tier pop from 383 to 341 cycles there, from 471 to 394 on a 310 Mbp repeat-rich
// genome, and from 290 to 241 on the high-divergence reads.
template <class P>
struct IndexViewT {
    static constexpr int kSuper = sizeof(P) == 8 ? kMaxSuper : kMaxSuper32;
    const uint4 *blk;                   // 2 x uint4 per block
    P primary, seq_len;
    P C[4];                             // L2[0..3]
    P sb[kSuper][4];                    // Occ before each superblock
};
using IndexView = IndexViewT<uint64_t>;

// per-batch options as the search uses them (the batch's local gap_opt_t, src/aln_host.c:23-38)
struct BatchOpt {
    int s_mm, s_gapo, s_gape, mode;
    int indel_end_skip, max_del_occ, max_entries;
    int max_diff, max_gapo, max_gape, max_seed_diff, seed_len, max_top2;
    int n_stacks;
    int wide;                           // 1: counts or lengths too large for the 16-byte entry
    int pad_;
};

template <class P>
__device__ __forceinline__ P sel4(int c, P a0, P a1, P a2, P a3)
{
    const P lo = (c & 1) ? a1 : a0, hi = (c & 1) ? a3 : a2;
    return (c & 2) ? hi : lo;
}

// bits 0 .. n-1 set, n clamped to [0, 32]
__device__ __forceinline__ uint32_t low_mask(int n)
{
    uint32_t m;
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(m) : "r"(n > 0 ? n : 0));
    return m;
}

// One position's block and what of it to count: the block's two halves, the symbols counted (0 for the position
// before row 0) and its block number.
struct OccBlk {
    uint4 c, x;
    int nb;
};

// Loads the block of position p ($-skipped below; ~0 = -1, which counts nothing: block 0's counts are zero).
template <int S, class P>
__device__ __forceinline__ P occ_load(const IndexViewT<P> &ix, P p, P &rank, uint32_t &sup, OccBlk &o)
{
    const bool none = p == (P)~(P)0;
    const P q = none ? 0 : p - (P)(p >= ix.primary);
    P b;
    if (S == kOcc64) { b = q >> 6; o.nb = none ? 0 : (int)(q & 63) + 1; }
    else { b = q / 80; o.nb = none ? 0 : (int)(q - 80 * b) + 1; }
    rank = none ? 0 : q + 1;
    sup = S == kOcc64 ? (uint32_t)((uint64_t)q >> 32) : (uint32_t)(b >> kOcc80SuperShift);
    const uint4 *a = ix.blk + ((size_t)b << 1);
    o.c = __ldg(a);
    o.x = __ldg(a + 1);
    return none ? (P)~(P)0 : b;
}

// Occ of the four bases from a loaded block: the counts before it plus those of its first nb symbols. With the
// planes masked once, the counts of C, G and T come from three population counts per word and A's from the
// rest.
template <int S, class P>
__device__ __forceinline__ void occ_counts(const IndexViewT<P> &ix, const OccBlk &o, P rank, uint32_t sup, P r[4])
{
    const uint32_t m0 = low_mask(o.nb), m1 = low_mask(o.nb - 32);
    const uint32_t a0 = o.x.x & m0, a1 = o.x.y & m1, b0 = o.x.z & m0, b1 = o.x.w & m1;
    int t = __popc(a0 & b0) + __popc(a1 & b1), c = __popc(a0) + __popc(a1), g = __popc(b0) + __popc(b1);
    if (S == kOcc80) {
        const uint32_t m2 = low_mask(o.nb - 64);
        const uint32_t h0 = o.c.w & m2 & 0xffffu, h1 = (o.c.w >> 16) & m2;
        t += __popc(h0 & h1); c += __popc(h0); g += __popc(h1);
    }
    const int a = o.nb - c - g + t;
    r[0] = (P)o.c.x + (P)a;
    r[1] = (P)o.c.y + (P)(c - t);
    r[2] = (P)o.c.z + (P)(g - t);
    if (S == kOcc64) {
        r[3] = (P)o.c.w + (P)t;
        if (sizeof(P) == 8) {   // 32-bit texts lie in superblock 0, whose counts are zero
#pragma unroll
            for (int q = 0; q < 4; ++q) r[q] += ix.sb[sup][q];
        }
    } else {
#pragma unroll
        for (int q = 0; q < 3; ++q) r[q] += ix.sb[sup][q];
        r[3] = rank - r[0] - r[1] - r[2];
    }
}

// Occ(c, k1) and Occ(c, l) for all four bases (positions in [-1, seq_len]; Occ(., -1) = 0), without a branch
// around the loads: both blocks are read (the same address twice when k1 and l share a block, which the L1
// merges), so threads of a warp that differ in that respect still wait for one round trip together.
// `fetches` counts the distinct 32-byte blocks (the roofline's unit of algorithmic traffic): one when both
// positions fall in one block.
template <int S, class P>
__device__ __forceinline__ void occ4_pair_u(const IndexViewT<P> &ix, P k1, P l, P ok[4], P ol[4], uint32_t &fetches)
{
    OccBlk ko, lo;
    P kr, lr;
    uint32_t ks, ls;
    const P kb = occ_load<S, P>(ix, k1, kr, ks, ko), lb = occ_load<S, P>(ix, l, lr, ls, lo);
    fetches += kb == lb && ko.nb && lo.nb ? 1u : (uint32_t)(ko.nb > 0) + (uint32_t)(lo.nb > 0);
    occ_counts<S, P>(ix, ko, kr, ks, ok);
    occ_counts<S, P>(ix, lo, lr, ls, ol);
}

// Occ of base c alone from a loaded block.
template <int S, class P>
__device__ __forceinline__ P occ_one(const IndexViewT<P> &ix, const OccBlk &o, P rank, uint32_t sup, int c)
{
    const uint32_t f0 = c & 1 ? 0u : ~0u, f1 = c & 2 ? 0u : ~0u;
    int n = __popc((o.x.x ^ f0) & (o.x.z ^ f1) & low_mask(o.nb)) + __popc((o.x.y ^ f0) & (o.x.w ^ f1) & low_mask(o.nb - 32));
    if (S == kOcc64) {
        P r = (P)sel4(c, o.c.x, o.c.y, o.c.z, o.c.w) + (P)n;
        if (sizeof(P) == 8) r += ix.sb[sup][c];
        return r;
    }
    n += __popc((o.c.w ^ f0) & ((o.c.w >> 16) ^ f1) & low_mask(o.nb - 64) & 0xffffu);
    const P a = (P)o.c.x + ix.sb[sup][0], b = (P)o.c.y + ix.sb[sup][1], g = (P)o.c.z + ix.sb[sup][2];
    return sel4(c, a, b, g, (P)(rank - (P)o.nb - a - b - g)) + (P)n;
}

__device__ __forceinline__ uint64_t trace_mix(uint64_t h, uint64_t v) { return (h ^ v) * kTracePrime; }

}  // namespace galn
