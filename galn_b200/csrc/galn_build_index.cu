// galn_build_index.cu -- `galn index` on the GPU: the .bwt and .sa files of bwa index 0.7.19 for the text
// T = F . revcomp(F) of a forward sequence F (codes 0..3).
//
// The reference builds them in src/index/gpu_index.cu:1-20 (BWT of T$ by libcubwt or its rank-based sorter,
// then pack + interleaved Occ on the GPU, SA samples by LF walks and list ranking). This builder:
//   1. sorts the suffixes by prefix doubling, refining only the groups still unsorted (Larsson-Sadakane):
//      the first round sorts 16-symbol prefixes as 32-bit keys (32 symbols as 64-bit keys in short texts), the
//      suffixes that end inside their prefix set apart by the order of the items (pd_key0); round r sorts the
//      unsorted suffixes i by (rank of i, rank of i + h), h = 16 * 2^(r-1) (or 32), where a rank is the
//      suffix-array index of the first suffix of its group. Every sort is a stable LSD radix sort written here:
//      8-bit digits, per-tile histogram, scan, and a scatter that ranks each tile's items in shared memory so
//      each digit's run leaves the tile as one contiguous write. Round 0's sorted positions are the suffix array;
//      later rounds put their items back at their slots. The first round is bound by its passes: with 32-bit keys
//      it makes 4 of 20 bytes an item (key and value in and out, keys once more for the histogram) where 21-symbol
//      63-bit keys made 8 of 32;
//   2. takes the BWT from the suffix array and the packed text (50 MB for 100 Mbp, so its gathers hit L2), packs it
//      2 bits a symbol with the Occ counts every 128 symbols (the .bwt layout of bwt_bwtupdate_core,
//      src/index/idxcommon.c:72-112);
//   3. gathers every 32nd suffix-array row (the .sa layout, src/index/idxcommon.c:137-153).
// Positions are 32-bit: texts up to 2^32 - 64 symbols (references up to about 2.1 Gbp), about 41 bytes of device
// memory per symbol in one block (the 64-bit path where that cannot be had). Everything but the file writes runs on the
// device.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "galn_internal.h"

namespace galn {
namespace ixb {

constexpr int kRThreads = 512, kRItems = 8, kRTile = kRThreads * kRItems, kRWarps = kRThreads / 32;
constexpr int kScanThreads = 256;
constexpr int kPrefix = 21;            // symbols in a first-round key of the 64-bit path
// and of the 32-bit one: 32 symbols (64-bit keys, 8 passes) for texts below kLongKeys, whose rounds cost launches and
// waits and not bytes and whose repeats are then mostly told apart at once; 16 (32-bit keys, 4 passes) above
constexpr int kPrefixLong = 32, kPrefixShort = 16;
constexpr uint64_t kLongKeys = 1ull << 24;
constexpr int kMaxRounds = 40;         // h = 16 * 2^39 exceeds any 32-bit text, 21 * 2^39 any 64-bit one

struct U4 {
    uint64_t c[4];
};
__host__ __device__ inline U4 operator+(const U4 &a, const U4 &b)
{
    return U4{{a.c[0] + b.c[0], a.c[1] + b.c[1], a.c[2] + b.c[2], a.c[3] + b.c[3]}};
}

// items a scan thread holds: 8 of 4- or 8-byte types, 2 of the 32-byte per-block counts
template <class T>
constexpr int scan_items() { return sizeof(T) > 8 ? 2 : 8; }
template <class T>
constexpr int scan_tile_n() { return kScanThreads * scan_items<T>(); }

template <class T>
struct OpSum {
    __device__ static T id() { return T{}; }
    __device__ static T op(const T &a, const T &b) { return a + b; }
};
template <class T>
struct OpMax {
    __device__ static T id() { return T(0); }
    __device__ static T op(const T &a, const T &b) { return a > b ? a : b; }
};

// ---- scans (reduce, scan of the tile sums, scan of each tile with its carry-in) ----

template <class T, class Op>
__global__ void __launch_bounds__(kScanThreads) scan_reduce(const T *__restrict__ x, uint64_t n, T *__restrict__ part)
{
    constexpr int kItems = scan_items<T>(), kTile = scan_tile_n<T>();
    __shared__ T s[kScanThreads];
    const int t = threadIdx.x;
    const uint64_t base = (uint64_t)blockIdx.x * kTile;
    T acc = Op::id();
    for (int j = 0; j < kItems; ++j) {
        const uint64_t i = base + (uint64_t)j * kScanThreads + t;
        if (i < n) acc = Op::op(acc, x[i]);
    }
    s[t] = acc;
    __syncthreads();
    for (int w = kScanThreads / 2; w > 0; w >>= 1) {
        if (t < w) s[t] = Op::op(s[t], s[t + w]);
        __syncthreads();
    }
    if (t == 0) part[blockIdx.x] = s[0];
}

// In place: inclusive (INCL) or exclusive scan of one tile, offset by carry[tile] when carry is given.
template <class T, class Op, bool INCL>
__global__ void __launch_bounds__(kScanThreads) scan_tile(T *__restrict__ x, uint64_t n, const T *__restrict__ carry)
{
    constexpr int kItems = scan_items<T>(), kTile = scan_tile_n<T>();
    __shared__ T s[kTile];
    __shared__ T tsum[kScanThreads];
    const int t = threadIdx.x;
    const uint64_t base = (uint64_t)blockIdx.x * kTile;
    for (int j = 0; j < kItems; ++j) {
        const uint64_t i = base + (uint64_t)j * kScanThreads + t;
        s[j * kScanThreads + t] = i < n ? x[i] : Op::id();
    }
    __syncthreads();
    T v[kItems];
    T acc = Op::id();
    for (int j = 0; j < kItems; ++j) {
        v[j] = s[t * kItems + j];
        acc = Op::op(acc, v[j]);
    }
    tsum[t] = acc;
    __syncthreads();
    for (int off = 1; off < kScanThreads; off <<= 1) {   // inclusive scan of the thread sums
        const T o = t >= off ? tsum[t - off] : Op::id();
        __syncthreads();
        if (t >= off) tsum[t] = Op::op(o, tsum[t]);
        __syncthreads();
    }
    T run = t ? tsum[t - 1] : Op::id();
    if (carry) run = Op::op(carry[blockIdx.x], run);
    for (int j = 0; j < kItems; ++j) {
        const T in = v[j];
        if (INCL) run = Op::op(run, in);
        s[t * kItems + j] = run;
        if (!INCL) run = Op::op(run, in);
    }
    __syncthreads();
    for (int j = 0; j < kItems; ++j) {
        const uint64_t i = base + (uint64_t)j * kScanThreads + t;
        if (i < n) x[i] = s[j * kScanThreads + t];
    }
}

// Device scratch for the scans' per-tile sums, taken as a stack.
struct Scratch {
    unsigned char *p = nullptr;
    size_t cap = 0, top = 0;
};

template <class T, class Op, bool INCL>
int scan(T *x, uint64_t n, Scratch &scr, cudaStream_t st)
{
    if (n == 0) return 0;
    const uint64_t tiles = (n + scan_tile_n<T>() - 1) / scan_tile_n<T>();
    if (tiles == 1) {
        scan_tile<T, Op, INCL><<<1, kScanThreads, 0, st>>>(x, n, nullptr);
        return cudaGetLastError() == cudaSuccess ? 0 : GALN_ECUDA;
    }
    const size_t bytes = (tiles * sizeof(T) + 255) & ~(size_t)255;
    if (scr.top + bytes > scr.cap) return GALN_ENOMEM;
    T *part = reinterpret_cast<T *>(scr.p + scr.top);
    scr.top += bytes;
    scan_reduce<T, Op><<<(unsigned)tiles, kScanThreads, 0, st>>>(x, n, part);
    int rc = scan<T, Op, false>(part, tiles, scr, st);
    if (!rc) scan_tile<T, Op, INCL><<<(unsigned)tiles, kScanThreads, 0, st>>>(x, n, part);
    scr.top -= bytes;
    if (rc) return rc;
    return cudaGetLastError() == cudaSuccess ? 0 : GALN_ECUDA;
}

// ---- stable LSD radix sort of (K key, V value) pairs, K and V = uint32 or uint64 ----

// counts[d * tiles + tile] = items of digit d in the tile
template <class K>
__global__ void __launch_bounds__(kRThreads) radix_hist(const K *__restrict__ keys, uint64_t n, int shift,
                                                         uint32_t *__restrict__ counts, uint32_t tiles)
{
    __shared__ uint32_t h[256];
    const int t = threadIdx.x, lane = t & 31;
    if (t < 256) h[t] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kRTile;
    uint32_t dg[kRItems];
#pragma unroll
    for (int j = 0; j < kRItems; ++j) {   // all loads first
        const uint64_t i = base + (uint64_t)j * kRThreads + t;
        dg[j] = i < n ? (uint32_t)(keys[i] >> shift) & 255u : 256u;
    }
#pragma unroll
    for (int j = 0; j < kRItems; ++j) {
        const uint32_t d = dg[j];
        if (__all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {   // one digit in the whole warp
            if (lane == 0 && d < 256u) atomicAdd(&h[d], 32u);
            continue;
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        if (d < 256u && lane == __ffs(peers) - 1) atomicAdd(&h[d], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (t < 256) counts[(uint64_t)t * tiles + blockIdx.x] = h[t];
}

template <class K, class V>
struct ScatterSmem {
    uint32_t wcnt[kRWarps][256];       // per warp: items of each digit, then their offset among the tile's
    uint32_t tstart[256];              // start of each digit in the tile's sorted order
    uint32_t gofs[256];                // the tile's first output index for each digit
    uint32_t wsum[8];
    K k[kRTile];
    V v[kRTile];
};

// Items of a tile in input order: warp w holds [w * 32 * kRItems, (w + 1) * 32 * kRItems), its step j the
// 32 items from j * 32 on, one per lane. A lane's rank among the warp's items of its digit comes from
// __match_any_sync; warps are ordered by a per-digit prefix over warps; the tile's items are placed in
// digit order in shared memory and leave it in runs.
template <class K, class V>
__global__ void __launch_bounds__(kRThreads) radix_scatter(const K *__restrict__ kin,
                                                            const V *__restrict__ vin,
                                                            K *__restrict__ kout, V *__restrict__ vout,
                                                            uint64_t n, int shift, const uint32_t *__restrict__ offsets,
                                                            uint32_t tiles)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ScatterSmem<K, V> &S = *reinterpret_cast<ScatterSmem<K, V> *>(smem_raw);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * kRTile;
    const uint64_t wbase = base + (uint64_t)w * (32 * kRItems);
    const uint32_t lt_mask = (1u << lane) - 1u;
    K key[kRItems];
    V val[kRItems];
    uint32_t rk[kRItems];
#pragma unroll
    for (int j = 0; j < kRItems; ++j) {   // all loads in flight while the counters are cleared
        const uint64_t i = wbase + (uint64_t)j * 32 + lane;
        const bool ok = i < n;
        key[j] = ok ? kin[i] : 0;
        val[j] = ok ? vin[i] : 0;
    }
    for (int i = t; i < kRWarps * 256; i += kRThreads) (&S.wcnt[0][0])[i] = 0;
    if (t < 256) S.gofs[t] = offsets[(uint64_t)t * tiles + blockIdx.x];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kRItems; ++j) {
        const bool ok = wbase + (uint64_t)j * 32 + lane < n;
        const uint32_t d = ok ? (uint32_t)(key[j] >> shift) & 255u : 256u;
        const bool uni = __all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0));
        const uint32_t peers = uni ? 0xffffffffu : __match_any_sync(0xffffffffu, d);
        const uint32_t c = ok ? S.wcnt[w][d] : 0u;
        rk[j] = c + (uint32_t)__popc(peers & lt_mask);
        __syncwarp();
        if (ok && (peers & lt_mask) == 0) S.wcnt[w][d] = c + (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    uint32_t tot = 0;
    if (t < 256) {
        for (int ww = 0; ww < kRWarps; ++ww) {
            const uint32_t c = S.wcnt[ww][t];
            S.wcnt[ww][t] = tot;
            tot += c;
        }
    }
    // exclusive scan of the 256 digit totals (threads 0..255 = warps 0..7)
    uint32_t inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (t < 256 && lane == 31) S.wsum[w] = inc;
    __syncthreads();
    if (t < 256) {
        uint32_t before = 0;
        for (int ww = 0; ww < w; ++ww) before += S.wsum[ww];
        S.tstart[t] = before + inc - tot;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kRItems; ++j) {
        const uint64_t i = wbase + (uint64_t)j * 32 + lane;
        if (i < n) {
            const uint32_t d = (uint32_t)(key[j] >> shift) & 255u;
            const uint32_t p = S.tstart[d] + S.wcnt[w][d] + rk[j];
            S.k[p] = key[j];
            S.v[p] = val[j];
        }
    }
    __syncthreads();
    const uint32_t tile_n = (uint32_t)min((uint64_t)kRTile, n - base);
    for (uint32_t i = t; i < tile_n; i += kRThreads) {
        const K kk = S.k[i];
        const uint32_t d = (uint32_t)(kk >> shift) & 255u;
        const uint64_t dst = (uint64_t)S.gofs[d] + (i - S.tstart[d]);
        kout[dst] = kk;
        vout[dst] = S.v[i];
    }
}

template <class V, class K = uint64_t>
struct Sorter {
    K *k[2] = {nullptr, nullptr};
    V *v[2] = {nullptr, nullptr};
    uint32_t *counts = nullptr;
    Scratch *scr = nullptr;
    int passes = 0;
    uint64_t scatter_items = 0;
    std::vector<cudaEvent_t> ev;       // start/stop pairs around each scatter launch
};

// Sorts the n pairs in (k[cur], v[cur]) on key bits [0, bits); returns the buffer that holds them sorted.
template <class V, class K>
int radix_sort(Sorter<V, K> &s, int cur, uint64_t n, int bits, cudaStream_t st, int &out)
{
    out = cur;
    if (n <= 1) return 0;
    const uint32_t tiles = (uint32_t)((n + kRTile - 1) / kRTile);
    for (int shift = 0; shift < bits; shift += 8) {
        radix_hist<K><<<tiles, kRThreads, 0, st>>>(s.k[cur], n, shift, s.counts, tiles);
        int rc = scan<uint32_t, OpSum<uint32_t>, false>(s.counts, (uint64_t)tiles * 256, *s.scr, st);
        if (rc) return rc;
        cudaEvent_t a, b;
        if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) return GALN_ECUDA;
        s.ev.push_back(a);
        s.ev.push_back(b);
        cudaEventRecord(a, st);
        radix_scatter<K, V><<<tiles, kRThreads, sizeof(ScatterSmem<K, V>), st>>>(s.k[cur], s.v[cur], s.k[cur ^ 1],
                                                                                 s.v[cur ^ 1], n, shift, s.counts, tiles);
        cudaEventRecord(b, st);
        if (cudaGetLastError() != cudaSuccess) return GALN_ECUDA;
        cur ^= 1;
        ++s.passes;
        s.scatter_items += n;
    }
    out = cur;
    return 0;
}

// ---- prefix doubling ----

// The text T = F . revcomp(F) two bits a symbol, sixteen symbols a word, the first in the top bits; zero past the end.
// *bad is set when a code of F is above 3.
__global__ void pack_text(const uint8_t *__restrict__ F, uint64_t l_pac, uint64_t n_words, uint32_t *__restrict__ W,
                          uint32_t *__restrict__ bad)
{
    const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= n_words) return;
    const uint64_t N = 2 * l_pac;
    uint32_t v = 0, seen = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint64_t i = 16 * w + j;
        uint32_t c = 0;
        if (i < l_pac) { c = F[i]; seen |= c; }
        else if (i < N) c = 3u - F[N - 1 - i];
        v |= (c & 3u) << (30 - 2 * j);
    }
    W[w] = v;
    if (seen > 3) *bad = 1;
}

__device__ __forceinline__ uint32_t text_symbol(const uint32_t *__restrict__ W, uint32_t p)
{
    return (__ldg(W + (p >> 4)) >> (30 - 2 * (p & 15))) & 3u;
}

// Round 0's items: SYM-symbol keys (zero past the end) and positions. The last SYM - 1 suffixes come first, the shortest
// at the head: the sort is stable, so among equal keys they stand before the others and in their order, each a group of
// its own (a suffix that ends inside its key sorts before one that goes on with symbol 0).
template <int SYM, class K>
__global__ void pd_key0(const uint32_t *__restrict__ W, uint64_t N, K *__restrict__ key, uint32_t *__restrict__ pos)
{
    static_assert(SYM == 4 * sizeof(K), "two bits a symbol");
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    const uint64_t n_short = min((uint64_t)(SYM - 1), N);
    const uint32_t p = (uint32_t)(k < n_short ? N - 1 - k : k - n_short);
    const uint32_t *w = W + (p >> 4);
    const int sh = 2 * (p & 15);
    K v = __funnelshift_l(__ldg(w + 1), __ldg(w), sh);
    if (SYM == 32) v = (K)((uint64_t)v << 32 | __funnelshift_l(__ldg(w + 2), __ldg(w + 1), sh));
    key[k] = v;
    pos[k] = p;
}

// whether sorted item k starts a group (equal keys; in round 0, SYM > 0, a suffix shorter than its key is a group of
// its own)
template <int SYM, class K>
__device__ __forceinline__ bool pd_head(const K *__restrict__ key, const uint32_t *__restrict__ P, uint64_t k, uint64_t N)
{
    if (k == 0 || key[k] != key[k - 1]) return true;
    return SYM > 0 && ((uint64_t)P[k] + SYM - 1 >= N || (uint64_t)P[k - 1] + SYM - 1 >= N);
}

// H[k] = the slot of item k if it starts a group of equal keys, else 0 (an inclusive max-scan then gives
// every item its group's first slot). Slots rise with k; round 0's slot of item k is k.
template <int SYM, class K>
__global__ void pd_heads(const K *__restrict__ key, const uint32_t *__restrict__ P, const uint32_t *__restrict__ slot,
                         uint64_t M, uint64_t N, uint32_t *__restrict__ H)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    H[k] = pd_head<SYM>(key, P, k, N) ? (SYM ? (uint32_t)k : slot[k]) : 0u;
}

// rank[position] = its group's first slot; C[k] = 1 when item k stays unsorted (its group has two or more). After
// round 0 the items are put back at their slots of the suffix array, where round 0's positions stand already.
template <int SYM, class K>
__global__ void pd_rank(const K *__restrict__ key, const uint32_t *__restrict__ P, const uint32_t *__restrict__ H,
                        const uint32_t *__restrict__ slot, uint64_t M, uint64_t N, uint32_t *__restrict__ rank,
                        uint32_t *__restrict__ C, uint32_t *__restrict__ sa)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const bool head = pd_head<SYM>(key, P, k, N);
    const bool last = k + 1 == M || pd_head<SYM>(key, P, k + 1, N);
    const uint32_t p = P[k];
    rank[p] = H[k];
    C[k] = (head && last) ? 0u : 1u;
    if (!SYM) sa[slot[k]] = p;
}

// C: inclusive count of kept items. Kept item k goes to C[k] - 1 with its position and slot.
__global__ void pd_compact(const uint32_t *__restrict__ P, const uint32_t *__restrict__ slot,
                           const uint32_t *__restrict__ C, uint64_t M, uint32_t *__restrict__ P2,
                           uint32_t *__restrict__ slot2)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const uint32_t c = C[k], prev = k ? C[k - 1] : 0u;
    if (c == prev) return;
    P2[c - 1] = P[k];
    slot2[c - 1] = slot ? slot[k] : (uint32_t)k;
}

// key of an unsorted suffix p: (rank of p, rank of p + h plus one; 0 when p + h is the end of the text)
__global__ void pd_key(const uint32_t *__restrict__ P, const uint32_t *__restrict__ rank, uint64_t M, uint64_t N,
                       uint64_t h, int lo_bits, uint64_t *__restrict__ K)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const uint64_t p = P[k], q = p + h;
    const uint64_t lo = q < N ? (uint64_t)rank[q] + 1 : 0;
    K[k] = ((uint64_t)rank[p] << lo_bits) | lo;
}

// ---- BWT, .bwt body, .sa samples ----

// One warp per block of 128 symbols of the BWT of T$ without the $ of row `primary` (row 0, the $ suffix, gives the
// text's last symbol; row r > 0 has the suffix sa[r - 1]): the block's eight words of sixteen symbols (first symbol in
// the top bits; words past the text are not written) and its counts.
__global__ void __launch_bounds__(256) bwt_blocks(const uint32_t *__restrict__ W, const uint32_t *__restrict__ sa,
                                                  uint64_t N, uint64_t primary, uint64_t nb, uint32_t *__restrict__ body,
                                                  U4 *__restrict__ cnt)
{
    const uint64_t b = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (b >= nb) return;
    const int lane = threadIdx.x & 31;
    uint32_t sym[4];
    bool ok[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {      // all gathers first
        const uint64_t s = b * 128 + 32 * j + lane, row = s < primary ? s : s + 1;
        ok[j] = s < N;
        sym[j] = ok[j] ? text_symbol(W, (uint32_t)((row == 0 ? N : (uint64_t)sa[row - 1]) - 1)) : 0u;
    }
    uint32_t c1 = 0, c2 = 0, c3 = 0, n = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t lo = __ballot_sync(0xffffffffu, sym[j] & 1u), hi = __ballot_sync(0xffffffffu, sym[j] & 2u);
        c1 += __popc(lo & ~hi); c2 += __popc(hi & ~lo); c3 += __popc(lo & hi);
        n += __popc(__ballot_sync(0xffffffffu, ok[j]));
        uint32_t word = sym[j] << (30 - 2 * (lane & 15));
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, o);
        if ((lane & 15) == 0 && ok[j]) body[b * 16 + 8 + 2 * j + (lane >> 4)] = word;
    }
    if (lane == 0) cnt[b] = U4{{n - c1 - c2 - c3, c1, c2, c3}};
}

// the four uint64 counts before each block of 128 symbols (incl = inclusive per-block counts), in its first 8 words
__global__ void bwt_counts(uint64_t nb, const U4 *__restrict__ incl, uint32_t *__restrict__ body)
{
    const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nb * 8) return;
    const uint64_t b = idx >> 3;
    const int j = (int)(idx & 7);
    const uint64_t v = b ? incl[b - 1].c[j >> 1] : 0;
    body[b * 16 + j] = (j & 1) ? (uint32_t)(v >> 32) : (uint32_t)v;
}

__global__ void bwt_block_counts(const uint8_t *__restrict__ L, uint64_t N, uint64_t nb, U4 *__restrict__ cnt)
{
    const uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const uint64_t s = b * 128, e = min(s + 128, N);
    uint64_t c0 = 0, c1 = 0, c2 = 0, c3 = 0;
    for (uint64_t i = s; i < e; ++i) {
        const uint8_t x = L[i];
        c0 += x == 0; c1 += x == 1; c2 += x == 2; c3 += x == 3;
    }
    cnt[b] = U4{{c0, c1, c2, c3}};
}

// 16 words per 128-symbol block: the four uint64 counts before it, then 8 words of 16 symbols, the first
// symbol in the top two bits. incl = inclusive per-block counts. Words past the text are not written.
__global__ void bwt_write(const uint8_t *__restrict__ L, uint64_t N, uint64_t nb, const U4 *__restrict__ incl,
                          uint32_t *__restrict__ body)
{
    const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nb * 16) return;
    const uint64_t b = idx >> 4;
    const int j = (int)(idx & 15);
    if (j < 8) {
        const uint64_t v = b ? incl[b - 1].c[j >> 1] : 0;
        body[idx] = (j & 1) ? (uint32_t)(v >> 32) : (uint32_t)v;
        return;
    }
    const uint64_t s0 = b * 128 + (uint64_t)(j - 8) * 16;
    if (s0 >= N) return;
    uint32_t word = 0;
    for (int t = 0; t < 16; ++t)
        if (s0 + t < N) word |= (uint32_t)L[s0 + t] << (30 - 2 * t);
    body[idx] = word;
}

// sa without row 0 (the $ suffix)
__global__ void sa_samples(const uint32_t *__restrict__ sa, uint64_t ns, uint64_t *__restrict__ out)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < ns) out[k] = sa[(k + 1) * 32 - 1];
}

__global__ void text_from_forward(const uint8_t *__restrict__ F, uint64_t l_pac, uint8_t *__restrict__ T)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * l_pac) return;
    T[i] = i < l_pac ? F[i] : (uint8_t)(3 - F[2 * l_pac - 1 - i]);
}

inline unsigned grid(uint64_t n, int b) { return (unsigned)((n + b - 1) / b); }
inline int bitlen(uint64_t x) { return x ? 64 - __builtin_clzll(x) : 0; }

// ---- the 64-bit path (texts of 2^32 - 64 symbols or more) ----
// Positions, ranks and slots are 64-bit. Round 0 runs bucket by bucket: suffixes are grouped by their first
// kWPre symbols (a histogram of those prefix codes, then runs of consecutive codes holding at most `chunk`
// suffixes), each bucket's suffixes are selected from the text, sorted by their 21-symbol keys and ranked;
// the unsorted ones are appended to one list U of (position, slot) in slot order. A later round walks U in
// chunks of whole groups: each item's key is (its group's number in the chunk, rank of p + h), the chunk is
// sorted, ranked and its still-unsorted items compacted back into U in place. Ranks are updated while the
// round goes on: a rank that another chunk has refined already is still consistent with the suffix order
// (its group only split into ordered parts), so sorting by it can only refine further (Larsson-Sadakane's
// argument). The BWT and the SA samples are scattered from the final ranks without a suffix array.
constexpr int kWPre = 5;                                  // symbols of a bucket prefix
constexpr uint32_t kWCodes = 1u << (3 * kWPre);           // prefix codes (3 bits a symbol)
constexpr int kWHistTile = 1 << 20;                       // text positions per histogram block
constexpr int kWSelTile = 1 << 14;                        // text positions per selection block
constexpr int kWSelThreads = 256;

__device__ __forceinline__ uint64_t key21(const uint8_t *__restrict__ T, uint64_t N, uint64_t i)
{
    uint64_t k = 0;
    for (int j = 0; j < kPrefix; ++j) {
        const uint64_t p = i + j;
        k = (k << 3) | (p < N ? (uint64_t)T[p] + 1 : 0);
    }
    return k;
}

__device__ __forceinline__ uint32_t code5(const uint8_t *__restrict__ T, uint64_t N, uint64_t i)
{
    uint32_t c = 0;
    for (int j = 0; j < kWPre; ++j) {
        const uint64_t p = i + j;
        c = (c << 3) | (p < N ? (uint32_t)T[p] + 1 : 0u);
    }
    return c;
}

// hist[c] += the text positions whose kWPre-symbol prefix code is c (a shared-memory histogram per block)
__global__ void __launch_bounds__(1024) w_hist(const uint8_t *__restrict__ T, uint64_t N,
                                               unsigned long long *__restrict__ hist)
{
    extern __shared__ uint32_t hs[];
    for (uint32_t c = threadIdx.x; c < kWCodes; c += blockDim.x) hs[c] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kWHistTile;
    const uint64_t end = min(N, base + kWHistTile);
    for (uint64_t i = base + threadIdx.x; i < end; i += blockDim.x) atomicAdd(&hs[code5(T, N, i)], 1u);
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < kWCodes; c += blockDim.x)
        if (hs[c]) atomicAdd(&hist[c], (unsigned long long)hs[c]);
}

// per selection tile: how many positions have a prefix code in [lo, hi]
__global__ void __launch_bounds__(kWSelThreads) w_sel_count(const uint8_t *__restrict__ T, uint64_t N, uint32_t lo,
                                                            uint32_t hi, uint32_t *__restrict__ tcount)
{
    __shared__ uint32_t s[kWSelThreads / 32];
    const uint64_t base = (uint64_t)blockIdx.x * kWSelTile;
    const uint64_t end = min(N, base + kWSelTile);
    uint32_t c = 0;
    for (uint64_t i = base + threadIdx.x; i < end; i += kWSelThreads) {
        const uint32_t x = code5(T, N, i);
        c += (x >= lo && x <= hi) ? 1u : 0u;
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < kWSelThreads / 32; ++w) t += s[w];
        tcount[blockIdx.x] = t;
    }
}

// writes the selected positions in text order (tile offsets from an exclusive scan of w_sel_count) with
// their 21-symbol keys
__global__ void __launch_bounds__(kWSelThreads) w_sel_write(const uint8_t *__restrict__ T, uint64_t N, uint32_t lo,
                                                            uint32_t hi, const uint32_t *__restrict__ toff,
                                                            uint64_t *__restrict__ K, uint64_t *__restrict__ P)
{
    __shared__ uint32_t s[kWSelThreads / 32];
    __shared__ uint32_t run;
    const uint64_t base = (uint64_t)blockIdx.x * kWSelTile;
    const uint64_t end = min(N, base + kWSelTile);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) run = toff[blockIdx.x];
    __syncthreads();
    for (uint64_t i0 = base; i0 < end; i0 += kWSelThreads) {
        const uint64_t i = i0 + threadIdx.x;
        const uint32_t x = i < end ? code5(T, N, i) : 0u;
        const bool sel = i < end && x >= lo && x <= hi;
        const uint32_t b = __ballot_sync(0xffffffffu, sel);
        if (lane == 0) s[w] = (uint32_t)__popc(b);
        __syncthreads();
        uint32_t before = run;
        for (int ww = 0; ww < w; ++ww) before += s[ww];
        if (sel) {
            const uint64_t o = before + (uint32_t)__popc(b & ((1u << lane) - 1u));
            K[o] = key21(T, N, i);
            P[o] = i;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (int ww = 0; ww < kWSelThreads / 32; ++ww) t += s[ww];
            run += t;
        }
        __syncthreads();
    }
}

// H[k] = slot of item k (slot0 + k, or slot[k]) if its key starts a group, else 0
__global__ void w_heads(const uint64_t *__restrict__ K, uint64_t M, uint64_t slot0, const uint64_t *__restrict__ slot,
                        uint64_t *__restrict__ H)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const bool head = k == 0 || K[k] != K[k - 1];
    H[k] = head ? (slot ? slot[k] : slot0 + k) : 0;
}

// rank[position] = its group's first slot; C[k] = 1 when item k stays unsorted
__global__ void w_rank(const uint64_t *__restrict__ K, const uint64_t *__restrict__ P, const uint64_t *__restrict__ H,
                       uint64_t M, uint64_t *__restrict__ rank, uint32_t *__restrict__ C)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const bool head = k == 0 || K[k] != K[k - 1];
    const bool last = k + 1 == M || K[k + 1] != K[k];
    rank[P[k]] = H[k];
    C[k] = (head && last) ? 0u : 1u;
}

// kept item k goes to U at out + C[k] - 1 with its position and slot (slot0 + k, or slot[k])
__global__ void w_compact(const uint64_t *__restrict__ P, const uint32_t *__restrict__ C, uint64_t M, uint64_t slot0,
                          const uint64_t *__restrict__ slot, uint64_t out, uint64_t *__restrict__ Upos,
                          uint64_t *__restrict__ Uslot)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const uint32_t c = C[k], prev = k ? C[k - 1] : 0u;
    if (c == prev) return;
    Upos[out + c - 1] = P[k];
    Uslot[out + c - 1] = slot ? slot[k] : slot0 + k;
}

// group starts of U's items [a, a + m): F[k] = 1 when item a + k starts a group (its rank differs from the
// item before it); the flags' inclusive scan numbers the groups
__global__ void w_group_flags(const uint64_t *__restrict__ Upos, uint64_t a, uint64_t m, const uint64_t *__restrict__ rank,
                              uint32_t *__restrict__ F)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    F[k] = (k == 0 || rank[Upos[a + k]] != rank[Upos[a + k - 1]]) ? 1u : 0u;
}

// the last group start in U's items (a, e], or a when there is none (one group fills the window)
__global__ void w_last_start(const uint64_t *__restrict__ Upos, uint64_t a, uint64_t e, const uint64_t *__restrict__ rank,
                             unsigned long long *__restrict__ best)
{
    const uint64_t k = a + 1 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k > e) return;
    if (rank[Upos[k]] != rank[Upos[k - 1]]) atomicMax(best, (unsigned long long)k);
}

// key of chunk item k: (its group number, rank of p + h plus one; 0 past the end), position as the value;
// the chunk's slots are copied aside (U's slot array is overwritten by the compaction)
__global__ void w_key(const uint64_t *__restrict__ Upos, const uint64_t *__restrict__ Uslot, uint64_t a, uint64_t m,
                      const uint32_t *__restrict__ G, const uint64_t *__restrict__ rank, uint64_t N, uint64_t h,
                      int lo_bits, uint64_t *__restrict__ K, uint64_t *__restrict__ P)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    const uint64_t p = Upos[a + k], q = p + h;
    const uint64_t lo = q < N ? rank[q] + 1 : 0;
    K[k] = ((uint64_t)(G[k] - 1) << lo_bits) | lo;
    P[k] = p;
}

__global__ void w_copy_u64(const uint64_t *__restrict__ src, uint64_t m, uint64_t *__restrict__ dst)
{
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) dst[k] = src[k];
}

// the BWT without the $ of row `primary` (row r's symbol is T[SA[r] - 1]; suffix i is at row rank[i] + 1,
// the $ suffix at row 0) and the SA samples of rows 32, 64, ...
__global__ void w_bwt_scatter(const uint8_t *__restrict__ T, const uint64_t *__restrict__ rank, uint64_t N,
                              uint64_t primary, uint8_t *__restrict__ L, uint64_t *__restrict__ smp)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    if (i == 0) L[0] = T[N - 1];
    const uint64_t row = rank[i] + 1;
    if (i > 0) L[row < primary ? row : row - 1] = T[i - 1];
    if ((row & 31) == 0) smp[row / 32 - 1] = i;
}

struct DevMem {
    std::vector<void *> ptrs;
    ~DevMem()
    {
        for (void *p : ptrs) cudaFree(p);
    }
    template <class T>
    T *get(size_t count)
    {
        void *p = nullptr;
        if (cudaMalloc(&p, std::max<size_t>(count * sizeof(T), 256)) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        ptrs.push_back(p);
        return static_cast<T *>(p);
    }
};

// Round 0 of the 64-bit path, then the doubling rounds over U; fills rank[0..N). Returns 0 or an error.
int wide_sort(const uint8_t *T, uint64_t N, uint64_t *rank, Sorter<uint64_t> &srt, Scratch &scr, uint64_t chunk,
              uint64_t *Upos, uint64_t *Uslot, uint64_t ucap, uint32_t *tcount, unsigned long long *hist,
              unsigned long long *best, cudaStream_t st, int &rounds, uint64_t &sorted)
{
    rounds = 0;
    sorted = 0;
    // bucket plan: runs of consecutive prefix codes holding at most `chunk` suffixes each
    if (cudaMemsetAsync(hist, 0, kWCodes * 8, st) != cudaSuccess) return GALN_ECUDA;
    w_hist<<<grid(N, kWHistTile), 1024, kWCodes * 4, st>>>(T, N, hist);
    std::vector<unsigned long long> h(kWCodes);
    if (cudaMemcpyAsync(h.data(), hist, kWCodes * 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return GALN_ECUDA;
    const uint64_t sel_tiles = (N + kWSelTile - 1) / kWSelTile;
    uint64_t u_n = 0, slot0 = 0;
    uint32_t lo = 0;
    while (lo < kWCodes) {
        uint64_t m = 0;
        uint32_t hi = lo;
        while (hi < kWCodes && (m + h[hi] <= chunk || (m == 0 && h[hi] <= chunk))) m += h[hi++];
        if (hi == lo) {
            fprintf(stderr, "[galn index] %llu suffixes share a %d-symbol prefix: more than %llu at once\n",
                    (unsigned long long)h[lo], kWPre, (unsigned long long)chunk);
            return GALN_ENOMEM;
        }
        if (m > 0) {
            w_sel_count<<<(unsigned)sel_tiles, kWSelThreads, 0, st>>>(T, N, lo, hi - 1, tcount);
            int rc = scan<uint32_t, OpSum<uint32_t>, false>(tcount, sel_tiles, scr, st);
            if (rc) return rc;
            w_sel_write<<<(unsigned)sel_tiles, kWSelThreads, 0, st>>>(T, N, lo, hi - 1, tcount, srt.k[0], srt.v[0]);
            int kb = 0;
            rc = radix_sort(srt, 0, m, 3 * kPrefix, st, kb);
            if (rc) return rc;
            sorted += m;
            uint64_t *H = srt.k[kb ^ 1];
            uint32_t *C = reinterpret_cast<uint32_t *>(srt.v[kb ^ 1]);
            w_heads<<<grid(m, 256), 256, 0, st>>>(srt.k[kb], m, slot0, nullptr, H);
            rc = scan<uint64_t, OpMax<uint64_t>, true>(H, m, scr, st);
            if (rc) return rc;
            w_rank<<<grid(m, 256), 256, 0, st>>>(srt.k[kb], srt.v[kb], H, m, rank, C);
            rc = scan<uint32_t, OpSum<uint32_t>, true>(C, m, scr, st);
            if (rc) return rc;
            uint32_t kept = 0;
            if (cudaMemcpyAsync(&kept, C + m - 1, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                return GALN_ECUDA;
            if (u_n + kept > ucap) {
                fprintf(stderr, "[galn index] %llu unsorted suffixes after the first sort: more than fit\n",
                        (unsigned long long)(u_n + kept));
                return GALN_ENOMEM;
            }
            w_compact<<<grid(m, 256), 256, 0, st>>>(srt.v[kb], C, m, slot0, nullptr, u_n, Upos, Uslot);
            u_n += kept;
            slot0 += m;
        }
        lo = hi;
    }
    if (slot0 != N) return GALN_ECUDA;
    // doubling rounds over U in chunks of whole groups
    const int lo_bits = bitlen(N);
    uint64_t h2 = kPrefix;
    while (u_n > 0) {
        if (++rounds > kMaxRounds) return GALN_EINVAL;
        uint64_t a = 0, out = 0;
        while (a < u_n) {
            uint64_t e = std::min(u_n, a + chunk);
            if (e < u_n) {   // end the chunk at the last group start inside the window
                unsigned long long b = a;
                if (cudaMemcpyAsync(best, &b, 8, cudaMemcpyHostToDevice, st) != cudaSuccess) return GALN_ECUDA;
                w_last_start<<<grid(e - a, 256), 256, 0, st>>>(Upos, a, e, rank, best);
                if (cudaMemcpyAsync(&b, best, 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                    cudaStreamSynchronize(st) != cudaSuccess)
                    return GALN_ECUDA;
                if (b == a) {
                    fprintf(stderr, "[galn index] a group of more than %llu suffixes\n", (unsigned long long)chunk);
                    return GALN_ENOMEM;
                }
                e = b;
            }
            const uint64_t m = e - a;
            uint32_t *G = reinterpret_cast<uint32_t *>(srt.k[1]);
            w_group_flags<<<grid(m, 256), 256, 0, st>>>(Upos, a, m, rank, G);
            int rc = scan<uint32_t, OpSum<uint32_t>, true>(G, m, scr, st);
            if (rc) return rc;
            uint32_t n_groups = 0;
            if (cudaMemcpyAsync(&n_groups, G + m - 1, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                return GALN_ECUDA;
            if (bitlen(n_groups) + lo_bits > 64) return GALN_EINVAL;
            w_key<<<grid(m, 256), 256, 0, st>>>(Upos, Uslot, a, m, G, rank, N, h2, lo_bits, srt.k[0], srt.v[0]);
            int kb = 0;
            rc = radix_sort(srt, 0, m, lo_bits + bitlen(n_groups - 1), st, kb);
            if (rc) return rc;
            sorted += m;
            uint64_t *H = srt.k[kb ^ 1];
            uint32_t *C = reinterpret_cast<uint32_t *>(srt.v[kb ^ 1]);
            w_heads<<<grid(m, 256), 256, 0, st>>>(srt.k[kb], m, 0, Uslot + a, H);
            rc = scan<uint64_t, OpMax<uint64_t>, true>(H, m, scr, st);
            if (rc) return rc;
            w_rank<<<grid(m, 256), 256, 0, st>>>(srt.k[kb], srt.v[kb], H, m, rank, C);
            rc = scan<uint32_t, OpSum<uint32_t>, true>(C, m, scr, st);
            if (rc) return rc;
            uint32_t kept = 0;
            if (cudaMemcpyAsync(&kept, C + m - 1, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                return GALN_ECUDA;
            // the chunk's slots aside (H is consumed), then compacted into U in place: every write lands at
            // or before the chunk's own start
            w_copy_u64<<<grid(m, 256), 256, 0, st>>>(Uslot + a, m, H);
            w_compact<<<grid(m, 256), 256, 0, st>>>(srt.v[kb], C, m, 0, H, out, Upos, Uslot);
            out += kept;
            a = e;
        }
        u_n = out;
        h2 *= 2;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : GALN_ECUDA;
}

}  // namespace ixb

// The 64-bit device part (see the 64-bit path above): forward sequence (host) -> <prefix>.bwt and
// <prefix>.sa. chunk: suffixes sorted at once (0: from free device memory).
static int dev_build_bwt_sa_wide(const uint8_t *F, uint64_t l_pac, const std::string &prefix, galn_build_stats *stats,
                                 uint64_t chunk)
{
    for (uint64_t i = 0; i < l_pac; ++i)
        if (F[i] > 3) return GALN_EINVAL;
    using namespace ixb;
    const uint64_t N = 2 * l_pac;
    if (l_pac == 0 || N >= (1ull << 40)) return GALN_EINVAL;
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return GALN_ECUDA;
    // fixed: text, ranks, bucket histogram, selection tile counts; per sorted suffix 32 bytes (keys, values)
    // plus radix tile counts; U: 16 bytes per unsorted suffix; the end: BWT bytes, block counts and body
    const uint64_t sel_tiles = (N + kWSelTile - 1) / kWSelTile;
    const size_t fixed = (size_t)N + 64 + (size_t)N * 8 + kWCodes * 8 + sel_tiles * 4 + (256ull << 20);
    if (!chunk) {
        const size_t spare = fr > fixed ? fr - fixed : 0;
        chunk = std::min<uint64_t>(N, std::max<uint64_t>(1 << 20, spare / 4 / 34));   // a quarter for sorting
        chunk = std::min<uint64_t>(chunk, 1ull << 31);
    }
    chunk = std::min<uint64_t>(chunk, N);
    const uint64_t rtiles = (chunk + kRTile - 1) / kRTile;
    const size_t sort_bytes = (size_t)chunk * 32 + rtiles * 1024 + (size_t)(chunk / 1000 + 4096) * 32;
    if (fixed + sort_bytes + (16ull << 20) > fr) {
        fprintf(stderr, "[galn index] a text of %llu symbols needs more than %.1f GB of device memory, %.1f GB free\n",
                (unsigned long long)N, (fixed + sort_bytes) / 1e9, fr / 1e9);
        return GALN_ENOMEM;
    }
    const uint64_t ucap = std::min<uint64_t>(N, (fr - fixed - sort_bytes - (16ull << 20)) / 16);
    cudaStream_t st;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return GALN_ECUDA;
    cudaFuncSetAttribute(radix_scatter<uint64_t, uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(ScatterSmem<uint64_t, uint64_t>));
    cudaFuncSetAttribute(w_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kWCodes * 4));
    const uint64_t nb = (N + 127) / 128, nw = (N + 15) / 16;
    const uint64_t body_words = 16 * nb - (8 - (nw - 8 * (nb - 1)));
    const uint64_t ns = (N + 32) / 32 - 1;
    uint64_t primary = 0;
    double ms_write = 0;
    int rc = 0;
    cudaEvent_t ea, e0, e1;
    cudaEventCreate(&ea);
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    Sorter<uint64_t> srt;
    Scratch scr;
    int rounds = 0;
    uint64_t sorted = 0;
    {
        DevMem m;
        uint8_t *T = m.get<uint8_t>(N + 64);
        uint64_t *rank = m.get<uint64_t>(N);
        unsigned long long *hist = m.get<unsigned long long>(kWCodes + 1);
        uint32_t *tcount = m.get<uint32_t>(sel_tiles);
        if (!T || !rank || !hist || !tcount) rc = GALN_ENOMEM;
        if (!rc) {
            cudaEventRecord(ea, st);
            // the forward half and its reverse complement, uploaded through the end of T (freed after)
            DevMem fm;
            uint8_t *F_d = fm.get<uint8_t>(l_pac);
            if (!F_d) rc = GALN_ENOMEM;
            if (!rc) {
                cudaMemcpyAsync(F_d, F, l_pac, cudaMemcpyHostToDevice, st);
                cudaEventRecord(e0, st);
                text_from_forward<<<grid(N, 256), 256, 0, st>>>(F_d, l_pac, T);
                cudaMemsetAsync(T + N, 0, 64, st);
                if (cudaStreamSynchronize(st) != cudaSuccess) rc = GALN_ECUDA;
            }
        }
        if (!rc) {
            DevMem sm;
            srt.k[0] = sm.get<uint64_t>(chunk);
            srt.k[1] = sm.get<uint64_t>(chunk);
            srt.v[0] = sm.get<uint64_t>(chunk);
            srt.v[1] = sm.get<uint64_t>(chunk);
            srt.counts = sm.get<uint32_t>(rtiles * 256);
            scr.cap = (size_t)(chunk / 1000 + 4096) * 32;
            scr.p = sm.get<unsigned char>(scr.cap);
            srt.scr = &scr;
            uint64_t *Upos = sm.get<uint64_t>(ucap), *Uslot = sm.get<uint64_t>(ucap);
            if (!srt.k[0] || !srt.k[1] || !srt.v[0] || !srt.v[1] || !srt.counts || !scr.p || !Upos || !Uslot)
                rc = GALN_ENOMEM;
            if (!rc) rc = wide_sort(T, N, rank, srt, scr, chunk, Upos, Uslot, ucap, tcount, hist, hist + kWCodes, st,
                                    rounds, sorted);
            if (rc) cudaStreamSynchronize(st);
        }
        if (!rc) {
            uint64_t r0 = 0;
            if (cudaMemcpyAsync(&r0, rank, 8, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                rc = GALN_ECUDA;
            primary = r0 + 1;
        }
        if (!rc) {
            DevMem em;
            uint8_t *L = em.get<uint8_t>(N);
            U4 *cnt = em.get<U4>(nb);
            uint32_t *body = em.get<uint32_t>(nb * 16);
            uint64_t *smp = em.get<uint64_t>(std::max<uint64_t>(ns, 1));
            scr.cap = (size_t)(nb / 100 + 4096) * 64;
            scr.top = 0;
            scr.p = em.get<unsigned char>(scr.cap);
            if (!L || !cnt || !body || !smp || !scr.p) rc = GALN_ENOMEM;
            if (!rc) {
                w_bwt_scatter<<<grid(N, 256), 256, 0, st>>>(T, rank, N, primary, L, smp);
                bwt_block_counts<<<grid(nb, 128), 128, 0, st>>>(L, N, nb, cnt);
                rc = scan<U4, OpSum<U4>, true>(cnt, nb, scr, st);
            }
            if (!rc) {
                bwt_write<<<grid(nb * 16, 256), 256, 0, st>>>(L, N, nb, cnt, body);
                U4 totals{};
                cudaEventRecord(e1, st);
                cudaMemcpyAsync(&totals, cnt + nb - 1, sizeof(U4), cudaMemcpyDeviceToHost, st);
                if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = GALN_ECUDA;
                const auto w0 = std::chrono::steady_clock::now();
                if (!rc) rc = write_index_files(prefix, primary, totals.c, N, body, body_words, smp, ns);
                ms_write = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - w0).count();
            }
            if (rc) cudaStreamSynchronize(st);
        }
        if (stats && !rc) {
            stats->n = N;
            stats->primary = primary;
            stats->rounds = rounds;
            stats->sorted_items = sorted;
            stats->sort_passes = srt.passes;
            stats->scatter_items = srt.scatter_items;
            float ms = 0, up = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            cudaEventElapsedTime(&up, ea, e0);
            stats->ms_device = ms;
            stats->ms_copies = up;
            stats->ms_files = ms_write;
            double sc = 0;
            for (size_t i = 0; i + 1 < srt.ev.size(); i += 2) {
                float x = 0;
                cudaEventElapsedTime(&x, srt.ev[i], srt.ev[i + 1]);
                sc += x;
            }
            stats->ms_scatter = sc;
        }
    }
    for (cudaEvent_t e : srt.ev) cudaEventDestroy(e);
    cudaEventDestroy(ea);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaStreamDestroy(st);
    if (rc == GALN_ECUDA) cudaGetLastError();
    return rc;
}

// The whole device part: forward sequence (host) -> <prefix>.bwt and <prefix>.sa. Which texts take the 64-bit path:
// galn_internal.h.
int dev_build_bwt_sa(const uint8_t *F, uint64_t l_pac, const std::string &prefix, galn_build_stats *stats,
                     const galn_build_how &how)
{
    using namespace ixb;
    const uint64_t N = 2 * l_pac;
    if (how.sort_chunk > 0 || (l_pac > 0 && N > 0xFFFFFFFFull - 64))
        return dev_build_bwt_sa_wide(F, l_pac, prefix, stats, how.sort_chunk > 0 ? (uint64_t)how.sort_chunk : 0);
    if (l_pac == 0) return GALN_EINVAL;
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return GALN_ECUDA;
    const uint64_t tiles = (N + kRTile - 1) / kRTile;
    const uint64_t nb = (N + 127) / 128, nw = (N + 15) / 16;
    const uint64_t body_words = 16 * nb - (8 - (nw - 8 * (nb - 1)));
    const uint64_t ns = (N + 32) / 32 - 1;
    // one allocation. K: round 0's two key arrays and its H and C, later the two arrays of 64-bit keys (H and C in the
    // free one), at the end the results; v: positions (the one that round 0 leaves sorted stays, as the suffix array)
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~(size_t)255; return o; };
    const size_t n4 = ((size_t)N * 4 + 255) & ~(size_t)255;
    const size_t o_w = take((nw + 4) * 4), o_rank = take(n4), o_k = take(4 * n4), o_v = take(3 * n4), o_s = take(2 * n4),
                 o_cnt = take(tiles * 1024), scr_cap = (size_t)(N / 1000 + 4096) * 32, o_scr = take(scr_cap),
                 o_bad = take(4);
    DevMem m;
    unsigned char *base = nullptr;
    if (at + ((size_t)64 << 20) <= fr && (how.max_block == 0 || at <= how.max_block)) base = m.get<unsigned char>(at);
    if (!base)   // none free, or not in one block (another program may have taken it): the 64-bit path sorts in pieces
        return dev_build_bwt_sa_wide(F, l_pac, prefix, stats, 0);
    cudaStream_t st;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return GALN_ECUDA;
    // per device: the attribute belongs to the current device's context
    cudaFuncSetAttribute(radix_scatter<uint64_t, uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(ScatterSmem<uint64_t, uint32_t>));
    cudaFuncSetAttribute(radix_scatter<uint32_t, uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(ScatterSmem<uint32_t, uint32_t>));
    uint64_t primary = 0;
    double ms_write = 0;
    int rc = 0;
    cudaEvent_t ea, e0, e1;   // upload start, text in HBM, results in HBM
    cudaEventCreate(&ea);
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    Sorter<uint32_t> srt, srt0l;           // later rounds, and round 0 with 64-bit keys
    Sorter<uint32_t, uint32_t> srt0;       // round 0 with 32-bit keys
    Scratch scr;
    {
        uint32_t *W = reinterpret_cast<uint32_t *>(base + o_w), *rank = reinterpret_cast<uint32_t *>(base + o_rank);
        unsigned char *kp = base + o_k;
        uint32_t *v[3], *slots[2];
        for (int t = 0; t < 3; ++t) v[t] = reinterpret_cast<uint32_t *>(base + o_v + t * n4);
        for (int t = 0; t < 2; ++t) slots[t] = reinterpret_cast<uint32_t *>(base + o_s + t * n4);
        uint8_t *F_d = reinterpret_cast<uint8_t *>(slots[0]);     // only until it is packed
        uint32_t *bad = reinterpret_cast<uint32_t *>(base + o_bad);
        scr.p = base + o_scr;
        scr.cap = scr_cap;
        srt.scr = srt0.scr = srt0l.scr = &scr;
        srt.counts = srt0.counts = srt0l.counts = reinterpret_cast<uint32_t *>(base + o_cnt);
        srt0.k[0] = reinterpret_cast<uint32_t *>(kp);
        srt0.k[1] = reinterpret_cast<uint32_t *>(kp + n4);
        srt.k[0] = srt0l.k[0] = reinterpret_cast<uint64_t *>(kp);
        srt.k[1] = srt0l.k[1] = reinterpret_cast<uint64_t *>(kp + 2 * n4);
        srt0.v[0] = srt0l.v[0] = v[0];
        srt0.v[1] = srt0l.v[1] = v[1];
        const bool long_keys = how.first_symbols ? how.first_symbols == kPrefixLong : N < kLongKeys;
        uint32_t h_bad = 0, kept = 0;
        int rounds = 0, kb = 0, sbuf = 0;
        uint64_t sorted = 0, M = N, h = long_keys ? kPrefixLong : kPrefixShort;
        const uint32_t *S = nullptr;
        uint32_t *sa = nullptr;                                   // row r + 1's suffix
        if (!rc) {
            cudaEventRecord(ea, st);
            cudaMemcpyAsync(F_d, F, l_pac, cudaMemcpyHostToDevice, st);
            cudaEventRecord(e0, st);
            cudaMemsetAsync(bad, 0, 4, st);
            pack_text<<<grid(nw + 4, 256), 256, 0, st>>>(F_d, l_pac, nw + 4, W, bad);
            cudaMemcpyAsync(&h_bad, bad, 4, cudaMemcpyDeviceToHost, st);
        }
        auto last_kept = [&](const uint32_t *C) -> int {
            if (cudaMemcpyAsync(&kept, C + M - 1, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                return GALN_ECUDA;
            return 0;
        };
        // round 0 over all N suffixes (H and C where the sorted keys are not); later rounds over the unsorted ones
        // (positions P, slots S)
        auto round0 = [&](auto sym, auto &s0) -> int {
            constexpr int SYM = decltype(sym)::value;
            pd_key0<SYM><<<grid(N, 256), 256, 0, st>>>(W, N, s0.k[0], s0.v[0]);
            int r = radix_sort(s0, 0, N, 2 * SYM, st, kb);
            if (r) return r;
            sorted = N;
            sa = v[kb];
            srt.v[0] = v[kb ^ 1];
            srt.v[1] = v[2];
            uint32_t *H = SYM == 16 || kb == 0 ? reinterpret_cast<uint32_t *>(kp + 2 * n4) : reinterpret_cast<uint32_t *>(kp);
            uint32_t *C = H + n4 / 4;
            pd_heads<SYM><<<grid(N, 256), 256, 0, st>>>(s0.k[kb], sa, (const uint32_t *)nullptr, N, N, H);
            r = scan<uint32_t, OpMax<uint32_t>, true>(H, N, scr, st);
            if (r) return r;
            pd_rank<SYM><<<grid(N, 256), 256, 0, st>>>(s0.k[kb], sa, H, (const uint32_t *)nullptr, N, N, rank, C,
                                                       (uint32_t *)nullptr);
            r = scan<uint32_t, OpSum<uint32_t>, true>(C, N, scr, st);
            if (!r) r = last_kept(C);
            if (!r && h_bad) r = GALN_EINVAL;
            if (!r && kept) pd_compact<<<grid(N, 256), 256, 0, st>>>(sa, S, C, N, srt.v[0], slots[0]);
            return r;
        };
        if (!rc) rc = long_keys ? round0(std::integral_constant<int, kPrefixLong>(), srt0l)
                                : round0(std::integral_constant<int, kPrefixShort>(), srt0);
        if (!rc && kept) {
            ++rounds;
            S = slots[0];
            sbuf = 1;
            M = kept;
            kb = 0;
        }
        while (!rc && kept) {
            const int lo_bits = bitlen(N);
            pd_key<<<grid(M, 256), 256, 0, st>>>(srt.v[kb], rank, M, N, h, lo_bits, srt.k[kb]);
            h *= 2;
            rc = radix_sort(srt, kb, M, lo_bits + bitlen(N - 1), st, kb);
            if (rc) break;
            sorted += M;
            const uint64_t *K = srt.k[kb];
            const uint32_t *P = srt.v[kb];
            // the other key buffer is free: two uint32 arrays of M
            uint32_t *H = reinterpret_cast<uint32_t *>(srt.k[kb ^ 1]);
            uint32_t *C = H + M;
            pd_heads<0><<<grid(M, 256), 256, 0, st>>>(K, P, S, M, N, H);
            rc = scan<uint32_t, OpMax<uint32_t>, true>(H, M, scr, st);
            if (rc) break;
            pd_rank<0><<<grid(M, 256), 256, 0, st>>>(K, P, H, S, M, N, rank, C, sa);
            rc = scan<uint32_t, OpSum<uint32_t>, true>(C, M, scr, st);
            if (!rc) rc = last_kept(C);
            if (rc || kept == 0) break;
            if (++rounds > kMaxRounds) { rc = GALN_EINVAL; break; }
            uint32_t *S2 = slots[sbuf];
            pd_compact<<<grid(M, 256), 256, 0, st>>>(P, S, C, M, srt.v[kb ^ 1], S2);
            S = S2;
            sbuf ^= 1;
            M = kept;
            kb ^= 1;
        }
        if (!rc) {
            uint32_t r0 = 0;
            if (cudaMemcpyAsync(&r0, rank, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                rc = GALN_ECUDA;
            primary = (uint64_t)r0 + 1;
            // nb * 32 and nb * 64 bytes (N / 4 and N / 2, a block more) and N / 4 of samples, in the keys' 16 N
            unsigned char *q = kp;
            U4 *cnt = reinterpret_cast<U4 *>(q);
            q += (nb * 32 + 255) & ~(uint64_t)255;
            uint32_t *body = reinterpret_cast<uint32_t *>(q);
            q += (nb * 64 + 255) & ~(uint64_t)255;
            uint64_t *smp = reinterpret_cast<uint64_t *>(q);
            if (!rc) {
                bwt_blocks<<<grid(nb * 32, 256), 256, 0, st>>>(W, sa, N, primary, nb, body, cnt);
                rc = scan<U4, OpSum<U4>, true>(cnt, nb, scr, st);
            }
            if (!rc) {
                bwt_counts<<<grid(nb * 8, 256), 256, 0, st>>>(nb, cnt, body);
                if (ns) sa_samples<<<grid(ns, 256), 256, 0, st>>>(sa, ns, smp);
                U4 totals{};
                cudaEventRecord(e1, st);
                cudaMemcpyAsync(&totals, cnt + nb - 1, sizeof(U4), cudaMemcpyDeviceToHost, st);
                if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = GALN_ECUDA;
                const auto w0 = std::chrono::steady_clock::now();
                if (!rc) rc = write_index_files(prefix, primary, totals.c, N, body, body_words, smp, ns);
                ms_write = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - w0).count();
            }
        }
        srt.ev.insert(srt.ev.end(), srt0.ev.begin(), srt0.ev.end());
        srt.ev.insert(srt.ev.end(), srt0l.ev.begin(), srt0l.ev.end());
        srt.passes += srt0.passes + srt0l.passes;
        srt.scatter_items += srt0.scatter_items + srt0l.scatter_items;
        if (stats && !rc) {
            stats->n = N;
            stats->primary = primary;
            stats->rounds = rounds;
            stats->sorted_items = sorted;
            stats->sort_passes = srt.passes;
            stats->scatter_items = srt.scatter_items;
            float ms = 0, up = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            cudaEventElapsedTime(&up, ea, e0);
            stats->ms_device = ms;
            stats->ms_copies = up;
            stats->ms_files = ms_write;
            double sc = 0;
            for (size_t i = 0; i + 1 < srt.ev.size(); i += 2) {
                float x = 0;
                cudaEventElapsedTime(&x, srt.ev[i], srt.ev[i + 1]);
                sc += x;
            }
            stats->ms_scatter = sc;
        }
        if (rc) cudaStreamSynchronize(st);
    }
    for (cudaEvent_t e : srt.ev) cudaEventDestroy(e);
    cudaEventDestroy(ea);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaStreamDestroy(st);
    if (rc == GALN_ECUDA) cudaGetLastError();
    return rc;
}

}  // namespace galn
