// galn_warp.cuh -- the heavy-read tier: one warp per read, many stack entries expanded at once.
//
// Why this is exact. With positive penalties (s_mm, s_gapo, s_gape > 0) every child of an entry popped from
// score bucket b goes to a bucket above b, except the exact-match child, which has score b and is pushed
// last, so it is the very next pop (src/bwtgap_hd.h:457-470 push order). Bucket b therefore receives no
// entry while it is being popped: its pops are the entries e_m, e_{m-1}, ..., e_1 (LIFO), each followed
// by its chain of exact-match children. Between two hits the expansion of a chain depends only on its
// first entry, the width arrays and max_diff, none of which change without a hit; so the chains of the
// top entries of bucket b can be expanded at the same time, in any order and on any lane.
//
// One wave takes up to kWE entries from the top of bucket b (entry 0 may be a pending exact child left by
// the previous wave). The warp runs in steps: in each step every busy lane expands one pop of its chain,
// and every idle lane takes the next entry not yet handed out (in entry order), so lanes stay busy however uneven the
// chains are. All lanes append their pushes to the warp's one log in global memory, each push with a tag: its entry, its
// list (one per distinct target bucket: b+s_mm, b+s_gapo, b+s_gape) and its place among the entry's pushes to that list, in
// the order bwt_match_gap pushes them. When a chain ends its lane writes the entry's record: lane, pops, pushes per list
// and prefix sums. A chain that pushes a score past n_stacks, or has no room left (pops of its lane, or the log), drops
// the entries past its own.
//
// Then the warp replays the entries in order exactly as the sequential search would pop them: the
// max_entries test before each pop, n_entries after each pop and push, the pop count, the trace hash, and
// the hits (handled one by one: best_score, max_diff, -R, gapped-hit de-duplication, gap_shadow, the record). A hit
// that changes neither max_diff nor a width test word leaves the chains behind it as they are; one that does drops
// them. Without the trace hash the entries are replayed at once from prefix sums; an entry that ends the replay
// otherwise (and, in trace mode, every entry) one pop at a time. The pushes of the replayed entries are committed to
// their buckets in replay order (per bucket: entry order, then pop order), so every bucket is the same LIFO as in the
// sequential search.
//
// Storage: each bucket is a chain of 64-entry chunks in the warp's arena (global memory), with its top
// chunk, fill and entry count in shared memory. The width test words, the query, the wave's entries and
// records are in shared memory; the log (and, in trace mode or for an entry replayed pop by pop, the data of each pop) in
// per-warp global areas. Reads the tier cannot take (length > 256, n_stacks > 128, a penalty <= 0, 32-byte
// entries) go to the thread tiers. Reads that outgrow the arena or the record buffer start anew in the team tier, which
// also takes over, as they stand, reads of many pops; with trace hashes, or without that tier, a read that outgrows a
// small arena goes to a warp with a big one, and what is left after a second pass to the thread tiers.
#pragma once

#include "galn_internal.h"
#include "galn_search.cuh"

namespace galn {

constexpr int kWMaxB = kWarpMaxStacks;   // buckets
constexpr int kWMaxLen = kWarpMaxLen;    // read length
constexpr int kWE = 192;         // entries per wave
constexpr int kEPL = kWE / 32;   // entries per lane in the replay and commit scans (lane j: entries kEPL*j ..)
static_assert(kWE % 32 == 0 && kWMaxB % 32 == 0, "wave and bucket layouts");
// Room per lane and wave: a chain that meets its end drops every chain behind its own, so long chains (150 bp reads
// in repeats: up to a pop per base, three pushes each) must fit. With 48 pops and 128 pushes half as many pops again
// were thrown away on a 310 Mbp repeat-rich genome, and its heaviest read took 1080 M cycles; with 96 and 240, 6%, 314 M.
constexpr int kWP = 96;          // pops per lane per wave
constexpr int kWLog = kWarpLog;  // staged pushes per warp and wave
static_assert(kWP * 9 < 1024 && kWE <= 256, "a staged push's tag: 10 bits of place, 8 of entry");
constexpr int kWCH = kWarpChunk;  // entries per chunk
constexpr int kWNewC = kWLog / kWCH + 6;   // chunks one commit may allocate
constexpr int kWGrabPops = 6;    // an idle lane takes an entry only with room for this many pops
constexpr int kWChain = kWE / kWCH + 2;   // chunks of the current bucket kept walked
constexpr int kFC = 64;          // free chunk ids kept in shared memory

constexpr int kWDbgN = 15;       // optional counters per read (the kDbg* list below)

// a warp's share of a wave
struct WaveRec {
    uint4 ent[kWE];                   // the entries, in pop order
    uint32_t e_info[kWE];             // per entry: lane (bits 0-7), first pop (8-15), pops (16-23), end code (24-31)
    uint16_t e_cnt[3][kWE];           // per entry and list: staged pushes; in the commit, those of the entries before it
    uint32_t e_a[kWE];                // per entry: net change of n_entries (signed, bits 0-15), its highest value before a pop (16-31)
    uint32_t e_b[kWE];                // per entry: highest value after a pop (bits 0-15), index blocks read (16-31)
    int32_t log_n;                    // staged pushes so far
};

struct WarpSmem {
    int32_t top_chunk[kWMaxB];
    int32_t n_in[kWMaxB];
    uint16_t top_cnt[kWMaxB];
    uint32_t mask[kWMaxB / 32];
    uint32_t T[kWMaxLen + 1];         // the width and seed-width test words (width_word)
    uint32_t ST[kWMaxLen + 1];
    uint8_t q[kWMaxLen];
    WaveRec w;
    int32_t newc[kWNewC];             // chunks allocated for one commit
    int32_t wch[kWChain];             // the current bucket's chunks from its top, as far as walked
    int32_t fcache[kFC];              // the top of the warp's free-chunk stack
    BatchOpt O;                       // the read's batch options (read from here, not held in registers)
    unsigned long long dv[kWDbgN];    // optional counters of this read (profiling runs)
    long long t_mark, t_read;
};

// Per-warp data that is written often but read rarely (at hits, pending children and the one entry a wave
// replays pop by pop), kept in global memory to leave shared memory for more resident warps.
struct WSide {
    uint4 lane_x[32];                 // pending exact child of a lane that stopped mid-chain
    uint4 hz[kWE];                    // the hit of an entry that ended in one, and its interval
    uint64_t hk[kWE], hl[kWE];
    uint64_t wb[kWMaxLen + 1];        // the width array (bid << 48 | w), which only a hit reads
    // per pop of each lane: pushes (bits 0-3, the fused exact child not counted), has an exact child
    // (bit 4), index blocks read (bits 5-15). Pop-major: the lanes of one step write neighbouring halfwords,
    // so a step's writes fill a few sectors instead of touching one sector per lane.
    uint16_t meta[kWP][32];
};

template <class P>
struct WArgs {
    IndexViewT<P> ix;
    const uint8_t *query;
    const int64_t *off;
    const int32_t *bidx;
    const int32_t *maxdiff;
    const BatchOpt *bopt;
    int seed_len;
    const int32_t *list;
    int n;
    int32_t *claim;
    int n_warps;
    uint4 *chunks;            // n_warps * arena_chunks * kWCH entries
    int32_t *chunk_prev;      // n_warps * arena_chunks
    int32_t *free_ids;        // n_warps * arena_chunks
    int arena_chunks;
    uint64_t *aln;            // n_warps * aln_cap * 3
    int aln_cap;
    uint4 *log;               // n_warps * kWLog staged pushes
    uint32_t *tags;           // and, with 64-bit positions, their tags
    uint4 *prec;              // n_warps * 32 lanes * kWP popped entries (trace mode)
    WSide *side;              // n_warps
    int32_t *out_n;
    int64_t *out_off;
    uint64_t *out_pops, *out_trace;
    int32_t *out_peak;
    uint32_t *out_fetch;
    int8_t *out_tier;
    int tier;
    uint64_t *out_rec;
    unsigned long long *rec_top;
    int64_t rec_cap;
    int32_t *ovf;
    int32_t *ovf_n;
    // Warps 0..n_big-1 have arenas of big_chunks chunks (room for the max_entries cut-off); the others
    // arena_chunks. A read that outgrows a small arena is queued in ovq (its tail at q_ctl[1]) for the big
    // warps, which take queued reads before new ones (q_ctl: 0 head, 1 tail, 2 small warps finished,
    // 3 set when a big warp gave up waiting; the host then re-runs every queued read).
    int n_big, big_chunks;
    int32_t *ovq;
    int32_t *q_ctl;
    uint64_t q_wait_ns;       // a big warp gives up waiting for queued work after this long
    unsigned long long *dbg;  // optional counters (kWDbg entries), or NULL
    // A read that has taken team_pops pops (0: none) leaves for the team tier as it stands, written to `save`
    // (save_top, in 16-byte units, counts what is taken of save_cap): its id, place and entries to the team lists.
    // When the space is used up it stays.
    unsigned long long team_pops;
    uint4 *save;
    unsigned long long *save_top, save_cap;
    int32_t *team_list, *team_n, *team_key;
    uint32_t *team_src;
};

// A read's state between two waves, as the team tier takes it over: this header, its records (24 bytes each, padded to
// 16), then the entries of its buckets, lowest bucket first, each from the bottom of its stack to the top.
struct __align__(16) SaveHdr {
    uint4 px;                         // the pending exact child
    uint64_t pops;
    int32_t n_entries, peak, best_score, best_cnt, n_aln, max_diff, pend, pend_b;
    uint32_t f_alg, pad;
    int32_t n_in[kWMaxB];
    uint32_t ST[kWMaxLen + 4];
    uint64_t wb[kWMaxLen + 2];
};
static_assert(sizeof(SaveHdr) % 16 == 0, "entries follow the header in 16-byte units");
__host__ __device__ inline uint32_t save_entries_at(int n_aln) { return (uint32_t)(sizeof(SaveHdr) / 16 + (24u * (uint32_t)n_aln + 15u) / 16u); }

// optional counters of the warp tier (per launch, summed over warps)
enum { kDbgReads, kDbgWaves, kDbgLanes, kDbgConsumed, kDbgPops, kDbgCont, kDbgHazard, kDbgCycChain,
       kDbgCycReplay, kDbgCycCommit, kDbgCycLoad, kDbgChainPops, kDbgCycRead, kDbgSteps, kDbgCycReadMax, kWDbg };
static_assert(kWDbg == kWDbgN, "counter list");

// profiling helpers: lane 0 keeps the read's counters in shared memory
#define WDBG_ADD(K, V) do { if (dbg && lane == 0) S->dv[K] += (unsigned long long)(V); } while (0)
#define WDBG_LAP(K) do { if (dbg && lane == 0) { long long t_ = clock64(); S->dv[K] += (unsigned long long)(t_ - S->t_mark); S->t_mark = t_; } } while (0)

// an entry in registers (the score is the bucket of the wave)
template <class P>
using WEnt = Fields<P>;

template <class P>
__device__ __forceinline__ uint4 wpack(const WEnt<P> &x)
{
    return pack_entry(x.k, x.l, x.i, x.n_mm, x.n_gapo, x.n_gape, x.n_ins, x.state, x.is_diff);
}

template <class P>
__device__ __forceinline__ WEnt<P> wunpack(uint4 v)
{
    WEnt<P> x;
    unpack_entry(v, x);
    return x;
}

// an entry from its interval and a packed entry whose interval is zero
__device__ __forceinline__ uint4 with_interval(uint32_t k, uint32_t l, uint4 rest) { return make_uint4(k, l, rest.z, rest.w); }
__device__ __forceinline__ uint4 with_interval(uint64_t k, uint64_t l, uint4 rest)
{
    return make_uint4((uint32_t)k, rest.y | ((uint32_t)(k >> 32) & 0x3fu), (uint32_t)l, rest.w | ((uint32_t)(l >> 32) & 0x3fu));
}

// A staged push's tag: its entry in the wave (bits 0-11), its list (12-13) and its place among that entry's pushes to the
// list (14-23). In the warp tier with 32-bit positions it sits in the entry's spare bits (8 bits are enough for the
// entry there, and positions in a read are at most 256, 9 of i's 16 bits); else in a word beside it.
__device__ __forceinline__ uint4 tag_push(uint4 v, int e, int L, int place)
{
    v.z |= (uint32_t)(e & 63) << 26 | (uint32_t)(e >> 6) << 9 | (uint32_t)L << 11;
    v.w |= (uint32_t)place << 22;
    return v;
}
__device__ __forceinline__ uint32_t tag_word(int e, int L, int place) { return (uint32_t)e | (uint32_t)L << 12 | (uint32_t)place << 14; }
__device__ __forceinline__ uint32_t untag_push(uint4 &v)   // the tag as a word, taken out of the entry
{
    const uint32_t t = v.z >> 26 | ((v.z >> 9) & 3u) << 6 | ((v.z >> 11) & 3u) << 12 | (v.w >> 22) << 14;
    v.z &= 0x03ff01ffu;
    v.w &= 0x003fffffu;
    return t;
}

// one asynchronous 16-byte copy from global to shared memory, through L2 (cp.async.cg: staged pushes were
// written by other lanes of the warp), and the wait for all of the thread's copies
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(s), "l"(gsrc) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

struct WCtx {
    int len, max_diff, max_diff0, use_seed, seed_len_r;
    bool gape, nonstop;
};

// The exact walk of a pop with no difference left (bwt_match_exact_alt, src/bwtgap_hd.h:195-211), kept
// across steps: one LF step per warp step, so that it shares the step's single index fetch with the other
// lanes' pops instead of stalling the warp for its whole length.
template <class P>
struct WWalk {
    P k, l;
    int i;                 // bases left to match (positions i-1 .. 0)
    uint32_t f;            // index blocks read by the walk so far
    bool on;
};

// One step of a lane's chain: a pop, or one LF step of a pop's exact walk. Returns the chain's end code:
// -2 = the pop's exact walk goes on (no pop finished), -1 = the pop finished and the chain continues with
// its exact child (now in x), 0 = the chain is finished, 1 = a hit at this pop (kept in D->hz[ce]), 2 = stopped with
// the exact child pending (no room left in this wave; the child is in D->lane_x), 3 = this pop pushes a
// score >= n_stacks (bwt_match_gap returns BWTGAP_ERR_SCORE there). A finished pop's data goes to
// mt (and, with rec, to D->meta[lp][lane]); its pushes are appended to the warp's log (tl: the list of each
// push kind, mismatch, gap open, gap extension; nl0-nl2: the entry's pushes per list so far); in trace mode the popped
// entry goes to pr[lp]. full: the log has no room for another step after this one.
// H: where hits are kept (by entry). EMB: tags sit in the entries.
template <bool TRACE, int ST, class P, bool EMB, class SM, class HS>
__device__ __forceinline__ int lane_step(const IndexViewT<P> &ix, const BatchOpt &O, const WCtx &c, const SM *S, WSide *D, HS *H,
                                         int lane, int ce, bool rec, bool full, WEnt<P> &x, WWalk<P> &wk, int b, uint32_t &fetches,
                                         uint4 *log, uint32_t *tags, int *log_n, const int tl[3], uint4 *pr, int &lp,
                                         int &nl0, int &nl1, int &nl2, uint32_t &mt)
{
    bool err = false;
    uint32_t npu = 0;
    int endc = -2;
    bool load = false;           // this step reads Occ at (k1, l1)
    P k1 = 0, l1 = 0;
    int diffs = 0, m = 0, i = x.i;
    // ---- before the fetch: the tests that need no index data ----
    if (wk.on) {
        if (S->q[wk.i - 1] > 3) { wk.on = false; mt = wk.f << 5; endc = 0; }
        else { load = true; k1 = wk.k - 1; l1 = wk.l; }
    } else {
        if (TRACE) pr[lp] = wpack<P>(x);
        diffs = x.n_mm + x.n_gapo + (c.gape ? x.n_gape : 0);
        m = c.max_diff - diffs;
        if (m < 0 || (i > 0 && m < (int)(S->T[i] & kBid))) {
            mt = 0; endc = 0;
        } else if (i == 0) {
            H->hz[ce] = wpack<P>(x); H->hk[ce] = x.k; H->hl[ce] = x.l;
            mt = 0; endc = 1;
        } else if (m == 0 && (x.state == kStM || c.gape || x.n_gape == O.max_gape)) {
            // bwt_match_exact_alt over positions i-1 .. 0
            if (S->q[i - 1] > 3) { mt = 0; endc = 0; }
            else { wk.on = true; wk.k = x.k; wk.l = x.l; wk.i = i; wk.f = 0; load = true; k1 = x.k - 1; l1 = x.l; }
        } else {
            load = true; k1 = x.k - 1; l1 = x.l;
        }
    }
    // ---- the step's one fetch ----
    P ck[4], cl[4];
    uint32_t df = 0;
    if (load) {
        const uint32_t f0 = fetches;
        occ4_pair_u<ST, P>(ix, k1, l1, ck, cl, fetches);
        df = fetches - f0;
    }
    if (load && wk.on) {
        // one LF step of the exact walk
        const int cc = S->q[wk.i - 1];
        const P kk = ix.C[cc] + sel4(cc, ck[0], ck[1], ck[2], ck[3]) + 1;
        const P ll = ix.C[cc] + sel4(cc, cl[0], cl[1], cl[2], cl[3]);
        wk.f += df;
        if (kk > ll) { wk.on = false; mt = wk.f << 5; endc = 0; }
        else if (--wk.i == 0) {
            wk.on = false;
            H->hz[ce] = wpack<P>(x); H->hk[ce] = kk; H->hl[ce] = ll;
            mt = wk.f << 5; endc = 1;
        } else { wk.k = kk; wk.l = ll; }
    } else if (load) {
        // the expansion of the pop (src/bwtgap_hd.h:396-470) as nine predicated push slots in the order
        // bwt_match_gap pushes them: the gap child that keeps the interval (insertion open or extension), the
        // four deletion children (open or extension), the mismatches; then the exact child
        --i;
        P kk[4], ll[4];
        uint32_t ex = 0;             // bit q: the child of base q exists
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            kk[q] = ix.C[q] + ck[q] + 1; ll[q] = ix.C[q] + cl[q];
            if (kk[q] <= ll[q]) ex |= 1u << q;
        }
        const uint64_t occ = (uint64_t)x.l - x.k + 1;
        int allow_diff = 1, allow_M = 1;
        if (i > 0) {
            const uint32_t tw = S->T[i];
            const int ba = (int)(tw & kBid), bb = (int)((tw >> 15) & kBid);
            if (ba > m - 1) allow_diff = 0;
            else if (ba == m - 1 && bb == m - 1 && ((tw >> 30) & 1u)) allow_M = 0;
            int ii = i - (c.len - c.seed_len_r);
            if (c.use_seed && ii > 0) {
                int m_seed = O.max_seed_diff - diffs;
                const uint32_t ts = S->ST[ii];
                const int sba = (int)(ts & kBid), sbb = (int)((ts >> 15) & kBid);
                if (sba > m_seed - 1) allow_diff = 0;
                else if (sba == m_seed - 1 && sbb == m_seed - 1 && ((ts >> 30) & 1u)) allow_M = 0;
            }
        }
        const int gaps = x.n_gapo + x.n_gape;
        const int tmp = (O.mode & kModeLoggap) ? (gaps ? (31 - __clz(gaps)) : 0) / 2 + 1 : gaps;
        const bool indel = allow_diff && i >= O.indel_end_skip + tmp && c.len - i >= O.indel_end_skip + tmp;
        const bool st_m = x.state == kStM, st_i = x.state == kStI;
        const bool open_ok = indel && st_m && x.n_gapo < O.max_gapo;
        const bool ext_i = indel && st_i && x.n_gape < O.max_gape;
        const bool ext_d = indel && x.state == kStD && x.n_gape < O.max_gape
                           && (gaps < c.max_diff || occ < (uint64_t)(int64_t)O.max_del_occ);
        // which slots push: gs bit 0 the kept-interval gap child (insertion: open from M, extension from I), bits 1-4
        // deletions by base (open from M, extension from D); ms bit j - 1 the mismatch to base (base + j) & 3, j = 1..4
        // (j = 4, the read's own base, is a mismatch only where that base is ambiguous)
        const int base = S->q[i];
        const uint32_t gs = ((open_ok || ext_i) ? 1u : 0u) | ((open_ok || ext_d) ? ex << 1 : 0u);
        uint32_t ms = ((ex | (ex << 4)) >> ((base + 1) & 3)) & (base > 3 ? 0xfu : 0x7u);
        if (!(allow_diff && allow_M)) ms = 0;
        // list and bucket of each slot kind (a gap open from M, an extension otherwise)
        const int g_list = st_m ? tl[1] : tl[2];
        const int g_bkt = b + (st_m ? O.s_gapo : O.s_gape);
        const int m_bkt = b + O.s_mm;
        // a push at or past n_stacks ends the read (BWTGAP_ERR_SCORE); nothing else of this pop matters then
        err = (gs && g_bkt >= O.n_stacks) || (ms && m_bkt >= O.n_stacks);
        if (!err) {
            // the gap children go to list g_list and the mismatches to list 0 (tl[0]), each kind in slot order; when
            // both kinds share list 0 the mismatches follow the gap children, as bwt_match_gap pushes them. All
            // lanes of the warp append to one log, in any order: each push's tag says where it belongs. A list per
            // lane and target took 220 MB over all warps, past L2, and its half-filled sectors went to DRAM and back;
            // with the log (and a commit that reads it in order instead of searching each place's entry) a pop took
            // 356 cycles instead of 383 on aDNA reads, 245 instead of 275 on high-divergence ones.
            const int ng = __popc(gs), nm = __popc(ms);
            npu = (uint32_t)(ng + nm);
            if (npu) {
                const int at = atomicAdd(log_n, (int)npu);
                uint4 *p = log + at;
                uint32_t *tg = tags + at;
                auto put = [&](int o, P k, P l, const uint4 &rest, int L, int place) {
                    const uint4 v = with_interval(k, l, rest);
                    if (EMB) p[o] = tag_push(v, ce, L, place);
                    else { p[o] = v; tg[o] = tag_word(ce, L, place); }
                };
                if (gs) {
                    int gi = g_list == 0 ? nl0 : (g_list == 1 ? nl1 : nl2);
                    const int go = st_m ? 1 : 0, ge = st_m ? 0 : 1;
                    const uint4 rs = pack_entry((P)0, (P)0, i, x.n_mm, x.n_gapo + go, x.n_gape + ge, x.n_ins + 1, kStI, 1);
                    const uint4 rd = pack_entry((P)0, (P)0, i + 1, x.n_mm, x.n_gapo + go, x.n_gape + ge, x.n_ins, kStD, 1);
                    if (gs & 1u) { put(0, x.k, x.l, rs, g_list, gi++); ++p; ++tg; }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (gs & (2u << q)) { put(0, kk[q], ll[q], rd, g_list, gi++); ++p; ++tg; }
                    if (g_list == 0) nl0 = gi;
                    else if (g_list == 1) nl1 = gi;
                    else nl2 = gi;
                }
                const uint4 rm = pack_entry((P)0, (P)0, i, x.n_mm + 1, x.n_gapo, x.n_gape, x.n_ins, kStM, 1);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int t = (q - base - 1) & 3;
                    const int o = __popc(ms & ((1u << t) - 1u));
                    if ((ms >> t) & 1u) put(o, kk[q], ll[q], rm, 0, nl0 + o);
                }
                nl0 += nm;
            }
        }
        if (err) {   // the read ends at this pop with BWTGAP_ERR_SCORE
            mt = df << 5; endc = 3;
        } else {
            const bool exact = base < 4 && ((ex >> base) & 1u);
            mt = npu | (exact ? 16u : 0u) | df << 5;
            endc = exact ? -1 : 0;
            if (exact) {
                x.k = sel4(base, kk[0], kk[1], kk[2], kk[3]); x.l = sel4(base, ll[0], ll[1], ll[2], ll[3]);
                x.i = i; x.is_diff = 0; x.state = kStM;
            }
        }
    }
    if (endc == -2) return endc;
    if (TRACE || rec) D->meta[lp][lane] = (uint16_t)mt;
    ++lp;
    // no room for one more pop
    if (endc == -1 && (lp == kWP || full)) {
        endc = 2;
        D->lane_x[lane] = wpack<P>(x);
    }
    return endc;
}

// A hit, as bwt_match_gap handles it (the whole warp; h packed, its interval k, l; T the width test words, wb the width
// array): 0 = chains expanded past it are still right (nothing they depend on changed: max_diff and the test words
// are as before), 1 = they are not, 2 = the read ends here.
template <class P>
__device__ __forceinline__ int take_hit(const IndexViewT<P> &ix, const BatchOpt &O, WCtx &c, uint32_t *T, uint64_t *wb,
                                        uint4 packed, uint64_t k, uint64_t l, uint64_t *aln, int aln_cap, int &n_aln,
                                        int &best_score, int &best_cnt, int &ret, int lane)
{
    const unsigned FULL = 0xffffffffu, lt_mask = (1u << lane) - 1u;
    const WEnt<P> h = wunpack<P>(packed);
    const int sc = h.n_mm * O.s_mm + h.n_gapo * O.s_gapo + h.n_gape * O.s_gape;
    const int diffs = h.n_mm + h.n_gapo + (c.gape ? h.n_gape : 0);
    bool changed = false;
    if (n_aln == 0) {
        best_score = sc;
        if (!c.nonstop) {
            const int md = diffs + 1 > c.max_diff0 ? c.max_diff0 : diffs + 1;
            changed = md != c.max_diff;
            c.max_diff = md;
        }
    }
    if (sc == best_score) best_cnt = (int)(uint32_t)((uint64_t)(int64_t)best_cnt + (l - k + 1));
    else if (best_cnt > O.max_top2) return 2;
    if (h.n_gapo) {   // a gapped hit found before is not recorded again
        bool dup = false;
        for (int q0 = 0; q0 < n_aln && !dup; q0 += 32) {
            const int q = q0 + lane;
            dup = __any_sync(FULL, q < n_aln && aln[3 * q + 1] == k && aln[3 * q + 2] == l);
        }
        if (dup) return changed ? 1 : 0;
    }
    // gap_shadow on the width array, then the test words of the positions it reached
    const int ldp = h.is_diff ? h.i : 0;
    const uint64_t xx = (uint64_t)(int64_t)(int)(l - k + 1);
    int jb = 0;
    for (int t0 = 0; t0 < ldp; t0 += 32) {
        const int tt = t0 + lane;
        const uint64_t v = tt < ldp ? wb[tt] : 0, wv = v & kW48;
        const bool eq = tt < ldp && wv == xx, gt = tt < ldp && wv > xx;
        const unsigned bal = __ballot_sync(FULL, eq);
        const int rank = __popc(bal & lt_mask);
        if (gt) wb[tt] = (v & ~kW48) | (wv - xx);
        if (eq) wb[tt] = (1ull << 48) | (((uint64_t)ix.seq_len - (uint64_t)(jb + rank + 1)) & kW48);
        jb += __popc(bal);
    }
    __syncwarp();
    bool words = false;
    for (int t = 1 + lane; t <= ldp; t += 32) {
        const uint32_t w = width_word(wb[t - 1], wb[t]);
        words = words || w != T[t];
        T[t] = w;
    }
    if (__any_sync(FULL, words)) changed = true;
    __syncwarp();
    if (n_aln == aln_cap) { ret = kErrAln; return 2; }
    if (lane == 0) {
        const int n_del = h.n_gapo + h.n_gape - h.n_ins;
        aln[3 * n_aln] = (uint64_t)(h.n_mm & 0xff) | (uint64_t)(h.n_gapo & 0xff) << 8
                       | (uint64_t)(h.n_gape & 0xff) << 16 | (uint64_t)(sc & 0xfffff) << 24
                       | (uint64_t)(h.n_ins & 0x3ff) << 44 | (uint64_t)(n_del & 0x3ff) << 54;
        aln[3 * n_aln + 1] = k;
        aln[3 * n_aln + 2] = l;
    }
    __syncwarp();
    ++n_aln;
    return changed ? 1 : 0;
}

// The widths of a read (which = 0: the width array wb and the test words T) or of its seed (which = 1: the words ST), on
// one thread each: two lanes run the two walks side by side and share a step's wait.
template <int ST_, class P>
__device__ __forceinline__ void width_walk(const IndexViewT<P> &ix, int len, int seed_len, int which, const uint8_t *q,
                                           uint64_t *wb, uint32_t *T, uint32_t *ST, uint32_t &fetches)
{
    WidthRun<P> w;
    w.k = 0; w.l = ix.seq_len; w.bid = 0; w.last = 0;
    const int n = which == 0 ? len : seed_len;
    if (which) q += len - n;
    uint32_t *words = which == 0 ? T : ST;
    for (int i = 0; i < n; ++i) {
        WidthFetch<ST_, P> f;
        f.load(ix, w);
        const uint64_t last = w.last, v = f.step(ix, w, width_base(q[i]), fetches);
        if (which == 0) wb[i] = v;
        words[i] = width_word(last, v);
    }
    if (which == 0) {
        const uint64_t v = (w.bid + 1) << 48;
        wb[len] = v;
        T[len] = width_word(w.last, v);
    }
}

// The chains of a wave's Wcap entries W->ent: idle lanes take the next entry, busy lanes pop, until every entry is done
// or no lane has room. Returns how many entries, from the first on, have their records in W (stops included); lp
// is the lane's pops.
template <bool TRACE, int ST, class P, class SM>
__device__ __forceinline__ int run_chains(const IndexViewT<P> &ix, const BatchOpt &O, const WCtx &c, const SM *S, WaveRec *W,
                                          WSide *D, int lane, bool rec, int Wcap, int b, uint32_t &fetches, uint4 *log,
                                          uint32_t *tags, const int tl[3], uint4 *prec, int &lp, unsigned long long *steps)
{
    const unsigned FULL = 0xffffffffu, lt_mask = (1u << lane) - 1u;
    int e_next = 0, limit = Wcap;                  // entries from limit on are dropped
    int ce = -1;                                   // this lane's entry
    int nl0 = 0, nl1 = 0, nl2 = 0;                 // its staged pushes per list
    int e_p0 = 0, e_np = 0, e_pre = 0, e_mpre = 0, e_pmax = 0;
    uint32_t e_fs = 0;
    lp = 0;
    WEnt<P> x;
    x.k = 0; x.l = 0; x.i = 0; x.is_diff = 0; x.n_mm = x.n_gapo = x.n_gape = x.n_ins = 0; x.state = 0;
    WWalk<P> wk;
    wk.k = 0; wk.l = 0; wk.i = 0; wk.f = 0; wk.on = false;
    if (lane == 0) W->log_n = 0;
    __syncwarp();
    for (;;) {
        // a step adds at most 9 pushes a lane; entries are handed out while the log holds kWGrabPops such steps
        const int used = *(volatile int32_t *)&W->log_n;
        const bool want = ce < 0 && lp + kWGrabPops <= kWP && used + 9 * 32 * kWGrabPops <= kWLog;
        const unsigned wb = __ballot_sync(FULL, want);
        if (wb && e_next < limit) {
            const int e = e_next + __popc(wb & lt_mask);
            if (want && e < limit) {
                ce = e;
                x = wunpack<P>(W->ent[e]);
                e_p0 = lp; e_np = 0; e_pre = 0; e_mpre = 0; e_pmax = 0; e_fs = 0;
                nl0 = nl1 = nl2 = 0;
            }
            e_next = min(limit, e_next + __popc(wb));
        }
        if (!__any_sync(FULL, ce >= 0)) break;
        if (steps && lane == 0) ++*steps;
        int stop_e = 0x7fffffff;
        if (ce >= 0) {
            uint32_t mt = 0;
            const int endc = lane_step<TRACE, ST, P, sizeof(P) == 4>(ix, O, c, S, D, D, lane, ce, rec, used + 2 * 9 * 32 > kWLog, x, wk, b,
                                              fetches, log, tags, &W->log_n, tl, prec, lp, nl0, nl1, nl2, mt);
            if (endc != -2) {                          // else an exact walk goes on
                ++e_np;
                if (e_pre > e_mpre) e_mpre = e_pre;     // n_entries before this pop, relative to the chain start
                e_pre += (int)(mt & 15u) + (int)((mt >> 4) & 1u) - 1;
                if (e_pre > e_pmax) e_pmax = e_pre;
                e_fs += mt >> 5;
                if (endc >= 0) {
                    W->e_info[ce] = (uint32_t)lane | (uint32_t)e_p0 << 8 | (uint32_t)e_np << 16 | (uint32_t)endc << 24;
                    W->e_cnt[0][ce] = (uint16_t)nl0;
                    W->e_cnt[1][ce] = (uint16_t)nl1;
                    W->e_cnt[2][ce] = (uint16_t)nl2;
                    W->e_a[ce] = ((uint32_t)e_pre & 0xffffu) | (uint32_t)e_mpre << 16;
                    W->e_b[ce] = (uint32_t)e_pmax | e_fs << 16;
                    if (endc > 1) stop_e = ce;
                    ce = -1;
                }
            }
        }
        __syncwarp();
        // a stop (no room, or an error) drops the entries past its own; a hit does not stop the wave
        if (__any_sync(FULL, stop_e != 0x7fffffff)) {
            limit = min(limit, (int)__reduce_min_sync(FULL, stop_e) + 1);
            if (ce >= limit) { ce = -1; wk.on = false; }
        }
    }
    __syncwarp();
    return min(e_next, limit);
}

// The pushes staged for one list by a share of n <= kWE entries (cnt: per entry): their total, and in cnt per entry
// `start` and those of the entries before it. MAX: the most that start and the share's pushes can come to.
template <uint32_t MAX, class C>
__device__ __forceinline__ int share_counts(C *cnt, int n, int lane, int start = 0)
{
    static_assert(MAX <= (C)~(C)0, "the counts of a share's entries add up past their type");
    int cnt_k[kEPL], lsum = 0;
#pragma unroll
    for (int k = 0; k < kEPL; ++k) {
        const int e = kEPL * lane + k;
        cnt_k[k] = e < n ? (int)cnt[e] : 0;
        lsum += cnt_k[k];
    }
    int incl = lsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const int T = __shfl_sync(0xffffffffu, incl, 31);
    if (T) {
        int run = start + incl - lsum;
#pragma unroll
        for (int k = 0; k < kEPL; ++k) {
            const int e = kEPL * lane + k;
            if (e < n) cnt[e] = (C)run;
            run += cnt_k[k];
        }
    }
    __syncwarp();
    return T;
}

// Stores the n logged pushes of the wave's first `consumed` entries where they belong: place(e, L, t) is the place of
// entry e's push t to list L. The log is read in order, kUnroll rounds of 32 pushes in flight.
template <bool EMB, class F>
__device__ __forceinline__ void copy_log(const uint4 *log, const uint32_t *tags, int n, int consumed, int lane, F place)
{
    constexpr int kUnroll = 4;
    for (int t0 = lane; t0 < n; t0 += 32 * kUnroll) {
        uint4 v[kUnroll];
        uint32_t tg[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int t = t0 + 32 * u;
            v[u] = t < n ? __ldcg(log + t) : make_uint4(0, 0, 0, 0);
            if (!EMB) tg[u] = t < n ? __ldcg(tags + t) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            if (EMB) tg[u] = untag_push(v[u]);
            const int e = (int)(tg[u] & 0xfffu);
            if (t0 + 32 * u < n && e < consumed) *place(e, (int)((tg[u] >> 12) & 3u), (int)(tg[u] >> 14)) = v[u];
        }
    }
}

// the warp's chunk allocator (warp-uniform state; every lane holds the same copy): a stack of free chunk
// ids whose top kFC entries live in shared memory (fc), the rest in global memory, then fresh chunks
struct WAlloc {
    int32_t *free_ids;
    int32_t *fc;
    int base, cap, bump, g_top, fc_n;
    // `need` chunk ids into out[0..need), lane-parallel; false if the arena is exhausted
    __device__ __forceinline__ bool alloc_n(int need, int32_t *out, int lane)
    {
        const int from_c = need < fc_n ? need : fc_n;
        const int from_g = need - from_c < g_top ? need - from_c : g_top;
        const int from_b = need - from_c - from_g;
        if (bump + from_b > cap) return false;
        for (int t = lane; t < need; t += 32) {
            int id;
            if (t < from_c) id = fc[fc_n - 1 - t];
            else if (t < from_c + from_g) id = free_ids[g_top - 1 - (t - from_c)];
            else id = base + bump + (t - from_c - from_g);
            out[t] = id;
        }
        fc_n -= from_c; g_top -= from_g; bump += from_b;
        __syncwarp();
        return true;
    }
    __device__ __forceinline__ void release(int id, int lane)
    {
        static_assert(kFC == 64, "spill layout");
        if (fc_n == kFC) {   // the cache's lower half to the global stack
            free_ids[g_top + lane] = fc[lane];
            const int v = fc[lane + 32];
            __syncwarp();
            fc[lane] = v;
            g_top += 32; fc_n -= 32;
        }
        if (lane == 0) fc[fc_n] = id;
        ++fc_n;
        __syncwarp();
    }
};

template <class P>
__device__ __forceinline__ uint64_t trace_pop(uint64_t h, uint32_t binfo, const WEnt<P> &y, int n_entries)
{
    h = trace_mix(h, binfo | (uint32_t)y.i);
    h = trace_mix(h, y.k);
    h = trace_mix(h, y.l);
    h = trace_mix(h, (uint64_t)((uint32_t)y.n_mm | (uint32_t)y.n_gapo << 8 | (uint32_t)y.n_gape << 16
                                | (uint32_t)y.state << 24));
    int n_del = y.n_gapo + y.n_gape - y.n_ins;
    h = trace_mix(h, (uint64_t)(y.n_ins & 0xffff) | (uint64_t)(n_del & 0xffff) << 16);
    h = trace_mix(h, (uint64_t)(uint32_t)(y.is_diff ? y.i : 0));
    h = trace_mix(h, (uint64_t)(uint32_t)n_entries);
    return h;
}

template <bool TRACE, int ST, class P>
__device__ void warp_read(const WArgs<P> &a, int r, int wid, WarpSmem *S, int lane)
{
    const unsigned FULL = 0xffffffffu;
    const int64_t s0 = a.off[r];
    const int len = (int)(a.off[r + 1] - s0);
    if (lane == 0) S->O = a.bopt[a.bidx[r]];
    __syncwarp();
    const BatchOpt &O = S->O;
    const int max_diff0 = a.maxdiff[r];
    const IndexViewT<P> &ix = a.ix;
    for (int t = lane; t < len; t += 32) S->q[t] = a.query[s0 + t];
    for (int t = lane; t < kWMaxB; t += 32) { S->top_chunk[t] = -1; S->n_in[t] = 0; S->top_cnt[t] = 0; }
    if (lane < kWMaxB / 32) S->mask[lane] = 0;
    __syncwarp();
    uint32_t fetches = 0;   // index blocks read by this lane (chains include discarded speculation)
    const bool use_seed = len > O.seed_len;
    WSide *D = a.side + wid;
    if (lane < 2) width_walk<ST, P>(ix, len, use_seed ? O.seed_len : 0, lane, S->q, D->wb, S->T, S->ST, fetches);
    __syncwarp();
    // algorithmic count: widths, then replayed chains
    uint32_t f_alg = __shfl_sync(FULL, fetches, 0) + __shfl_sync(FULL, fetches, 1);
    uint4 *chunks = a.chunks;
    WAlloc A;
    {
        const bool big = wid < a.n_big;
        const int64_t base = big ? (int64_t)wid * a.big_chunks
                                 : (int64_t)a.n_big * a.big_chunks + (int64_t)(wid - a.n_big) * a.arena_chunks;
        A.free_ids = a.free_ids + base;
        A.fc = S->fcache;
        A.base = (int)base; A.cap = big ? a.big_chunks : a.arena_chunks; A.bump = 0; A.g_top = 0; A.fc_n = 0;
    }
    uint4 *log = a.log + (size_t)wid * kWLog;
    uint32_t *tags = a.tags + (size_t)wid * kWLog;
    uint4 *prec_w = a.prec + (size_t)wid * 32 * kWP;                 // pop t of lane j at + j * kWP + t
    // the staging list of each push kind: kinds whose target buckets coincide share a list, so the
    // bucket keeps the push order
    int tl[3];
    tl[0] = 0;
    tl[1] = O.s_gapo == O.s_mm ? 0 : 1;
    tl[2] = O.s_gape == O.s_mm ? 0 : (O.s_gape == O.s_gapo ? tl[1] : 2);
    const int lst_pen[3] = {O.s_mm, tl[1] == 1 ? O.s_gapo : -1, tl[2] == 2 ? O.s_gape : -1};
    uint64_t *aln = a.aln + (size_t)wid * a.aln_cap * 3;

    WCtx c;
    c.len = len; c.max_diff0 = max_diff0; c.max_diff = max_diff0; c.use_seed = use_seed;
    c.seed_len_r = len > O.seed_len ? O.seed_len : 0x7fffffff;
    c.gape = (O.mode & kModeGape) != 0; c.nonstop = (O.mode & kModeNonstop) != 0;
    const int n_stacks = O.n_stacks;
    int best_score = (max_diff0 + 1) * O.s_mm + (O.max_gapo + 1) * O.s_gapo + (O.max_gape + 1) * O.s_gape;
    int best_cnt = 0, n_aln = 0, ret = 0, n_entries = 0, peak = 0;
    uint64_t pops = 0, trace = kTraceInit;
    const bool dbg = a.dbg != nullptr;
    if (dbg && lane == 0) {
        for (int q = 0; q < kWDbgN; ++q) S->dv[q] = 0;
        S->t_read = clock64();
    }

    bool left_read = false;      // it left for the team tier
    int n_amb = 0;
    for (int j = 0; j < len; ++j) n_amb += S->q[j] > 3;
    if (n_amb > c.max_diff) goto publish;

    {
        // the root is the pending entry of the first wave
        bool pend = true;
        int pend_b = 0;
        WEnt<P> px;
        px.k = 0; px.l = ix.seq_len; px.i = len; px.is_diff = 0; px.n_mm = px.n_gapo = px.n_gape = px.n_ins = 0;
        px.state = kStM;
        if (n_stacks <= 0) { ret = kErrScore; goto publish; }
        n_entries = 1; peak = 1;
        unsigned long long leave_at = a.team_pops ? a.team_pops : ~0ull;
        bool rec = TRACE;            // the wave keeps each pop's data (one entry, to be replayed pop by pop)
        int wch_b = -1, wch_n = 0;   // bucket whose chunk chain S->wch holds, and its length
        auto on_hit = [&](int e) -> int {
            return take_hit<P>(ix, O, c, S->T, D->wb, D->hz[e], D->hk[e], D->hl[e], aln, a.aln_cap, n_aln, best_score,
                               best_cnt, ret, lane);
        };
        for (;;) {
            if (n_entries == 0) break;
            if (n_entries > O.max_entries) break;
            if (!TRACE && pops >= leave_at) {
                // to the team tier
                unsigned held = 0;
                for (int t = lane; t < kWMaxB; t += 32) held += (unsigned)max(0, S->n_in[t]);
                const uint32_t at = save_entries_at(n_aln), need = at + __reduce_add_sync(FULL, held);
                unsigned long long o = 0;
                if (lane == 0) o = atomicAdd(a.save_top, (unsigned long long)need);
                o = __shfl_sync(FULL, o, 0);
                if (o + need > a.save_cap) leave_at = ~0ull;
                else {
                    SaveHdr *h = reinterpret_cast<SaveHdr *>(a.save + o);
                    if (lane == 0) {
                        h->px = wpack<P>(px); h->pops = pops; h->n_entries = n_entries; h->peak = peak;
                        h->best_score = best_score; h->best_cnt = best_cnt; h->n_aln = n_aln; h->max_diff = c.max_diff;
                        h->pend = pend; h->pend_b = pend_b; h->f_alg = f_alg;
                    }
                    for (int t = lane; t < kWMaxB; t += 32) h->n_in[t] = S->n_in[t];
                    for (int t = lane; t <= len; t += 32) { h->ST[t] = S->ST[t]; h->wb[t] = D->wb[t]; }
                    uint64_t *recs = reinterpret_cast<uint64_t *>(h + 1);
                    for (int t = lane; t < 3 * n_aln; t += 32) recs[t] = aln[t];
                    uint4 *dst = a.save + o + at;
                    for (int t = 0; t < kWMaxB; ++t) {
                        int left = S->n_in[t], ch = S->top_chunk[t], n = S->top_cnt[t];
                        if (left <= 0) continue;
                        uint4 *d = dst;
                        dst += left;
                        while (left > 0 && ch >= 0) {          // the top chunk's entries are the last ones
                            const int below = a.chunk_prev[ch];
                            n = min(n, left);
                            left -= n;
                            for (int j = lane; j < n; j += 32) d[left + j] = chunks[(size_t)ch * kWCH + j];
                            ch = below;
                            n = kWCH;
                        }
                    }
                    if (lane == 0) {
                        const int slot = atomicAdd(a.team_n, 1);
                        a.team_list[slot] = r; a.team_src[slot] = (uint32_t)o; a.team_key[slot] = n_entries;
                    }
                    left_read = true;
                    break;
                }
            }
            // the bucket of the next pop
            int b;
            if (pend) b = pend_b;
            else {
                b = kWMaxB;
                for (int w = 0; w < kWMaxB / 32; ++w)
                    if (S->mask[w]) { b = w * 32 + __ffs(S->mask[w]) - 1; break; }
            }
            if (b >= kWMaxB || (!pend && S->n_in[b] <= 0)) { ret = kErrStack; break; }   // inconsistent: re-run elsewhere
            const uint32_t binfo = (uint32_t)b << 21;
            const int pend_i = pend ? 1 : 0;
            // early stop (the same for the whole bucket until a hit): the sequential search pops one entry
            if (!c.nonstop && b > best_score + O.s_mm) {
                --n_entries;
                ++pops;
                if (TRACE) {
                    WEnt<P> y = pend ? px : wunpack<P>(chunks[(size_t)S->top_chunk[b] * kWCH + S->top_cnt[b] - 1]);
                    trace = trace_pop<P>(trace, binfo, y, n_entries);
                }
                break;
            }
            if (dbg && lane == 0) S->t_mark = clock64();
            // the wave's entries, in pop order: the pending child (if any), then bucket b from the top
            const int navail = pend_i + S->n_in[b];
            const int Wcap = !TRACE && rec ? 1 : navail < kWE ? navail : kWE;
            // the bucket's chunks down to the wave's last entry; bucket b gets no pushes while it is popped,
            // so the chain walked for earlier waves of b is still valid below its top
            if (b != wch_b) { wch_b = b; wch_n = 0; }
            int walk_ok = 1, k = wch_n;
            if (lane == 0) {
                const int need = Wcap - pend_i;
                if (k == 0 && need > 0) {
                    if (S->top_chunk[b] < 0) walk_ok = 0;
                    else { S->wch[0] = S->top_chunk[b]; k = 1; }
                }
                int cov = k ? S->top_cnt[b] + (k - 1) * kWCH : 0;
                while (walk_ok && cov < need) {
                    if (k >= kWChain) { walk_ok = 0; break; }
                    const int nx = a.chunk_prev[S->wch[k - 1]];
                    if (nx < 0) { walk_ok = 0; break; }
                    S->wch[k++] = nx;
                    cov += kWCH;
                }
            }
            walk_ok = __shfl_sync(FULL, walk_ok, 0);
            wch_n = __shfl_sync(FULL, k, 0);
            if (!walk_ok) { ret = kErrStack; break; }
            __syncwarp();
            {
                // the bucket's entries come in by asynchronous 16-byte copies, all of a lane's started before it
                // waits once
                const int cnt = S->top_cnt[b];
                for (int e = lane; e < Wcap; e += 32) {
                    if (e < pend_i) S->w.ent[e] = wpack<P>(px);
                    else {
                        const int d = e - pend_i;
                        int ci, p;
                        if (d < cnt) { ci = 0; p = cnt - 1 - d; }
                        else { const int d2 = d - cnt; ci = 1 + d2 / kWCH; p = kWCH - 1 - d2 % kWCH; }
                        cp_async16(&S->w.ent[e], chunks + (size_t)S->wch[ci] * kWCH + p);
                    }
                }
                cp_async_wait_all();
            }
            __syncwarp();
            WDBG_LAP(kDbgCycLoad);

            int lp = 0;
            const int E = run_chains<TRACE, ST, P>(ix, O, c, S, &S->w, D, lane, rec, Wcap, b, fetches, log, tags, tl,
                                                   prec_w + (size_t)lane * kWP, lp, dbg ? &S->dv[kDbgSteps] : nullptr);
            __syncwarp();
            if (dbg) {
                const unsigned cp = __reduce_add_sync(FULL, (unsigned)lp);
                WDBG_LAP(kDbgCycChain);
                WDBG_ADD(kDbgWaves, 1);
                WDBG_ADD(kDbgLanes, E);
                WDBG_ADD(kDbgChainPops, cp);
            }

            // ---- replay in sequential order. Without the trace hash the entries are replayed at once from prefix
            // sums, up to the first whose chain is unfinished, fails or crosses the max_entries cut-off, with their
            // hits handled one by one in order. A crossing entry is expanded again in a wave of its own that keeps
            // each pop's data (rec), and it, as every entry in trace mode, is replayed one pop at a time. Lane j
            // holds entries kEPL*j .. kEPL*j + kEPL - 1.
            int consumed = 0;
            bool stop = false, search_end = false, new_pend = false;
            int j_first = 0;
            if (!TRACE && !rec) {
                int pre_k[kEPL], lsum = 0;
                unsigned hits = 0;
#pragma unroll
                for (int k = 0; k < kEPL; ++k) {
                    const int e = kEPL * lane + k;
                    pre_k[k] = e < E ? (int)(int16_t)(S->w.e_a[e] & 0xffffu) : 0;
                    lsum += pre_k[k];
                }
                int incl = lsum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += v;
                }
                const int run0 = n_entries + incl - lsum;   // n_entries before this lane's first entry
                int run = run0, first = 4 * E;      // 4 * entry + its end code, or + 0 where it crosses the cut-off
#pragma unroll
                for (int k = 0; k < kEPL; ++k) {
                    const int e = kEPL * lane + k;
                    if (e < E) {
                        const int endc = (int)(S->w.e_info[e] >> 24);
                        const bool cross = run + (int)(S->w.e_a[e] >> 16) > O.max_entries;
                        if (cross || endc > 1) first = min(first, 4 * e + (cross ? 0 : endc));
                        if (endc == 1) hits |= 1u << k;
                    }
                    run += pre_k[k];
                }
                first = __reduce_min_sync(FULL, first);
                const int first_c = first & 3;
                int cut = first >> 2;               // the hits before it
                for (unsigned hl = __ballot_sync(FULL, hits != 0); hl && !stop; hl &= hl - 1) {
                    const int j = __ffs(hl) - 1;
                    for (unsigned hb = __shfl_sync(FULL, hits, j); hb && !stop; hb &= hb - 1) {
                        const int e = kEPL * j + __ffs(hb) - 1;
                        if (e >= cut) { hl = 1; break; }
                        const int r = on_hit(e);
                        if (r) { cut = e + 1; stop = true; search_end = r == 2; }
                    }
                }
                if (!stop && cut < E) {
                    stop = true;
                    if (first_c == 0) rec = true;                                       // it crosses the cut-off
                    else if (first_c == 2) { new_pend = true; ++cut; }                  // its chain goes on
                    else { ret = kErrScore; search_end = true; ++cut; }                 // BWTGAP_ERR_SCORE at its last pop
                }
                int t_np = 0, t_pre = 0, pk = 0;
                uint32_t t_fs = 0;
                run = run0;
#pragma unroll
                for (int k = 0; k < kEPL; ++k) {
                    const int e = kEPL * lane + k;
                    if (e < cut) {
                        const uint32_t eb = S->w.e_b[e];
                        t_np += (int)((S->w.e_info[e] >> 16) & 0xffu);
                        t_pre += pre_k[k];
                        t_fs += eb >> 16;
                        pk = max(pk, run + (int)(eb & 0xffffu));
                    }
                    run += pre_k[k];
                }
                pops += (uint64_t)__reduce_add_sync(FULL, (unsigned)t_np);
                n_entries += (int)__reduce_add_sync(FULL, (unsigned)t_pre);
                f_alg += __reduce_add_sync(FULL, t_fs);
                const int pkm = (int)__reduce_max_sync(FULL, (unsigned)pk);
                if (pkm > peak) peak = pkm;
                consumed = cut;
                j_first = E;
            } else if (!TRACE) rec = false;
            // Lane t holds pop t of 32 (its data, and in trace mode its entry); the first 32 of the next entry are on
            // their way while one is replayed. (A load per pop, waited for in turn, was most of a trace run's replay:
            // 1299 cycles per pop in all on 36-150 bp reads, 1178 with this.)
            uint32_t next_m = 0;
            uint4 next_v = make_uint4(0, 0, 0, 0);
            auto fetch_pops = [&](int e, int t0, uint32_t &m, uint4 &v) {
                const uint32_t inf = S->w.e_info[e];
                const int ln = (int)(inf & 0xffu), q = (int)((inf >> 8) & 0xffu) + t0 + lane;
                if (t0 + lane >= (int)((inf >> 16) & 0xffu)) return;
                m = D->meta[q][ln];
                if (TRACE) v = prec_w[(size_t)ln * kWP + q];
            };
            if (j_first < E) fetch_pops(j_first, 0, next_m, next_v);
            for (int e = j_first; e < E && !stop; ++e) {
                const uint32_t inf = S->w.e_info[e];
                const int np = (int)((inf >> 16) & 0xffu), endc = (int)(inf >> 24);
                uint32_t m = next_m;
                uint4 v = next_v;
                if (e + 1 < E) fetch_pops(e + 1, 0, next_m, next_v);
                for (int t = 0; t < np; ++t) {
                    if (n_entries > O.max_entries) { search_end = true; stop = true; break; }
                    --n_entries;
                    ++pops;
                    const int tl32 = t & 31;
                    if (t > 0 && tl32 == 0) fetch_pops(e, t, m, v);
                    const uint32_t meta = __shfl_sync(FULL, m, tl32);
                    f_alg += meta >> 5;
                    if (TRACE) {
                        const uint4 y = make_uint4(__shfl_sync(FULL, v.x, tl32), __shfl_sync(FULL, v.y, tl32),
                                                   __shfl_sync(FULL, v.z, tl32), __shfl_sync(FULL, v.w, tl32));
                        trace = trace_pop<P>(trace, binfo, wunpack<P>(y), n_entries);
                    }
                    if (t == np - 1 && endc == 3) { ret = kErrScore; search_end = true; stop = true; break; }
                    if (t == np - 1 && endc == 1) {
                        const int r = on_hit(e);
                        if (r) { consumed = e + 1; stop = true; search_end = r == 2; }
                        break;
                    }
                    n_entries += (int)(meta & 15u) + (int)((meta >> 4) & 1u);
                    if (n_entries > peak) peak = n_entries;
                }
                if (stop) break;
                consumed = e + 1;
                if (endc == 2) { new_pend = true; stop = true; }
            }
            if (dbg) {
                WDBG_LAP(kDbgCycReplay);
                WDBG_ADD(kDbgConsumed, consumed);
                WDBG_ADD(kDbgCont, new_pend ? 1 : 0);
                WDBG_ADD(kDbgHazard, stop && !search_end && !new_pend && !rec ? 1 : 0);
            }
            if (search_end) break;
            if (consumed == 0) continue;      // the wave's first entry crosses the cut-off: expand it again, alone
            // take the consumed entries off bucket b (entry 0 may have been the pending child)
            const int C = consumed - pend_i;
            if (C > 0) {
                // whole chunks emptied: wch[0..j); the new top is wch[j], or the chunk below the last walked one
                int cnt = S->top_cnt[b], left = C, j = 0;
                while (j < wch_n && left >= cnt) { left -= cnt; ++j; cnt = kWCH; }
                const int tc = j < wch_n ? S->wch[j] : (j > 0 ? a.chunk_prev[S->wch[j - 1]] : S->top_chunk[b]);
                if (tc < 0 && left > 0) { ret = kErrStack; break; }
                for (int t = 0; t < j; ++t) A.release(S->wch[t], lane);
                // drop them from the kept chain
                const int keep = wch_n - j;
                const int v = lane < keep ? S->wch[j + lane] : 0;
                __syncwarp();
                if (j > 0) {
                    if (keep > 0) { if (lane < keep) S->wch[lane] = v; wch_n = keep; }
                    else { if (lane == 0 && tc >= 0) S->wch[0] = tc; wch_n = tc >= 0 ? 1 : 0; }
                }
                if (lane == 0) {
                    S->top_chunk[b] = tc;
                    S->top_cnt[b] = (uint16_t)(tc >= 0 ? cnt - left : 0);
                    S->n_in[b] -= C;
                    if (S->n_in[b] == 0) S->mask[b >> 5] &= ~(1u << (b & 31));
                }
                __syncwarp();
            }
            pend = false;
            if (new_pend) {
                pend = true;
                pend_b = b;
                px = wunpack<P>(D->lane_x[S->w.e_info[consumed - 1] & 0xffu]);
            }
            // commit the pushes of the consumed entries (one list per target bucket), in replay order: entry order,
            // then the order the entry's lane staged them. The new chunks of all lists go to newc, list L's from
            // nb_l[L] on; its pushes start at place cnt_l[L] of chunk c_l[L] (none: -1, and then at 0 of its first)
            bool fail = false;
            int c_l[3], cnt_l[3], nb_l[3], t_l[3], nbase = 0;
#pragma unroll
            for (int L = 0; L < 3; ++L) {
                c_l[L] = -1; cnt_l[L] = 0; nb_l[L] = nbase; t_l[L] = 0;
                if (lst_pen[L] < 0 || fail) continue;
                const int X = b + lst_pen[L];
                t_l[L] = share_counts<kWLog>(S->w.e_cnt[L], consumed, lane);
                if (t_l[L] == 0) continue;
                if (X >= n_stacks || X >= kWMaxB) { ret = kErrScore; fail = true; continue; }
                const int c0 = S->top_chunk[X], cnt0 = c0 >= 0 ? S->top_cnt[X] : 0;
                const int need = (cnt0 + t_l[L] + kWCH - 1) / kWCH - (c0 >= 0 ? 1 : 0);
                int32_t *nc = S->newc + nbase;
                if (nbase + need > kWNewC || !A.alloc_n(need, nc, lane)) { ret = kErrStack; fail = true; continue; }
                // chain the new chunks on top of c0
                for (int t = lane; t < need; t += 32) a.chunk_prev[nc[t]] = t == 0 ? c0 : nc[t - 1];
                c_l[L] = c0; cnt_l[L] = cnt0;
                nbase += need;
            }
            if (!fail) {
                auto chunk_at = [&](int L, int g) -> int {     // the chunk of place g from the start of c_l[L]
                    const int c0 = L == 0 ? c_l[0] : L == 1 ? c_l[1] : c_l[2];
                    const int nb0 = L == 0 ? nb_l[0] : L == 1 ? nb_l[1] : nb_l[2];
                    const int ci = g / kWCH - (c0 >= 0 ? 1 : 0);
                    return ci < 0 ? c0 : S->newc[nb0 + ci];
                };
                __syncwarp();
                copy_log<sizeof(P) == 4>(log, tags, S->w.log_n, consumed, lane, [&](int e, int L, int t) -> uint4 * {
                    const int g = (L == 0 ? cnt_l[0] : L == 1 ? cnt_l[1] : cnt_l[2]) + (int)S->w.e_cnt[L][e] + t;
                    return chunks + (size_t)chunk_at(L, g) * kWCH + (g % kWCH);
                });
                __syncwarp();
                if (lane == 0) {
#pragma unroll
                    for (int L = 0; L < 3; ++L) {
                        if (t_l[L] == 0) continue;
                        const int X = b + lst_pen[L], last = cnt_l[L] + t_l[L] - 1;
                        S->top_chunk[X] = chunk_at(L, last);
                        S->top_cnt[X] = (uint16_t)(last % kWCH + 1);
                        S->n_in[X] += t_l[L];
                        S->mask[X >> 5] |= 1u << (X & 31);
                    }
                }
                __syncwarp();
            }
            WDBG_LAP(kDbgCycCommit);
            if (fail) break;
        }
        if (ret == 0) ret = n_aln;
    }
publish:
    if (ret > 0 && !left_read) {
        unsigned long long o = 0;
        if (lane == 0) o = atomicAdd(a.rec_top, (unsigned long long)ret);
        o = __shfl_sync(FULL, o, 0);
        if ((int64_t)(o + ret) > a.rec_cap) ret = kErrAln;
        else {
            for (int j = lane; j < 3 * ret; j += 32) a.out_rec[o * 3 + j] = aln[j];
            if (lane == 0) a.out_off[r] = (int64_t)o;
        }
    }
    if (dbg && lane == 0) {
        S->dv[kDbgReads] = 1;
        S->dv[kDbgPops] = pops;
        const unsigned long long cyc = (unsigned long long)(clock64() - S->t_read);
        S->dv[kDbgCycRead] = cyc;
        for (int q = 0; q < kWDbgN; ++q)
            if (q != kDbgCycReadMax) atomicAdd(a.dbg + q, S->dv[q]);
        atomicMax(a.dbg + kDbgCycReadMax, cyc);
    }
    if (lane == 0 && !left_read) {
        a.out_n[r] = ret;
        a.out_pops[r] = pops;
        a.out_trace[r] = TRACE ? trace : 0;
        a.out_peak[r] = peak;
        a.out_fetch[r] = f_alg;
        a.out_tier[r] = (int8_t)a.tier;
        if (ret == kErrStack && wid >= a.n_big && a.n_big > 0) {
            // to a big warp (its results overwrite these)
            __threadfence();
            const int slot = atomicAdd(a.q_ctl + 1, 1);
            atomicExch(a.ovq + slot, r);
        } else if (ret == kErrStack || ret == kErrAln) a.ovf[atomicAdd(a.ovf_n, 1)] = r;
    }
    __syncwarp();
}

__device__ __forceinline__ uint64_t gtimer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// A big warp's next read (lane 0): a queued one first, else one from the list; -1 when the list is done, every
// small warp has finished and the queue is empty, or after a.q_wait_ns of waiting: the reads still queued
// then go to the next pass. If the wait was for a claimed slot whose read id had not arrived, q_ctl[3] is set
// and the host re-runs every read that was ever queued (a read a big warp finished is searched again with the
// same result). A wait of 0 sets q_ctl[3] whenever it gives up, so that path can be exercised on purpose.
template <class P>
__device__ __noinline__ int big_next(const WArgs<P> &a)
{
    volatile int32_t *qc = a.q_ctl;
    const int n_small = a.n_warps - a.n_big;
    const uint64_t t0 = gtimer_ns();
    for (;;) {
        if (gtimer_ns() - t0 > a.q_wait_ns) {
            if (a.q_wait_ns == 0) atomicExch(a.q_ctl + 3, 1);
            return -1;
        }
        const int h = qc[0], t = qc[1];
        if (h < t) {
            if (atomicCAS(a.q_ctl, h, h + 1) == h) {
                // the producer has taken slot h; its read id follows its atomicAdd at once
                for (;;) {
                    const int r = atomicAdd(a.ovq + h, 0);
                    if (r >= 0) { __threadfence(); return r; }
                    if (gtimer_ns() - t0 > a.q_wait_ns) { atomicExch(a.q_ctl + 3, 1); return -1; }
                    __nanosleep(100);
                }
            }
            continue;
        }
        if (*(volatile int32_t *)a.claim < a.n) {
            const int p = atomicAdd(a.claim, 1);
            if (p < a.n) return a.list[p];
            continue;
        }
        if (qc[2] == n_small) {
            __threadfence();
            if (qc[0] >= qc[1]) return -1;
            continue;
        }
        __nanosleep(2000);
    }
}

template <bool TRACE, int ST, class P>
__global__ void __launch_bounds__(32, 16) warp_kernel(const __grid_constant__ WArgs<P> a)
{
    extern __shared__ __align__(16) unsigned char wsm_raw[];
    WarpSmem *S = (WarpSmem *)wsm_raw;
    const int lane = threadIdx.x & 31;
    const int wid = blockIdx.x;
    if (wid >= a.n_warps) return;
    const bool big = wid < a.n_big;
    for (;;) {
        int r = -1;
        if (lane == 0) {
            if (big) r = big_next(a);
            else {
                const int p = atomicAdd(a.claim, 1);
                r = p < a.n ? a.list[p] : -1;
            }
        }
        r = __shfl_sync(0xffffffffu, r, 0);
        if (r < 0) break;
        warp_read<TRACE, ST, P>(a, r, wid, S, lane);
    }
    if (!big && a.n_big > 0 && lane == 0) {
        __threadfence();
        atomicAdd(a.q_ctl + 2, 1);
    }
}

}  // namespace galn
