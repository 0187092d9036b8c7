// galn_team.cuh -- the heaviest reads: a block of kTW warps per read.
//
// The warp tier (galn_warp.cuh) searches a read on one warp. A few reads need a thousand times the pops of the
// others (a read of 2 M aDNA reads needed 1.5 M pops, one of 200 k reads on a 310 Mbp repeat-rich genome 4 M), and
// such a read alone kept the device waiting when all others were done. Here the wave of entries of the current score
// bucket is spread over the warps of a block, up to kTE entries at once: the lanes of all warps take its entries in
// order from one counter, each warp replays the records of a contiguous share, the shares' prefix sums give n_entries
// before each entry, hits are handled in order by the warps whose share holds them, and every warp commits the
// pushes of its own log at places that follow from the entries' counts. It is the warp tier's wave, replay and commit with
// the same reasons why it is exact.
//
// Storage: a bucket is a stack of positions 0 .. n_in - 1 paged into chunks of kTCH entries; a directory per bucket
// names its chunks, so any position is one lookup away (the warp tier walks a chain of chunks, which is too slow for
// waves of thousands of entries). A read comes from the warp tier as it stood after some number of pops (SaveHdr and
// its entries), and goes on from there; a read that the warp tier could not finish comes without and starts anew.
//
// What bounds it: as in the warp tier the chain of dependent instructions behind each index fetch, and the barriers of a
// wave, behind which all warps wait for its last chain (4.75 of some 10 stalls per issue where searches end at 100 k
// entries; less in longer waves). One block of 16 warps per SM (128 registers a thread, as the warp tier).
// Measured (calls with the team tier off / on, two seeds, one B200): 262 k aDNA reads on 100 Mbp 162 / 58 and 199 / 60 ms,
// 2 M of them 413 / 331 and 313 / 330 (no read there ran long alone; the launch costs what it moves), 10 k high-divergence
// reads 459 / 262 and 486 / 264, 200 k reads on 310 Mbp 223 / 86 and 361 / 94. Entries are taken from one counter, so that
// no warp waits for one whose share had the long chains: with contiguous shares this tier's launch took 278 ms and
// not 245 on the high-divergence reads, 101 and not 25 on the 310 Mbp ones.
#pragma once

#include "galn_warp.cuh"

namespace galn {

constexpr int kTW = 16;             // warps per team
constexpr int kTCH = kTeamChunk;    // entries per chunk

constexpr int kTE = kTW * kWE;      // entries per wave
static_assert(kTE <= 4096, "a tag's entry field");

// The hits of a wave, by entry.
struct TeamSide {
    uint4 hz[kTE];
    uint64_t hk[kTE], hl[kTE];
};

struct TeamSmem {
    uint4 ent[kTE];                 // the wave's entries, in pop order, and their records (as WaveRec's)
    uint32_t e_info[kTE];           // lane in the team (bits 0-8), first pop (9-15), pops (16-23), end code (24-31)
    // In the commit, the place of the entry's first push in its bucket. (A share's entries may be run by the lanes of all
    // warps, so no one log bounds the sum of their pushes, as it does in the warp tier, whose sums fit 16 bits.)
    uint32_t e_cnt[3][kTE];
    uint32_t e_a[kTE], e_b[kTE];
    int32_t next, limit;            // the next entry to be taken; entries from limit on are dropped
    int32_t log_n[kTW];
    int32_t n_in[kWMaxB];
    uint32_t mask[kWMaxB / 32];
    uint32_t T[kWMaxLen + 1], ST[kWMaxLen + 1];
    uint8_t q[kWMaxLen];
    BatchOpt O;
    // per warp, each wave
    int32_t pre[kTW];               // net change of n_entries
    int32_t first[kTW];             // 4 * the first entry that ends the replay + why
    int32_t hits[kTW];
    int32_t np[kTW], net[kTW], peak[kTW], cnt[3][kTW];
    uint32_t fs[kTW];
    // written by one warp for all
    struct {
        int32_t cut, stop, end, ret, n_aln, best_score, best_cnt, max_diff, n_entries, peak, new_pend;
        uint32_t f_alg;
        uint64_t pops;
    } ctl;
    int32_t item;
};

template <class P>
struct TeamArgs {
    IndexViewT<P> ix;
    const uint8_t *query;
    const int64_t *off;
    const int32_t *bidx;
    const int32_t *maxdiff;
    const BatchOpt *bopt;
    const int32_t *list;            // reads
    const uint32_t *src;            // where each read's state is in `save` (16-byte units), or ~0: it starts anew
    int n;
    int32_t *claim;
    const uint4 *save;
    uint4 *arena;                   // per team: arena_chunks * kTCH entries
    int32_t *dir;                   // per team and bucket: arena_chunks chunk numbers
    int32_t *free_ids;              // per team: arena_chunks
    int arena_chunks;
    uint64_t *aln;                  // per team: aln_cap * 3
    int aln_cap;
    uint4 *log;                     // per warp, as the warp tier's
    uint32_t *tags;
    WSide *side;                    // per warp; the first one's wb is the team's
    TeamSide *hits;                 // per team
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
};

// The chains of a wave's Wcap entries S->ent, by all warps: idle lanes take the next entry from S->next, busy lanes pop,
// until no entry is left (or no lane has room). The entries before min(S->next, S->limit) then have their records.
template <int ST, class P>
__device__ __forceinline__ void team_chains(const IndexViewT<P> &ix, const BatchOpt &O, const WCtx &c, TeamSmem *S, WSide *D,
                                            TeamSide *H, int w, int lane, bool rec, int Wcap, int b, uint32_t &fetches,
                                            uint4 *log, uint32_t *tags, const int tl[3])
{
    const unsigned FULL = 0xffffffffu, lt_mask = (1u << lane) - 1u;
    int ce = -1;                                   // this lane's entry
    int nl0 = 0, nl1 = 0, nl2 = 0;                 // its staged pushes per list
    int e_p0 = 0, e_np = 0, e_pre = 0, e_mpre = 0, e_pmax = 0, lp = 0;
    uint32_t e_fs = 0;
    bool more = true;                              // entries may be left
    WEnt<P> x;
    x.k = 0; x.l = 0; x.i = 0; x.is_diff = 0; x.n_mm = x.n_gapo = x.n_gape = x.n_ins = 0; x.state = 0;
    WWalk<P> wk;
    wk.k = 0; wk.l = 0; wk.i = 0; wk.f = 0; wk.on = false;
    if (lane == 0) S->log_n[w] = 0;
    __syncwarp();
    for (;;) {
        // a step adds at most 9 pushes a lane; entries are taken while the log holds kWGrabPops such steps
        const int used = *(volatile int32_t *)&S->log_n[w];
        const int limit = __shfl_sync(FULL, *(volatile int32_t *)&S->limit, 0);
        if (ce >= limit) { ce = -1; wk.on = false; }
        const bool want = more && ce < 0 && lp + kWGrabPops <= kWP && used + 9 * 32 * kWGrabPops <= kWLog;
        const unsigned wb = __ballot_sync(FULL, want);
        if (wb) {
            int e0 = 0;
            if (lane == 0) e0 = atomicAdd(&S->next, __popc(wb));
            e0 = __shfl_sync(FULL, e0, 0);
            const int e = e0 + __popc(wb & lt_mask);
            more = e0 + __popc(wb) < limit;
            if (want && e < limit) {
                ce = e;
                x = wunpack<P>(S->ent[e]);
                e_p0 = lp; e_np = 0; e_pre = 0; e_mpre = 0; e_pmax = 0; e_fs = 0;
                nl0 = nl1 = nl2 = 0;
            }
        }
        if (!__any_sync(FULL, ce >= 0)) break;
        if (ce >= 0) {
            uint32_t mt = 0;
            const int endc = lane_step<false, ST, P, false>(ix, O, c, S, D, H, lane, ce, rec, used + 2 * 9 * 32 > kWLog, x, wk, b,
                                                     fetches, log, tags, &S->log_n[w], tl, nullptr, lp, nl0, nl1, nl2, mt);
            if (endc != -2) {                          // else an exact walk goes on
                ++e_np;
                if (e_pre > e_mpre) e_mpre = e_pre;     // n_entries before this pop, relative to the chain start
                e_pre += (int)(mt & 15u) + (int)((mt >> 4) & 1u) - 1;
                if (e_pre > e_pmax) e_pmax = e_pre;
                e_fs += mt >> 5;
                if (endc >= 0) {
                    S->e_info[ce] = (uint32_t)(w * 32 + lane) | (uint32_t)e_p0 << 9 | (uint32_t)e_np << 16 | (uint32_t)endc << 24;
                    S->e_cnt[0][ce] = (uint32_t)nl0;
                    S->e_cnt[1][ce] = (uint32_t)nl1;
                    S->e_cnt[2][ce] = (uint32_t)nl2;
                    S->e_a[ce] = ((uint32_t)e_pre & 0xffffu) | (uint32_t)e_mpre << 16;
                    S->e_b[ce] = (uint32_t)e_pmax | e_fs << 16;
                    if (endc > 1) atomicMin(&S->limit, ce + 1);   // no room, or an error: entries past it are dropped
                    ce = -1;
                }
            }
        }
        __syncwarp();
    }
}

template <int ST, class P>
__device__ void team_read(const TeamArgs<P> &a, int r, uint32_t src, int team, TeamSmem *S)
{
    const unsigned FULL = 0xffffffffu;
    constexpr int kThreads = kTW * 32, kNone = 0x7fffffff;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int64_t q0 = a.off[r];
    const int len = (int)(a.off[r + 1] - q0);
    const int max_diff0 = a.maxdiff[r];
    const IndexViewT<P> &ix = a.ix;
    WSide *side = a.side + (size_t)team * kTW, *D = side + w;
    uint64_t *wb = side->wb, *aln = a.aln + (size_t)team * a.aln_cap * 3;
    uint4 *arena = a.arena + (size_t)team * a.arena_chunks * kTCH;
    int32_t *dir = a.dir + (size_t)team * kWMaxB * a.arena_chunks;
    int32_t *free_ids = a.free_ids + (size_t)team * a.arena_chunks;
    uint4 *log = a.log + ((size_t)team * kTW + w) * kWLog;
    uint32_t *tags = a.tags + ((size_t)team * kTW + w) * kWLog;
    TeamSide *H = a.hits + team;
    if (tid == 0) S->O = a.bopt[a.bidx[r]];
    for (int t = tid; t < len; t += kThreads) S->q[t] = a.query[q0 + t];
    static_assert(kWMaxB <= kThreads && kWMaxB % 32 == 0, "one thread per bucket");
    if (tid < kWMaxB) S->n_in[tid] = 0;
    if (tid < kWMaxB / 32) S->mask[tid] = 0;
    __syncthreads();
    const BatchOpt &O = S->O;
    const int n_stacks = O.n_stacks;
    WCtx c;
    c.len = len; c.max_diff0 = max_diff0; c.max_diff = max_diff0; c.use_seed = len > O.seed_len;
    c.seed_len_r = len > O.seed_len ? O.seed_len : 0x7fffffff;
    c.gape = (O.mode & kModeGape) != 0; c.nonstop = (O.mode & kModeNonstop) != 0;
    int tl[3];
    tl[0] = 0;
    tl[1] = O.s_gapo == O.s_mm ? 0 : 1;
    tl[2] = O.s_gape == O.s_mm ? 0 : (O.s_gape == O.s_gapo ? tl[1] : 2);
    const int lst_pen[3] = {O.s_mm, tl[1] == 1 ? O.s_gapo : -1, tl[2] == 2 ? O.s_gape : -1};
    // the read's state, the same in every thread
    int best_score = (max_diff0 + 1) * O.s_mm + (O.max_gapo + 1) * O.s_gapo + (O.max_gape + 1) * O.s_gape;
    int best_cnt = 0, n_aln = 0, ret = 0, n_entries = 0, peak = 0;
    int bump = 0, g_top = 0;           // the chunk allocator: fresh chunks from bump, returned ones in free_ids
    uint64_t pops = 0;
    uint32_t f_alg = 0, fetches = 0;
    bool pend = false, rec = false;
    int pend_b = 0;
    uint4 px = make_uint4(0, 0, 0, 0);

    if (src != ~0u) {
        const SaveHdr *h = reinterpret_cast<const SaveHdr *>(a.save + src);
        n_entries = h->n_entries; peak = h->peak; best_score = h->best_score; best_cnt = h->best_cnt;
        n_aln = h->n_aln; c.max_diff = h->max_diff; pend = h->pend != 0; pend_b = h->pend_b; pops = h->pops;
        f_alg = h->f_alg; px = h->px;
        for (int t = tid; t <= len; t += kThreads) {
            wb[t] = h->wb[t];
            S->ST[t] = h->ST[t];
            if (t) S->T[t] = width_word(h->wb[t - 1], h->wb[t]);
        }
        const uint64_t *rec_in = reinterpret_cast<const uint64_t *>(a.save + src + sizeof(SaveHdr) / 16);
        for (int t = tid; t < 3 * n_aln; t += kThreads) aln[t] = rec_in[t];
        const uint4 *ent = a.save + src + save_entries_at(n_aln);
        if (tid < kWMaxB) {
            const int n = max(0, h->n_in[tid]);
            S->n_in[tid] = n;
            const unsigned m = __ballot_sync(FULL, n > 0);
            if (lane == 0) S->mask[w] = m;
        }
        __syncthreads();
        for (int b = 0; b < kWMaxB; ++b) {
            const int n = S->n_in[b];
            if (n <= 0) continue;
            const int nc = (n + kTCH - 1) / kTCH;
            if (bump + nc > a.arena_chunks) { ret = kErrStack; break; }
            for (int t = tid; t < nc; t += kThreads) dir[(size_t)b * a.arena_chunks + t] = bump + t;
            for (int t = tid; t < n; t += kThreads) arena[(size_t)bump * kTCH + t] = ent[t];
            ent += n;
            bump += nc;
        }
    } else {
        if (tid < 2) width_walk<ST, P>(ix, len, c.use_seed ? O.seed_len : 0, tid, S->q, wb, S->T, S->ST, fetches);
        if (w == 0) {
            const uint32_t f = __shfl_sync(FULL, fetches, 0) + __shfl_sync(FULL, fetches, 1);
            if (lane == 0) S->ctl.f_alg = f;
        }
        __syncthreads();
        f_alg = S->ctl.f_alg;
        int n_amb = 0;
        for (int j = 0; j < len; ++j) n_amb += S->q[j] > 3;
        if (n_stacks <= 0) ret = kErrScore;
        else if (n_amb <= c.max_diff) {
            px = pack_entry((P)0, ix.seq_len, len, 0, 0, 0, 0, kStM, 0);
            pend = true;
            n_entries = peak = 1;
        }
    }
    __syncthreads();

    while (ret == 0) {
        if (n_entries == 0 || n_entries > O.max_entries) break;
        int b = kWMaxB;
        if (pend) b = pend_b;
        else
            for (int t = 0; t < kWMaxB / 32; ++t)
                if (S->mask[t]) { b = t * 32 + __ffs(S->mask[t]) - 1; break; }
        if (b >= kWMaxB || (!pend && S->n_in[b] <= 0)) { ret = kErrStack; break; }   // inconsistent: re-run elsewhere
        if (!c.nonstop && b > best_score + O.s_mm) { --n_entries; ++pops; break; }
        // ---- the wave, and this warp's share of its records: entries s0 .. s0 + kWE - 1 ----
        const int pend_i = pend ? 1 : 0, nb = S->n_in[b];
        const bool rec_wave = rec;
        const int Wcap = rec ? 1 : min(pend_i + nb, kTE);
        const int s0 = w * kWE;
        if (tid == 0) { S->next = 0; S->limit = Wcap; }
        for (int e = tid; e < Wcap; e += kThreads) {
            if (e < pend_i) S->ent[e] = px;
            else {
                const int pos = nb - 1 - (e - pend_i);
                cp_async16(&S->ent[e], arena + (size_t)dir[(size_t)b * a.arena_chunks + pos / kTCH] * kTCH + pos % kTCH);
            }
        }
        cp_async_wait_all();
        __syncthreads();                                                        // the wave's entries
        team_chains<ST, P>(ix, O, c, S, D, H, w, lane, rec, Wcap, b, fetches, log, tags, tl);
        __syncthreads();                                                        // its records
        const int E_all = min(min(S->next, S->limit), Wcap), E = max(0, min(E_all - s0, kWE));
        uint32_t *e_info = S->e_info + s0, *e_a = S->e_a + s0, *e_b = S->e_b + s0;
        int pre_k[kEPL], lsum = 0;
#pragma unroll
        for (int k = 0; k < kEPL; ++k) {
            const int e = kEPL * lane + k;
            pre_k[k] = e < E ? (int)(int16_t)(e_a[e] & 0xffffu) : 0;
            lsum += pre_k[k];
        }
        int incl = lsum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) S->pre[w] = incl;
        __syncthreads();                                                        // the shares' sums
        int cut = 0, run0 = 0;
        bool stop = false, search_end = false, new_pend = false;
        if (rec_wave) {
            // one entry, pop by pop: it crosses the max_entries cut-off
            rec = false;
            if (w == 0) {
                const uint32_t inf = e_info[0];
                const int ln = (int)(inf & 31u), np = (int)((inf >> 16) & 0xffu), endc = (int)(inf >> 24);
                const WSide *DL = side + ((inf >> 5) & 15u);
                for (int t = 0; t < np; ++t) {
                    if (n_entries > O.max_entries) { search_end = true; break; }
                    --n_entries;
                    ++pops;
                    const uint32_t meta = DL->meta[t][ln];
                    f_alg += meta >> 5;
                    if (t == np - 1 && endc == 3) { ret = kErrScore; search_end = true; break; }
                    if (t == np - 1 && endc == 1) {
                        search_end = take_hit<P>(ix, O, c, S->T, wb, H->hz[0], H->hk[0], H->hl[0], aln, a.aln_cap, n_aln,
                                                 best_score, best_cnt, ret, lane) == 2;
                        break;
                    }
                    n_entries += (int)(meta & 15u) + (int)((meta >> 4) & 1u);
                    if (n_entries > peak) peak = n_entries;
                }
                if (lane == 0) {
                    S->ctl.end = search_end; S->ctl.ret = ret; S->ctl.n_aln = n_aln; S->ctl.best_score = best_score;
                    S->ctl.best_cnt = best_cnt; S->ctl.max_diff = c.max_diff; S->ctl.n_entries = n_entries;
                    S->ctl.peak = peak; S->ctl.f_alg = f_alg; S->ctl.pops = pops; S->ctl.new_pend = endc == 2;
                }
            }
            __syncthreads();
            search_end = S->ctl.end != 0; ret = S->ctl.ret; n_aln = S->ctl.n_aln; best_score = S->ctl.best_score;
            best_cnt = S->ctl.best_cnt; c.max_diff = S->ctl.max_diff; n_entries = S->ctl.n_entries; peak = S->ctl.peak;
            f_alg = S->ctl.f_alg; pops = S->ctl.pops; new_pend = S->ctl.new_pend != 0;
            if (search_end) break;
            cut = 1;
        } else {
            int base = n_entries;
            for (int v = 0; v < w; ++v) base += S->pre[v];
            run0 = base + incl - lsum;               // n_entries before this lane's first entry
            // 4 * the share's first entry that ends the replay + why: 0 it crosses the max_entries cut-off, 2 its chain
            // goes on, 3 BWTGAP_ERR_SCORE
            int run = run0, first = kNone;
            unsigned hits = 0;
#pragma unroll
            for (int k = 0; k < kEPL; ++k) {
                const int e = kEPL * lane + k;
                if (e < E) {
                    const int endc = (int)(e_info[e] >> 24);
                    const bool cross = run + (int)(e_a[e] >> 16) > O.max_entries;
                    if (cross || endc > 1) first = min(first, 4 * e + (cross ? 0 : endc));
                    if (endc == 1) hits |= 1u << k;
                }
                run += pre_k[k];
            }
            first = __reduce_min_sync(FULL, first);
            const unsigned hit_lanes = __ballot_sync(FULL, hits != 0);
            if (lane == 0) { S->first[w] = first == kNone ? kNone : first + 4 * s0; S->hits[w] = hit_lanes != 0; }
            __syncthreads();                                                    // where the replay ends
            int key = 4 * E_all + 1, any = 0;
            for (int v = 0; v < kTW; ++v) { key = min(key, S->first[v]); any |= S->hits[v]; }
            cut = key >> 2;
            if (any) {
                // hits before the cut, in order: share by share, each by its own warp
                for (int v = 0; v < kTW && v * kWE < cut && !stop; ++v) {
                    if (!S->hits[v]) continue;
                    if (w == v) {
                        for (unsigned hl = hit_lanes; hl && !stop; hl &= hl - 1) {
                            const int j = __ffs(hl) - 1;
                            for (unsigned hb = __shfl_sync(FULL, hits, j); hb && !stop; hb &= hb - 1) {
                                const int e = kEPL * j + __ffs(hb) - 1;
                                if (s0 + e >= cut) { hl = 1; break; }
                                const int t = take_hit<P>(ix, O, c, S->T, wb, H->hz[s0 + e], H->hk[s0 + e], H->hl[s0 + e], aln, a.aln_cap,
                                                          n_aln, best_score, best_cnt, ret, lane);
                                if (t) { cut = s0 + e + 1; stop = true; search_end = t == 2; }
                            }
                        }
                        if (lane == 0) {
                            S->ctl.cut = cut; S->ctl.stop = stop; S->ctl.end = search_end; S->ctl.ret = ret;
                            S->ctl.n_aln = n_aln; S->ctl.best_score = best_score; S->ctl.best_cnt = best_cnt;
                            S->ctl.max_diff = c.max_diff;
                        }
                    }
                    __syncthreads();
                    cut = S->ctl.cut; stop = S->ctl.stop != 0; search_end = S->ctl.end != 0; ret = S->ctl.ret;
                    n_aln = S->ctl.n_aln; best_score = S->ctl.best_score; best_cnt = S->ctl.best_cnt;
                    c.max_diff = S->ctl.max_diff;
                    __syncthreads();
                }
            }
            if (!stop && cut < E_all) {
                const int why = key & 3;
                if (why == 0) rec = true;
                else if (why == 2) { new_pend = true; ++cut; }
                else if (why == 3) { ret = kErrScore; search_end = true; ++cut; }
            }
        }
        // ---- sums of the replayed entries, and their pushes per list ----
        const int lc = max(0, min(cut - s0, E));
        {
            int t_np = 0, t_pre = 0, pk = 0, run = run0;
            uint32_t t_fs = 0;
            unsigned c0 = 0, c1 = 0, c2 = 0;
#pragma unroll
            for (int k = 0; k < kEPL; ++k) {
                const int e = kEPL * lane + k;
                if (e < lc) {
                    const uint32_t eb = e_b[e];
                    t_np += (int)((e_info[e] >> 16) & 0xffu);
                    t_pre += pre_k[k];
                    t_fs += eb >> 16;
                    pk = max(pk, run + (int)(eb & 0xffffu));
                    c0 += S->e_cnt[0][s0 + e]; c1 += S->e_cnt[1][s0 + e]; c2 += S->e_cnt[2][s0 + e];
                }
                run += pre_k[k];
            }
            t_np = (int)__reduce_add_sync(FULL, (unsigned)t_np);
            t_pre = (int)__reduce_add_sync(FULL, (unsigned)t_pre);
            t_fs = __reduce_add_sync(FULL, t_fs);
            pk = (int)__reduce_max_sync(FULL, (unsigned)pk);
            c0 = __reduce_add_sync(FULL, c0); c1 = __reduce_add_sync(FULL, c1); c2 = __reduce_add_sync(FULL, c2);
            if (lane == 0) {
                S->np[w] = t_np; S->net[w] = t_pre; S->fs[w] = t_fs; S->peak[w] = pk;
                S->cnt[0][w] = (int)c0; S->cnt[1][w] = (int)c1; S->cnt[2][w] = (int)c2;
            }
        }
        __syncthreads();                                                        // sums and counts
        int tot_l[3] = {0, 0, 0}, base_l[3] = {0, 0, 0};
        for (int v = 0; v < kTW; ++v) {
            if (!rec_wave) {
                pops += (uint64_t)S->np[v];
                n_entries += S->net[v];
                f_alg += S->fs[v];
                peak = max(peak, S->peak[v]);
            }
#pragma unroll
            for (int L = 0; L < 3; ++L) {
                const int t = S->cnt[L][v];
                if (v < w) base_l[L] += t;
                tot_l[L] += t;
            }
        }
        if (search_end) break;
        if (cut == 0) { __syncthreads(); continue; }   // the first entry crosses the cut-off: expand it again, alone
        pend = false;
        if (new_pend) {
            const uint32_t inf = S->e_info[cut - 1];
            pend = true;
            pend_b = b;
            px = __ldcg(&side[(inf >> 5) & 15u].lane_x[inf & 31u]);
        }
        // ---- chunks for the pushes: returned ones first, then fresh ones ----
        int at_l[3];
        bool fail = false;
#pragma unroll
        for (int L = 0; L < 3; ++L) {
            at_l[L] = 0;
            if (lst_pen[L] < 0 || tot_l[L] == 0 || fail) continue;
            const int X = b + lst_pen[L];
            if (X >= n_stacks || X >= kWMaxB) { ret = kErrScore; fail = true; continue; }
            const int nx = S->n_in[X], c_lo = (nx + kTCH - 1) / kTCH, need = (nx + tot_l[L] + kTCH - 1) / kTCH - c_lo;
            const int from_g = min(need, g_top);
            if (bump + need - from_g > a.arena_chunks) { ret = kErrStack; fail = true; continue; }
            for (int t = tid; t < need; t += kThreads)
                dir[(size_t)X * a.arena_chunks + c_lo + t] = t < from_g ? free_ids[g_top - 1 - t] : bump + t - from_g;
            g_top -= from_g;
            bump += need - from_g;
            at_l[L] = nx;
        }
        if (fail) break;
#pragma unroll
        for (int L = 0; L < 3; ++L) {
            share_counts<0x7fffffffu>(S->e_cnt[L] + s0, lc, lane, at_l[L] + base_l[L]);
        }
        __syncthreads();                                                        // the directories and the places
        // ---- commit: every warp the pushes of its own log, at their places in replay order ----
        copy_log<false>(log, tags, S->log_n[w], cut, lane, [&](int e, int L, int k) -> uint4 * {
            const int g = (int)S->e_cnt[L][e] + k;
            const int X = b + (L == 0 ? lst_pen[0] : L == 1 ? lst_pen[1] : lst_pen[2]);
            return arena + (size_t)dir[(size_t)X * a.arena_chunks + g / kTCH] * kTCH + g % kTCH;
        });
        // ---- the consumed entries leave bucket b, with the chunks they emptied ----
        const int nb2 = nb - (cut - pend_i);
        const int keep = (nb2 + kTCH - 1) / kTCH, gone = (nb + kTCH - 1) / kTCH - keep;
        for (int t = tid; t < gone; t += kThreads) free_ids[g_top + t] = dir[(size_t)b * a.arena_chunks + keep + t];
        g_top += gone;
        if (tid == 0) {
            S->n_in[b] = nb2;
            if (nb2 == 0) S->mask[b >> 5] &= ~(1u << (b & 31));
            for (int L = 0; L < 3; ++L)
                if (tot_l[L] > 0 && lst_pen[L] >= 0) {
                    const int X = b + lst_pen[L];
                    S->n_in[X] += tot_l[L];
                    S->mask[X >> 5] |= 1u << (X & 31);
                }
        }
        __syncthreads();                                                        // the wave is done
    }
    if (ret == 0) ret = n_aln;
    __syncthreads();
    if (w == 0) {
        if (ret > 0) {
            unsigned long long o = 0;
            if (lane == 0) o = atomicAdd(a.rec_top, (unsigned long long)ret);
            o = __shfl_sync(FULL, o, 0);
            if ((int64_t)(o + ret) > a.rec_cap) ret = kErrAln;
            else {
                for (int j = lane; j < 3 * ret; j += 32) a.out_rec[o * 3 + j] = aln[j];
                if (lane == 0) a.out_off[r] = (int64_t)o;
            }
        }
        if (lane == 0) {
            a.out_n[r] = ret;
            a.out_pops[r] = pops;
            a.out_trace[r] = 0;
            a.out_peak[r] = peak;
            a.out_fetch[r] = f_alg;
            a.out_tier[r] = (int8_t)a.tier;
            if (ret == kErrStack || ret == kErrAln) a.ovf[atomicAdd(a.ovf_n, 1)] = r;
        }
    }
}

template <int ST, class P>
__global__ void __launch_bounds__(kTW * 32, 1) team_kernel(const __grid_constant__ TeamArgs<P> a)
{
    extern __shared__ __align__(16) unsigned char tsm_raw[];
    TeamSmem *S = reinterpret_cast<TeamSmem *>(tsm_raw);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) S->item = atomicAdd(a.claim, 1);
        __syncthreads();
        const int p = S->item;
        if (p >= a.n) break;
        team_read<ST, P>(a, a.list[p], a.src[p], blockIdx.x, S);
    }
}

}  // namespace galn
