// Hamming scoring and the selection plan.
//
// score_hist_kernel streams the key-hash pages once: one 16-byte word per token per kv-head carries
// the four 32-bit codes of the kv-head's query heads, so a lane scores 4 heads per load,
// score = popcount(~(q_code ^ k_code)) in 0..32. Each CTA builds the 4 x 33 histogram of the scores
// of the candidate tokens of its chunk, adds it to the totals of its (sequence, kv-head) with atomic
// adds, and publishes per score the number of its tokens AT OR ABOVE that score, bin-major
// ([bin][chunk]); it also writes the scores of its tokens, one byte per token and query head
// (score + 1, 0 = not a candidate), in one plane per head.
//
// The CTA that finishes last for a (sequence, kv-head) - an arrival counter, no waiting - derives
// the plan of that unit (select_plan): the threshold T of each head and how many tokens tied at T still
// fit from the totals (pick_threshold: both selection rules of the reference), then how many selected /
// tied tokens precede each chunk from two published counts per chunk and head.
//
// select_attend_kernel (select_attend.cuh) then classifies each chunk's score bytes against T, compacts
// the selected tokens and attends them - no sort, no atomics in the output path.
//
// score_select_cluster_kernel does scoring and selection in one kernel for short sequences.
//
// Together they replace the +-1 dot product of USA.forward and the sort/scatter (or threshold) of
// compute_mask_multi (hashattention/hashattention_llama.py:171-187, 423-443).
// A stable descending sort picks, among tokens tied at the threshold, the lowest indices;
// the tie fill reproduces exactly that set.
//
// Tiling of score_hist_kernel: a CTA of 256 threads owns a chunk of 4 * ROUNDS pages of one (sequence,
// kv-head) and walks it in rounds of 1024 tokens; in a round warp w owns tokens [128 w, 128 w + 128)
// (half a page), four per lane. The words of two rounds are on their way at a time; the copies of a round are issued
// together without branches between them (indices are clamped into range instead of guarded). Everything that does not
// depend on the preceding kernel - the sequence length, page ids and the first rounds' hash words - is fetched before
// the grid-dependency wait.
//
// What bounds it: a CTA spends about 1.5 us on its first words and 1.5 us on publishing its counts, so the stream of the
// others has to cover that. With the words in flight in shared memory (cp.async) six CTAs fit on an SM, where the
// registers to hold them allowed four: scoring and plan of 32 sequences of 16384 - 65536 tokens x 8 kv-heads take 47.8 us
// instead of 54.7 (5 CTAs 50.5), of 4 x 131072 17.7 instead of 18.6, of 32 x 20000 21.3 instead of 24.3; the hash words
// alone would take 28.2, 10.2 and 12.5. (Registers capped as for 8 CTAs, of which the shared memory holds six all the same:
// 47.2 and, with spills, 21.4.) Chunks of one round keep them in registers: there the trip through shared memory costs 0.3
// us (3 x 9001 - 15000: 5.5 us, else 5.2) and the grid is small.
//
// Layout of a score plane: inside every block of 128 tokens the byte of token 32 it + lane (the it-th
// token of a lane in the warp's round) sits at offset 4 lane + it, so that a lane stores its four
// tokens of one head as one 32-bit word and a warp 128 contiguous bytes per head.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace ha {

namespace cg = cooperative_groups;

constexpr int kShMinCtas = 6;                         // CTAs of score_hist_kernel<2 or 4> per SM (40 registers per thread, 37 KB)
constexpr int kRoundPages = 4;                        // pages per round
constexpr int kRoundTokens = kRoundPages * kPage;     // 1024
constexpr int kLaneTokens = kRoundTokens / kSelThreads;  // 4 tokens per lane and round

struct SelectParams {
    const uint32_t* q_codes;   // [B][Hq]
    const uint4* hash_pages;   // [num_pages][Hkv][256] x 16 B
    const int32_t* page_table;
    const int32_t* seq_lens;
    const int32_t* budget_lens;  // [B] or null: the length the heavy budget is a fraction of, if not seq_lens
    uint32_t* hist;            // workspace: [B][Hkv][4*33][nchunks] per chunk: tokens at or above each score
    uint32_t* arrive;          // workspace: [B][Hkv][kArriveStride] chunks of the unit that have published, the unit's
                               // histogram totals (all 0 between calls)
    int32_t* ready;            // workspace: [B][Hkv][kReadyStride] ready words (0 between calls), or null: nobody waits for them
    int32_t* sel_idx;          // [B][Hq][sel_stride] token indices
    int32_t* sel_rows;         // workspace: [B][Hq][sel_stride] page * 256 + slot of the same tokens
    int32_t* sel_cnt;          // [B][Hq]
    int32_t* plan;             // workspace: [B][Hkv][8 + 8 * nchunks]: T[4], need[4], then per chunk base[4], eqb[4]
    uint8_t* scores;           // workspace: [B][Hq][nchunks * chunk tokens]: score + 1, 0 = not a candidate (layout above)
    uint8_t* scores_dbg;       // [B][Hq][max_pages*256] or null
    int32_t* status;
    int B, Hkv, max_pages, num_pages, sel_stride, nchunks;
    int kvh0;                  // first kv-head of this launch (a launch may cover a slice of the kv-heads)
    int init_budget, recent_budget;
    double heavy_budget;
    int eval_mode, depth;      // HA_EVAL_*; usa_retrieve_depth (HA_EVAL_DEPTH only)
};

// One round of one warp: 128 consecutive tokens of one page, token it*32 + lane for it = 0..3.
// A round whose 128 tokens are all selection candidates (and do not include the newest token,
// whose hash word the encoder kernel may still be writing) is "interior": no per-token masks.
struct RoundWords {
    uint4 w[kLaneTokens];
    int page;          // page id of the warp's half page (clamped into the pool)
    uint32_t cand;     // bit it: token is a selection candidate
    uint32_t valid;    // bit it: token exists
    bool interior;     // warp-uniform: all 128 tokens are candidates, none is the newest token
    bool bad_page;

    // first token of this warp in round `rd` of chunk starting at `chunk_start`
    static __device__ __forceinline__ int first_token(int chunk_start, int rd, int warp) {
        return chunk_start + rd * kRoundTokens + warp * (kLaneTokens * 32);
    }

    // page id (unchecked) of the page that holds token t0
    static __device__ __forceinline__ int page_of(const SelectParams& p, int b, int t0) {
        return __ldg(p.page_table + (size_t)b * p.max_pages + min(t0 / kPage, p.max_pages - 1));
    }

    __device__ __forceinline__ void load(const SelectParams& p, int b, int kvh, int t0, int lane, const SeqRange& r) {
        load(p, kvh, t0, lane, r, page_of(p, b, t0));
    }

    // pg: what page_of() returned for t0 (fetched ahead of time, so that the hash words are the only loads on the way)
    __device__ __forceinline__ void load(const SelectParams& p, int kvh, int t0, int lane, const SeqRange& r, int pg) {
        const bool page_ok = pg >= 0 && pg < p.num_pages;
        page = page_ok ? pg : 0;
        const uint4* src = p.hash_pages + ((size_t)page * p.Hkv + kvh) * kPage;
        interior = page_ok && t0 >= r.lo && t0 + kLaneTokens * 32 <= r.hi &&
                   (unsigned)(r.S - 1 - t0) >= (unsigned)(kLaneTokens * 32);
        bad_page = false;
        if (interior) {
            const uint4* s0 = src + t0 % kPage + lane;
#pragma unroll
            for (int it = 0; it < kLaneTokens; ++it) w[it] = __ldg(s0 + it * 32);
            cand = valid = (1u << kLaneTokens) - 1u;
            return;
        }
        valid = 0;
        cand = 0;
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it) {
            const int t = t0 + it * 32 + lane;
            const bool ok = t < r.S;
            bad_page |= ok && !page_ok;
            w[it] = __ldg(src + (ok ? t : r.S - 1) % kPage);  // clamp: always an in-range slot
            if (ok && page_ok) {
                valid |= 1u << it;
                if (t >= r.lo && t < r.hi) cand |= 1u << it;
            }
        }
    }

    // Re-reads the newest token's word, which the encoder kernel may have written after load().
    __device__ __forceinline__ void refresh_newest(const SelectParams& p, int kvh, int t0, int lane, const SeqRange& r) {
        if (interior) return;
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it)
            if (t0 + it * 32 + lane == r.S - 1 && ((valid >> it) & 1u))
                w[it] = __ldcg(p.hash_pages + ((size_t)page * p.Hkv + kvh) * kPage + (r.S - 1) % kPage);
    }
};

// A round whose words are on their way to shared memory instead of registers: a lane copies its four words (cp.async) and
// reads back what it has copied itself, so nothing but its own copies has to be waited for. Tokens as in RoundWords.
struct StagedRound {
    int page, t0;
    bool page_ok;

    __device__ __forceinline__ void copy(const SelectParams& p, int kvh, int first, int lane, const SeqRange& r, int pg, uint4* slot) {
        t0 = first;
        page_ok = pg >= 0 && pg < p.num_pages;
        page = page_ok ? pg : 0;
        const uint4* src = p.hash_pages + ((size_t)page * p.Hkv + kvh) * kPage;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(slot + lane);
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it) {
            const uint4* w = src + min(t0 + it * 32 + lane, r.S - 1) % kPage;  // clamp: always an in-range slot
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + it * 32 * 16), "l"(w) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // every token is a candidate, and none is the newest one, whose word the encoder may have written after the copy
    __device__ __forceinline__ bool interior(const SeqRange& r) const {
        return page_ok && t0 >= r.lo && t0 + kLaneTokens * 32 <= r.hi && (unsigned)(r.S - 1 - t0) >= (unsigned)(kLaneTokens * 32);
    }
};

// qn = ~q_code per head, so that popcount(qn ^ k) = popcount(~(q ^ k)) = number of agreeing bits
__device__ __forceinline__ uint4 load_qn(const SelectParams& p, int b, int kvh) {
    const uint4 qc = __ldcg(reinterpret_cast<const uint4*>(p.q_codes + ((size_t)b * p.Hkv + kvh) * kGroup));
    return make_uint4(~qc.x, ~qc.y, ~qc.z, ~qc.w);
}

// bit 7 of byte g -> bit g
__device__ __forceinline__ uint32_t flags_to_nibble(uint32_t f) { return (((f >> 7) * 0x01020408u) >> 24) & 0xFu; }

// What is kept of one head's candidates, worked out from the totals per score bin by one full
// warp: lane l passes n = total of bin 32 - l and cum = the inclusive prefix of n over the lanes
// (candidates scoring >= 32 - l); tot0 = total of bin 0; hb = min(budget, candidates).
//   T      tokens scoring above T are kept, of those scoring T the first `need` by token index;
//          T = 33 keeps nothing
//   count  tokens kept in all, cut to sel_stride (`overflow` says whether it had to be)
// HA_EVAL_SIMPLE: the hb best (hashattention/hashattention_llama.py:436-438). HA_EVAL_DEPTH: every
// candidate scoring at least max(best - depth, score of the hb-th best) (:439-443; one score step
// is a span step of 2).
struct Threshold {
    int T, need, count;
};

__device__ __forceinline__ Threshold pick_threshold(const SelectParams& p, int n, int cum, int tot0, int hb,
                                                    bool& overflow) {
    Threshold t;
    t.T = kBins; t.need = 0; t.count = 0;
    overflow = false;
    int hbe = hb;
    if (p.eval_mode == HA_EVAL_SIMPLE && hbe > p.sel_stride) {
        overflow = true;
        hbe = p.sel_stride;
    }
    if (hbe <= 0) return t;
    // the score of the hbe-th best candidate and the number of candidates above it
    const uint32_t reached = __ballot_sync(0xffffffffu, cum >= hbe);
    const int l = reached != 0 ? __ffs(reached) - 1 : 31;  // first lane whose cumulative count reaches the budget
    const int cum31 = __shfl_sync(0xffffffffu, cum, 31);
    const int above_l = __shfl_sync(0xffffffffu, cum - n, l);
    const int T_num = reached != 0 ? 32 - l : 0;  // bins 32..1 hold fewer than the budget: the threshold is 0
    const int above = reached != 0 ? above_l : cum31;
    if (p.eval_mode == HA_EVAL_SIMPLE) {
        t.T = T_num;
        t.need = hbe - above;
        t.count = hbe;
        return t;
    }
    const uint32_t nonzero = __ballot_sync(0xffffffffu, n > 0);
    const int top = nonzero != 0 ? 32 - (__ffs(nonzero) - 1) : 0;  // hbe >= 1: some candidate exists
    const int T = min(max(top - p.depth, T_num), kBins);
    const int at_least = __shfl_sync(0xffffffffu, cum, min(max(32 - T, 0), 31));
    t.T = T;
    t.need = 0x3fffffff;  // every tied token
    t.count = T >= kBins ? 0 : (T >= 1 ? at_least : cum31 + tot0);
    if (t.count > p.sel_stride) {
        overflow = true;
        t.count = p.sel_stride;
    }
    return t;
}

// byte g of each of the 4 words, gathered into one word (byte w of the result = byte g of a[w])
template <int NW>
__device__ __forceinline__ uint32_t gather_byte(const uint32_t (&a)[NW], int g) {
    static_assert(NW == 4, "four words");
    const uint32_t sel = 0x0040u + 0x11u * g;  // bytes g of x (index g) and of y (index 4 + g)
    return __byte_perm(__byte_perm(a[0], a[1], sel), __byte_perm(a[2], a[3], sel), 0x5410u);
}

constexpr int kPlanRows = kGroup * kBins;  // 132 (head, bin) rows
constexpr int kArriveStride = 136;         // words per unit behind p.arrive: the arrival counter, then the 132 totals
// Words behind p.ready: a head's is > 0 while its plan waits for CTAs that will take it. Every waiting CTA polls its head's
// word, so a unit has a 128-byte line of its own, a head 32 bytes of it: with the words of four units in one line, a step of
// one sequence x 8 kv-heads took 21.9 us instead of 21.2 at 65536 tokens and 59.4 instead of 58.0 at 32768 with half of them
// attended (a line per head: 21.2 and 57.8).
constexpr int kReadyHead = 8;                       // words per head
constexpr int kReadyStride = kGroup * kReadyHead;   // words per unit
static_assert(kReadyStride * sizeof(int32_t) % 128 == 0, "a line per unit");

// The plan of one head of a (sequence, kv-head), worked out by warp g of the CTA that published the unit's last histogram.
// The scoring CTAs have added their histograms up in the unit's totals (33 bins x 4 heads, behind the arrival counter) and
// stored, per chunk, the counts of tokens at or above every score: the warp picks the head's threshold T and tie quota from
// the totals (lane l: bin 32 - l), reads what each chunk holds at or above T and above T (lane = chunk), and a scan gives the
// number of selected and of tied tokens that precede each chunk. The totals are left at zero for the next call. A head is
// announced by itself and no warp waits for another one. Against a plan of all four heads by 256 threads, with common
// staging, three barriers and one announcement per unit, scoring and plan take 54.7 us instead of 63.0 for 32 sequences of
// 16384 - 65536 tokens x 8 kv-heads, 18.6 instead of 21.4 for 4 x 131072, 5.2 instead of 5.7 for 3 x 9001 - 15000 (steps:
// 32 x 16000 91.4 / 94.0, 4 x 16000 29.8 / 30.2). Left out altogether, with the sums made by the chunks' CTAs, it saved
// another 0.5 - 1 us here and cost the attention kernel 8 %.
__device__ __forceinline__ void select_plan(const SelectParams& p, int b, int kvh, const SeqRange& r, int nchunks_b, int g, int lane) {
    const size_t u = (size_t)b * p.Hkv + kvh;
    const uint32_t* hbase = p.hist + (u * kPlanRows + g * kBins) * p.nchunks;
    int32_t* plan = p.plan + u * (8 + 8 * p.nchunks);
    uint32_t* unit = p.arrive + u * kArriveStride;
    uint32_t* totals = unit + 1 + g * kBins;
    const int n = (int)__ldcg(totals + 32 - lane), tot0 = (int)__ldcg(totals);
    int cum = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, cum, d);
        if (lane >= d) cum += up;
    }
    bool overflow;
    const Threshold th = pick_threshold(p, n, cum, tot0, r.hb, overflow);
    const uint32_t* ge_row = hbase + (size_t)min(th.T, kBins - 1) * p.nchunks;  // (T = 33 keeps nothing)
    int gt_carry = 0, eq_carry = 0;
    for (int c0 = 0; c0 < nchunks_b; c0 += 32) {
        const int c = c0 + lane;
        int gt = 0, eq = 0;
        if (c < nchunks_b && th.T < kBins) {
            const int ge = (int)__ldcg(ge_row + c);
            gt = th.T + 1 < kBins ? (int)__ldcg(ge_row + p.nchunks + c) : 0;
            eq = ge - gt;
        }
        int pg = gt, pe = eq;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u0 = __shfl_up_sync(0xffffffffu, pg, d), u1 = __shfl_up_sync(0xffffffffu, pe, d);
            if (lane >= d) {
                pg += u0;
                pe += u1;
            }
        }
        if (c < nchunks_b) {
            const int eq_before = eq_carry + pe - eq;
            plan[8 + 8 * c + g] = gt_carry + pg - gt + min(eq_before, th.need);
            plan[8 + 8 * c + 4 + g] = eq_before;
        }
        gt_carry += __shfl_sync(0xffffffffu, pg, 31);
        eq_carry += __shfl_sync(0xffffffffu, pe, 31);
    }
    if (lane == 0) {
        plan[g] = th.T;
        plan[4 + g] = th.need;
    }
    // hand the head over: one count per CTA of select_attend_kernel that will take this plan (a chunk each). Those CTAs run
    // while other units are still being scored; each takes its count back, so the word is zero again when the step is over.
    // (The totals and sel_cnt are written behind the announcement: they are read by kernels behind select_attend_kernel only,
    // whose edge CTAs wait for this grid to end.)
    __syncwarp();
    if (lane == 0 && p.ready != nullptr) {
        __threadfence();  // the warp's stores (ordered before this lane by the barrier) are visible device-wide
        atomicAdd(p.ready + u * kReadyStride + g * kReadyHead, nchunks_b);
    }
    totals[32 - lane] = 0u;
    if (lane == 0) {
        totals[0] = 0u;
        if (overflow) report(p.status, HA_ERR_SEL_OVERFLOW);
        p.sel_cnt[u * kGroup + g] = th.count;
    }
}

template <int ROUNDS>
__global__ void __launch_bounds__(kSelThreads, ROUNDS == 1 ? 4 : kShMinCtas) score_hist_kernel(const SelectParams p) {
    const int c = blockIdx.x, kvh = p.kvh0 + blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Hq = p.Hkv * kGroup;
    constexpr int chunk_tokens = ROUNDS * kRoundTokens;
    constexpr bool kStaged = ROUNDS > 1;  // words in flight to shared memory; else in registers

    __shared__ uint4 s_words[kStaged ? kSelWarps : 1][2][kLaneTokens * 32];
    __shared__ uint32_t s_hist[kSelWarps][kGroup * kBins];
    __shared__ int s_last;

    const int S = p.seq_lens[b];
    const bool s_ok = S >= 1 && S <= p.max_pages * kPage;
    const int chunk_start = c * chunk_tokens;
    const bool active = s_ok && chunk_start < S;
    const SeqRange r = seq_range(s_ok ? S : 1, p.init_budget, p.recent_budget, p.heavy_budget,
                                 p.budget_lens != nullptr ? p.budget_lens[b] : -1);
    // with several rounds the words of two are in flight: while one is scored the next is on its way
    RoundWords rw;
    StagedRound st[2];
    int pgs[ROUNDS];  // page ids of this warp's half pages, all requested up front
    if (active) {
#pragma unroll
        for (int rd = 0; rd < ROUNDS; ++rd) pgs[rd] = RoundWords::page_of(p, b, RoundWords::first_token(chunk_start, rd, warp));
        if constexpr (kStaged) {
#pragma unroll
            for (int rd = 0; rd < 2; ++rd)
                if (chunk_start + rd * kRoundTokens < S)
                    st[rd].copy(p, kvh, RoundWords::first_token(chunk_start, rd, warp), lane, r, pgs[rd], s_words[warp][rd]);
        } else {
            rw.load(p, kvh, RoundWords::first_token(chunk_start, 0, warp), lane, r, pgs[0]);
        }
    }
    for (int i = tid; i < kSelWarps * kGroup * kBins; i += kSelThreads) (&s_hist[0][0])[i] = 0;

    pdl_wait();
    pdl_launch_dependents();

    if (!s_ok) {
        if (tid == 0 && c == 0 && blockIdx.y == 0) report(p.status, HA_ERR_BAD_SEQ_LEN);
        return;
    }
    if (!active) return;
    const uint4 qn = load_qn(p, b, kvh);
    __syncthreads();  // s_hist is zero

    uint32_t* h0 = &s_hist[warp][0];
    const size_t pitch = (size_t)p.nchunks * chunk_tokens;
    uint8_t* plane0 = p.scores + ((size_t)b * Hq + kvh * kGroup) * pitch;
    bool bad_page = false;
#pragma unroll
    for (int rd = 0; rd < ROUNDS; ++rd) {
        if (chunk_start + rd * kRoundTokens >= S) break;
        StagedRound& cur = st[rd % 2];
        int t0, page;
        const uint4* words = s_words[kStaged ? warp : 0][rd % 2] + lane;
        bool interior, page_ok;
        if constexpr (kStaged) {
            if (rd + 1 < ROUNDS && chunk_start + (rd + 1) * kRoundTokens < S) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            t0 = cur.t0;
            interior = cur.interior(r);
            page_ok = cur.page_ok;
            page = cur.page;
        } else {
            t0 = RoundWords::first_token(chunk_start, 0, warp);
            interior = rw.interior;
            page_ok = pgs[0] >= 0 && pgs[0] < p.num_pages;
            page = rw.page;
        }
        uint32_t plane[kGroup] = {0u, 0u, 0u, 0u};  // per head: byte it = score + 1 of this lane's it-th token
        if (interior && p.scores_dbg == nullptr) {
            // the common round: every token is a candidate. The four scores of a token are packed with byte
            // permutes and the 4 x 4 bytes of the lane's tokens transposed at the end.
            uint32_t tok[kLaneTokens];
#pragma unroll
            for (int it = 0; it < kLaneTokens; ++it) {
                const uint4 w = kStaged ? words[it * 32] : rw.w[it];
                const uint32_t s0 = __popc(qn.x ^ w.x), s1 = __popc(qn.y ^ w.y);
                const uint32_t s2 = __popc(qn.z ^ w.z), s3 = __popc(qn.w ^ w.w);
                atomicAdd(h0 + s0, 1u);
                atomicAdd(h0 + kBins + s1, 1u);
                atomicAdd(h0 + 2 * kBins + s2, 1u);
                atomicAdd(h0 + 3 * kBins + s3, 1u);
                // bytes (s0, s1, s2, s3): byte 1 of a score register is zero and fills the unused positions
                tok[it] = __byte_perm(__byte_perm(s0, s1, 0x1140u), __byte_perm(s2, s3, 0x1140u), 0x5410u) + 0x01010101u;
            }
#pragma unroll
            for (int g = 0; g < kGroup; ++g) plane[g] = gather_byte<kLaneTokens>(tok, g);
        } else {
#pragma unroll
            for (int it = 0; it < kLaneTokens; ++it) {
                const int t = t0 + it * 32 + lane;
                const bool exists = t < S;
                bad_page |= exists && !page_ok;
                uint4 w = kStaged ? words[it * 32] : rw.w[it];
                if (t == S - 1 && page_ok)  // the newest token's word, which the encoder may have written in the meantime
                    w = __ldcg(p.hash_pages + ((size_t)page * p.Hkv + kvh) * kPage + t % kPage);
                const uint32_t s0 = __popc(qn.x ^ w.x), s1 = __popc(qn.y ^ w.y);
                const uint32_t s2 = __popc(qn.z ^ w.z), s3 = __popc(qn.w ^ w.w);
                if (page_ok && t >= r.lo && t < r.hi) {
                    atomicAdd(h0 + s0, 1u);
                    atomicAdd(h0 + kBins + s1, 1u);
                    atomicAdd(h0 + 2 * kBins + s2, 1u);
                    atomicAdd(h0 + 3 * kBins + s3, 1u);
                    plane[0] |= (s0 + 1u) << (8 * it);
                    plane[1] |= (s1 + 1u) << (8 * it);
                    plane[2] |= (s2 + 1u) << (8 * it);
                    plane[3] |= (s3 + 1u) << (8 * it);
                }
                if (p.scores_dbg != nullptr && exists && page_ok) {
                    const size_t dpitch = (size_t)p.max_pages * kPage;
                    uint8_t* d = p.scores_dbg + ((size_t)b * Hq + kvh * kGroup) * dpitch + t;
                    d[0] = (uint8_t)s0;
                    d[dpitch] = (uint8_t)s1;
                    d[2 * dpitch] = (uint8_t)s2;
                    d[3 * dpitch] = (uint8_t)s3;
                }
            }
        }
        // the round after next takes this round's place
        if constexpr (kStaged) {
            if (rd + 2 < ROUNDS && chunk_start + (rd + 2) * kRoundTokens < S)
                cur.copy(p, kvh, RoundWords::first_token(chunk_start, rd + 2, warp), lane, r, pgs[rd + 2 < ROUNDS ? rd + 2 : 0], s_words[warp][rd % 2]);
        }
        // the selection works from these bytes instead of the 16-byte hash words
#pragma unroll
        for (int g = 0; g < kGroup; ++g)
            *reinterpret_cast<uint32_t*>(plane0 + g * pitch + t0 + lane * 4) = plane[g];
    }
    if (bad_page) report(p.status, HA_ERR_BAD_PAGE);
    __syncthreads();
    // the chunk's histogram: added to the unit's totals, and stored as counts of tokens at or above each score.
    // Warp g takes head g, lane l the score 32 - l (a scan over the lanes gives "at or above"); lane 0 also score 0.
    uint32_t* unit = p.arrive + ((size_t)b * p.Hkv + kvh) * kArriveStride;
    if (warp < kGroup) {
        const int row0 = warp * kBins;
        uint32_t v = 0, v0 = 0;
#pragma unroll
        for (int w = 0; w < kSelWarps; ++w) {
            v += s_hist[w][row0 + 32 - lane];
            v0 += s_hist[w][row0];
        }
        if (v != 0u) atomicAdd(unit + 1 + row0 + 32 - lane, v);
        if (lane == 0 && v0 != 0u) atomicAdd(unit + 1 + row0, v0);
        uint32_t ge = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, ge, d);
            if (lane >= d) ge += u;
        }
        uint32_t* dst = p.hist + (((size_t)b * p.Hkv + kvh) * (kGroup * kBins) + row0) * p.nchunks + c;
        dst[(size_t)(32 - lane) * p.nchunks] = ge;
        if (lane == 31) dst[0] = ge + v0;
    }

    // ---- the CTA that publishes last for this (sequence, kv-head) works the unit's plan out. Nobody waits:
    //      every CTA makes its histogram visible, then counts itself in; the one that finds all the others
    //      counted reads their histograms and leaves the counter at zero for the next call.
    __syncthreads();
    const int nchunks_b = (S + chunk_tokens - 1) / chunk_tokens;
    if (tid == 0) {
        __threadfence();  // what the CTA has written (ordered before this thread by the barrier) is visible device-wide
        uint32_t* counter = unit;
        const uint32_t before = atomicAdd(counter, 1u);
        s_last = before + 1u == (uint32_t)nchunks_b;
        if (s_last) {
            *counter = 0u;
            __threadfence();  // what the other CTAs made visible before they counted themselves in is read behind this
        }
    }
    __syncthreads();
    if (s_last && warp < kGroup) select_plan(p, b, kvh, r, nchunks_b, warp, lane);
}

// ------------------------------------------------------------------------------------------
// Single-kernel variant for few units of up to 65536 tokens, where the chain of dependent steps is all there is (hash
// words, exchange, threshold, counts, emission): a cluster of 8 CTAs owns one (sequence, kv-head), CTA r the r-th eighth
// of the sequence, a warp one block of 128 consecutive tokens, held in registers (two blocks, 32 apart, beyond 32768
// tokens). A CTA so has one histogram and one place in each list. The CTAs push their histograms into one another's shared
// memory (a remote store costs the sender nothing, a remote read a round trip), the threshold warps add them up on the
// way, and every warp sums the counts of the blocks in front of its own. The hash pages are read once, and no histogram, plan
// or score byte passes through global memory. Results are identical to score_hist_kernel + select_attend_kernel.
//
// Threads follow the length, so that a warp has one block where 1024 threads allow it: with 512 threads (which several
// CTAs on an SM and the neighbouring kernels can live with) up to 16384 tokens. Decode step of one sequence x 8 kv-heads,
// against CTAs of 1024 threads that walked the sequence in common rounds of 32768 tokens and read one another's
// histograms (both in turn, mean over placements of the buffers, +-0.05 us): 13.3 -> 11.3 us at 700 tokens, 20.5 -> 16.1
// at 4096 (1/4 budget), 17.4 -> 14.2 at 16000, 16.8 -> 15.6 at 20000, 18.2 -> 17.8 at 28000, 22.4 -> 20.2 at 40000, 24.0 ->
// 22.3 at 50000; at 32768, where the division of the work is the same, 18.15 -> 18.22 on one box and 17.97 -> 17.71 on
// another. 8 sequences x 1 kv-head at 33001: 20.3 -> 19.0. With the blocks' prefixes scanned by one warp per head behind a
// barrier of its own, instead of the sums every warp makes for itself: 18.59 and 18.07 at 32768, 20.4 at 8 x 33001, 21.1
// at 40000, 0.1 to 0.2 us more than now at the others.
// ------------------------------------------------------------------------------------------
constexpr int kClCtas = 8;                                    // portable cluster size
constexpr int kClBlock = kLaneTokens * 32;                    // 128 tokens of a warp: half a page
__host__ __device__ constexpr int cluster_tokens(int threads, int blocks) { return kClCtas * (threads / 32) * blocks * kClBlock; }
constexpr int kClMaxTokens = cluster_tokens(1024, 2);         // 65536

__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// kBlocks: blocks of a warp
template <int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, 1) score_select_cluster_kernel(const SelectParams p) {
    constexpr int kWarps = kThreads / 32, kSlots = kWarps * kBlocks;  // blocks of a CTA, in token order
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int kvh = p.kvh0 + blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Hq = p.Hkv * kGroup;
    constexpr int kHist = kGroup * kBins;  // 132
    constexpr int kCopies = 8;             // warp w counts in copy w % 8

    __shared__ uint32_t s_hist[kCopies][kHist];
    __shared__ uint32_t s_all[kClCtas][kHist];  // every CTA's histogram, pushed by its owner
    __shared__ int s_T[kGroup], s_need[kGroup], s_base[kGroup], s_eqb[kGroup];
    __shared__ uint2 s_count[kSlots];                // per block: tokens above / at the threshold, a byte per head
    for (int i = tid; i < kCopies * kHist; i += kThreads) (&s_hist[0][0])[i] = 0;

    const int S = p.seq_lens[b];
    const bool s_ok = S >= 1 && S <= p.max_pages * kPage && S <= cluster_tokens(kThreads, kBlocks);
    const SeqRange r = seq_range(s_ok ? S : 1, p.init_budget, p.recent_budget, p.heavy_budget,
                                 p.budget_lens != nullptr ? p.budget_lens[b] : -1);
    // whole blocks per CTA, spread evenly over the cluster
    const int nblk = (r.S + kClCtas * kClBlock - 1) / (kClCtas * kClBlock);
    auto first_of = [&](int nb) { return (rank * nblk + nb * kWarps + warp) * kClBlock; };
    auto has = [&](int nb) { return s_ok && nb * kWarps + warp < nblk && first_of(nb) < r.S; };  // warp-uniform
    RoundWords rw;
    if (has(0)) rw.load(p, b, kvh, first_of(0), lane, r);
    cluster_arrive_relaxed();  // (the matching wait stands in front of the first push: by then every CTA has started)

    pdl_wait();
    pdl_launch_dependents();
    if (!s_ok && tid == 0 && rank == 0 && blockIdx.y == 0) report(p.status, HA_ERR_BAD_SEQ_LEN);

    const uint4 qn = load_qn(p, b, kvh);
    __syncthreads();  // s_hist is zero
    // token it * 32 + lane of a block: byte g = head g's score + 1, 0 = not a candidate
    uint32_t word[kBlocks][kLaneTokens];
    int row[kBlocks];  // physical row of the block's first token (used where a token was selected: its page is good)
    uint32_t* h0 = &s_hist[warp % kCopies][0];
#pragma unroll
    for (int nb = 0; nb < kBlocks; ++nb) {
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it) word[nb][it] = 0u;
        row[nb] = 0;
        if (!has(nb)) continue;
        const int t0 = first_of(nb);
        if (nb > 0) rw.load(p, b, kvh, t0, lane, r);
        rw.refresh_newest(p, kvh, t0, lane, r);
        if (rw.bad_page) report(p.status, HA_ERR_BAD_PAGE);
        row[nb] = rw.page * kPage + t0 % kPage;
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it) {
            const uint32_t s0 = __popc(qn.x ^ rw.w[it].x), s1 = __popc(qn.y ^ rw.w[it].y);
            const uint32_t s2 = __popc(qn.z ^ rw.w[it].z), s3 = __popc(qn.w ^ rw.w[it].w);
            if (rw.interior || ((rw.cand >> it) & 1u)) {
                atomicAdd(h0 + s0, 1u);
                atomicAdd(h0 + kBins + s1, 1u);
                atomicAdd(h0 + 2 * kBins + s2, 1u);
                atomicAdd(h0 + 3 * kBins + s3, 1u);
                word[nb][it] = __byte_perm(__byte_perm(s0, s1, 0x1140u), __byte_perm(s2, s3, 0x1140u), 0x5410u) + 0x01010101u;
            }
            if (p.scores_dbg != nullptr && ((rw.valid >> it) & 1u)) {
                const size_t pitch = (size_t)p.max_pages * kPage;
                uint8_t* d = p.scores_dbg + ((size_t)b * Hq + kvh * kGroup) * pitch + t0 + it * 32 + lane;
                d[0] = (uint8_t)s0;
                d[pitch] = (uint8_t)s1;
                d[2 * pitch] = (uint8_t)s2;
                d[3 * pitch] = (uint8_t)s3;
            }
        }
    }

    // ---- push the histogram to every CTA of the cluster
    cluster_wait();
    __syncthreads();
    if (tid < kHist) {
        uint32_t v = 0;
#pragma unroll
        for (int k = 0; k < kCopies; ++k) v += s_hist[k][tid];
#pragma unroll
        for (int k = 0; k < kClCtas; ++k) *cluster.map_shared_rank(&s_all[rank][tid], k) = v;
    }
    cluster_arrive();
    cluster_wait();
    if (!s_ok) return;  // the same in every CTA of the cluster; nothing is read from another CTA's shared memory

    // ---- threshold, tie quota and this CTA's place in the list: warp g for head g, lane l holds score 32 - l
    if (warp < kGroup) {
        const int g = warp;
        int n = 0, nb = 0, tot0 = 0, bef0 = 0;  // candidates with that score: in all, and in the CTAs in front of this one
#pragma unroll
        for (int k = 0; k < kClCtas; ++k) {
            const int v = (int)s_all[k][g * kBins + 32 - lane], v0 = (int)s_all[k][g * kBins];
            n += v;
            tot0 += v0;
            nb += k < rank ? v : 0;
            bef0 += k < rank ? v0 : 0;
        }
        int cum = n, cumb = nb;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, cum, d), ub = __shfl_up_sync(0xffffffffu, cumb, d);
            if (lane >= d) {
                cum += u;
                cumb += ub;
            }
        }
        bool overflow;
        const Threshold th = pick_threshold(p, n, cum, tot0, r.hb, overflow);
        const int lt = min(max(32 - th.T, 0), 31);
        const int gt_l = __shfl_sync(0xffffffffu, cumb - nb, lt), eq_l = __shfl_sync(0xffffffffu, nb, lt);
        const int all31 = __shfl_sync(0xffffffffu, cumb, 31);
        int gt_before = 0, eq_before = 0;
        if (th.T >= 1 && th.T <= 32) {
            gt_before = gt_l;
            eq_before = eq_l;
        } else if (th.T == 0) {
            gt_before = all31;
            eq_before = bef0;
        }
        if (lane == 0) {
            s_T[g] = th.T;
            s_need[g] = th.need;
            s_eqb[g] = eq_before;
            s_base[g] = gt_before + min(eq_before, th.need);
            if (rank == 0) {
                if (overflow) report(p.status, HA_ERR_SEL_OVERFLOW);
                p.sel_cnt[(size_t)b * Hq + kvh * kGroup + g] = th.count;
            }
        }
    }
    __syncthreads();

    // ---- classify: stored bytes are score + 1 (0: no candidate) and are compared with T + 1 >= 1
    const uint32_t t4 = ((uint32_t)s_T[0] | ((uint32_t)s_T[1] << 8) | ((uint32_t)s_T[2] << 16) | ((uint32_t)s_T[3] << 24)) + 0x01010101u;
    const uint32_t gt_add = 0x7F7F7F7Fu - t4, ge_add = 0x80808080u - t4;
    uint32_t cgt[kBlocks], ceq[kBlocks];
#pragma unroll
    for (int nb = 0; nb < kBlocks; ++nb) {
        uint32_t cg_ = 0, ce_ = 0;
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it) {
            const uint32_t gt = (word[nb][it] + gt_add) & 0x80808080u;
            cg_ += gt >> 7;
            ce_ += ((word[nb][it] + ge_add) & 0x80808080u & ~gt) >> 7;
        }
        cgt[nb] = __reduce_add_sync(0xffffffffu, cg_);  // <= 128 per byte: no carry between heads
        ceq[nb] = __reduce_add_sync(0xffffffffu, ce_);
        if (lane == 0) s_count[nb * kWarps + warp] = make_uint2(cgt[nb], ceq[nb]);
    }
    __syncthreads();
    // ---- emission: position in the head's list, ties by token index
    const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
    for (int nb = 0; nb < kBlocks; ++nb) {
        if ((cgt[nb] | ceq[nb]) == 0) continue;  // nothing of any head in this block
        // what the CTA's blocks in front of this one hold, 16 bits per head (at most 64 blocks of at most 128). Every warp
        // adds them up for itself: a scan by one warp per head costs a second barrier of all threads (times above).
        uint32_t gt01 = 0, gt23 = 0, eq01 = 0, eq23 = 0;
#pragma unroll
        for (int k = 0; k <= nb; ++k) {
            const bool in = lane < kWarps && (k < nb || lane < warp);
            const uint2 c = in ? s_count[k * kWarps + lane] : make_uint2(0u, 0u);
            gt01 += __byte_perm(c.x, 0u, 0x4140u);
            gt23 += __byte_perm(c.x, 0u, 0x4342u);
            eq01 += __byte_perm(c.y, 0u, 0x4140u);
            eq23 += __byte_perm(c.y, 0u, 0x4342u);
        }
        gt01 = __reduce_add_sync(0xffffffffu, gt01);
        gt23 = __reduce_add_sync(0xffffffffu, gt23);
        eq01 = __reduce_add_sync(0xffffffffu, eq01);
        eq23 = __reduce_add_sync(0xffffffffu, eq23);
        int base_pos[kGroup], eqb[kGroup];
        uint32_t full4 = 0, straddle = 0;
#pragma unroll
        for (int g = 0; g < kGroup; ++g) {
            const int gt_before = (int)(((g < 2 ? gt01 : gt23) >> (16 * (g & 1))) & 0xffffu);
            const int eq_before = (int)(((g < 2 ? eq01 : eq23) >> (16 * (g & 1))) & 0xffffu);
            const int need = s_need[g], eqb0 = s_eqb[g], eq_in = (int)((ceq[nb] >> (8 * g)) & 0xffu);
            eqb[g] = eqb0 + eq_before;
            base_pos[g] = s_base[g] + gt_before + (min(eqb[g], need) - min(eqb0, need));
            if (eqb[g] + eq_in <= need) full4 |= 0x80u << (8 * g);
            else if (eqb[g] < need) straddle |= 1u << g;
        }
        uint32_t sel[kLaneTokens], eq[kLaneTokens];
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it) {
            const uint32_t gt = (word[nb][it] + gt_add) & 0x80808080u;
            eq[it] = (word[nb][it] + ge_add) & 0x80808080u & ~gt;
            sel[it] = gt | (eq[it] & full4);
        }
        if (straddle != 0) {  // warp-uniform, at most once per (sequence, head): rank ties by token index
#pragma unroll
            for (int g = 0; g < kGroup; ++g) {
                if (!((straddle >> g) & 1u)) continue;
                int eq_run = eqb[g];
#pragma unroll
                for (int it = 0; it < kLaneTokens; ++it) {
                    const bool e = (eq[it] >> (8 * g + 7)) & 1u;
                    const uint32_t m_eq = __ballot_sync(0xffffffffu, e);
                    if (e && eq_run + __popc(m_eq & lt_mask) < s_need[g]) sel[it] |= 0x80u << (8 * g);
                    eq_run += __popc(m_eq);
                }
            }
        }
        uint32_t cnt4 = 0, bits = 0;
#pragma unroll
        for (int it = 0; it < kLaneTokens; ++it) {
            cnt4 += sel[it] >> 7;
            bits |= flags_to_nibble(sel[it]) << (4 * it);
        }
        uint32_t excl = cnt4;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, excl, d);
            if (lane >= d) excl += u;
        }
        excl -= cnt4;
        const int t_lane = first_of(nb) + lane, row_lane = row[nb] + lane;
        while (bits != 0) {
            const int i = __ffs(bits) - 1;
            bits &= bits - 1;
            const int it = i >> 2, g = i & 3;
            const int bp = g == 0 ? base_pos[0] : (g == 1 ? base_pos[1] : (g == 2 ? base_pos[2] : base_pos[3]));
            const int pos = bp + (int)((excl >> (8 * g)) & 0xffu);
            excl += 1u << (8 * g);
            if (pos < p.sel_stride) {
                const size_t o = ((size_t)b * Hq + kvh * kGroup + g) * p.sel_stride + pos;
                p.sel_idx[o] = t_lane + it * 32;
                p.sel_rows[o] = row_lane + it * 32;
            }
        }
    }
}

}  // namespace ha
