// Rows with a top-k cut, a row to a team of one, two, four or eight CTAs (a thread-block cluster),
// which look at its columns side by side.
//
// What bounds a batch that leaves the GPU room is a chain of latencies, not the bytes: ask for the data, find
// a bound, look, order, add up.  So everything that can happen side by side does, the chain is kept
// short in instructions as well as in barriers, and every step is work of all threads:
//
//   1. every warp asks the copy engine for its part of the columns, as far as shared memory reaches (64 or
//      80 KB a CTA; what has been looked at makes room for what follows);
//   2. meanwhile the token history becomes a bitmap of the CTA's columns;
//   3. the admission bound: every warp finds the j-th largest of its lanes' largest logits whose ids the history
//      has not seen, j = ceil(k / warps); at least k logits are as large as the smallest of these;
//   4. what reaches the bound, penalised if the history has seen its id, goes on a list, one entry to a
//      thread.  Columns that did not fit shared memory at once come after that, turn by turn: vectors that hold
//      something at or above the bound go into a queue as they are, so that the scan does not wait for what it
//      finds, and from there on the list; when that grows long it is cut to its k best, which lifts the bound.
//      A bound that lets whole vectors through -- a mask leaves fewer than k of the CTA's logits, they are all the same, or
//      each is larger than those before -- shows in that most lanes find something.  Such vectors are sifted first
//      (`sift`, `crowded`): logits equal to the bound count up to its id, those under it if the history has
//      seen them, infinities never.  (64 fp32 rows of 151,936, 40 ids allowed, k = 50, us a call without it / with it / ring
//      kernel: mask of -inf 66 / 17 / 118, of the lowest value 150 / 35 / 148, with penalties that raise 182 / 52 / 103
//      (streaming kernel); rows that rise 220 / 134 / 219; ordinary ones 18.7 with and without);
//   5. occurrences, if they matter, are counted in one walk over the tokens, with the entries' ids in a
//      hash table (an entry is on the list by the most it can be worth, which is the charge for one occurrence);
//   6. every CTA ranks its entries by counting the larger ones and hands its k best, in order, to the
//      team's first CTA, where each finds its place by binary searches in the other CTAs' lists.
//      The first CTA ends the row (src/sampler.c:80-122).  This is the only time the CTAs meet: a
//      cluster's barrier costs 0.6 us.
//
// Penalties may raise a logit as long as the frequency penalty is not negative: the charge for
// one occurrence still bounds what a seen id can be worth, so such rows look at what lies somewhat
// under the bound too (`raw_floor`).
//
// 256 threads with 128 registers: with 512 threads and 64 the same steps took half as long again (four warps
// of a scheduler in step make every instruction cost four cycles), and what they spilled was read back from L2,
// since shared memory leaves the L1 cache nothing.  For the same reason no function that is not inlined is
// given the kernel's parameters: it would read them through memory.
//
// The cluster's barriers are the hardware's; the waits for the copy engine are bounded.  A wait that runs
// out fails the row with FG_ERR_LIMIT.  No TMA multicast.
#include <cooperative_groups.h>

#include <cstring>

#include "fg_block_select.cuh"
#include "fg_kernels.h"
#include "fg_row_scan.cuh"

namespace fgk {
namespace team {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr uint32_t kListCap = kThreads;         // entries of a CTA's list
constexpr uint32_t kListLong = 192;             // the list is cut between two turns of the scan from here on
constexpr uint32_t kQueueCap = kThreads;        // vectors in the queue
constexpr uint32_t kQueueLong = 128;            // it is worked off between two turns from here on
constexpr uint32_t kMostTeam = 8;
constexpr uint32_t kMostRounds = 11;            // keys a warp contributes to a tight bound
constexpr uint32_t kHashBits = 9, kHashSlots = 1u << kHashBits;  // twice the list
constexpr uint32_t kLooseMost = 32;             // candidates that a loose bound is for: with more the list runs over at times
constexpr float kFarApart = 64.0f;              // a bound so far below the largest logit is a mask's, and made tight
constexpr uint32_t kDefaultPolls = 1u << 21;    // polls before a wait gives up: a second or two

// Which rows a launch takes.
enum Rows : uint32_t { kAllRows = 0, kLoweringRows = 1, kRaisingRows = 2 };

struct Params {
    const void *logits;
    uint64_t row_stride;  // elements
    uint32_t rows, vocab;
    uint32_t vocab_offset, vocab_total;
    uint32_t team;                  // CTAs that share a row
    uint32_t chunk;                 // columns of a CTA, a multiple of 128
    uint32_t which;                 // Rows
    const uint32_t *history_tokens;
    const uint64_t *history_offsets;
    uint32_t history_max;
    uint32_t bitmap_words;          // of a CTA's columns, a multiple of 32; 0: the batch has no history
    const SamplerConfig *configs;   // device copy when config_count > 1
    SamplerConfig config0;
    uint32_t config_count;
    uint32_t shard_k;               // != 0: write candidates instead of sampling
    const float *uniforms;
    float *shard_scores;
    uint32_t *shard_ids;
    uint32_t shard_stride;          // elements between consecutive candidates (2: interleaved pairs)
    PushTargets push;               // ranks != 0: candidates go straight to every rank's window
    // Session tables instead of token lists: see persist::Params.
    const uint32_t *slot_counts;
    const uint32_t *slot_bitmaps;
    const uint32_t *row_slots;
    uint32_t slot_bitmap_words;
    uint32_t wait_polls;            // polls before a wait gives up
    uint32_t withhold_cta, withhold_issue;  // test seam: that CTA's first warp never makes that request
    SelectOutput out;
};

// What the CTA knows about its row.
struct Row {
    const uint32_t *tokens;        // the row's history
    const uint32_t *counts;        // or: its session's count table, from the CTA's first column on
    uint32_t history_len;
    uint32_t id_base, columns;     // global id of the CTA's first column, and how many it has
    uint32_t k;
    float flat_offset;             // charge for count = 1 (the exact charge when frequency is +-0)
    float presence, frequency, repetition;
    uint32_t odd;                  // bits of |x| from here on: greedy rows must see it
    bool greedy, seen_any, with_counts, raises;
};

struct alignas(128) Shared {
    uint64_t landed[kWarps][2];        // "the half has landed"
    // The list.  An entry's key is its (score, ~id) or, while it waits to be counted, that of the most it
    // can be worth; 0: dead.
    uint64_t key[kListCap];
    float value[kListCap];
    uint32_t column[kListCap];
    uint32_t waiting[kListCap / 32];   // a bit per entry: a seen id whose occurrences have not been counted (the value is raw)
    uint32_t rank[kListCap];
    uint32_t count;                    // slots handed out (may run past kListCap)
    uint32_t queue_count;              // slots handed out (may run past kQueueCap)
    uint32_t bad_history, lost;        // a status; a wait ran out
    unsigned long long bound;          // (score, ~id) key: at least k logits of the row are as good (only ever rises)
    unsigned long long wild;           // greedy rows: min over NaN/Inf of (id << 32 | value bits)
    alignas(16) uint32_t warp_key[kWarps * kMostRounds];  // the warps' part of a bound
    alignas(16) uint32_t warp_top[kWarps];
    uint32_t tight_key;
    union {
        struct {
            uint32_t id[kHashSlots], count[kHashSlots];
        } hash;                             // for counting
        alignas(16) uint64_t order[kMostTeam * kMaxK];  // for ranking
        struct {
            uint4 vector[kQueueCap];
            uint32_t column[kQueueCap];
            uint8_t mask[kQueueCap];        // which elements
        } queue;
    };
    Row row;
    // the first CTA's: every CTA's k best in order
    float inbox_score[kMostTeam][kMaxK];
    uint32_t inbox_id[kMostTeam][kMaxK];
    unsigned long long inbox_wild[kMostTeam];
    uint32_t inbox_count[kMostTeam], inbox_bad[kMostTeam];
    FinishBuffer fin;
};

// Dynamic shared memory: the above, the bitmap of the CTA's columns, where every warp's vectors land.
__device__ __forceinline__ Shared &shared() {
    extern __shared__ __align__(128) unsigned char team_memory[];
    return *reinterpret_cast<Shared *>(team_memory);
}
__device__ __forceinline__ uint32_t *seen_bitmap() { return reinterpret_cast<uint32_t *>(&shared() + 1); }
__device__ __forceinline__ uint4 *stages(const Params &p) { return reinterpret_cast<uint4 *>(seen_bitmap() + p.bitmap_words); }

// The CTAs that share a row.
__device__ __forceinline__ void team_arrive(uint32_t team) {
    if (team > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void team_wait(uint32_t team) {
    if (team > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    else __syncthreads();
}
template <class V>
__device__ __forceinline__ V *in_first_cta(V *mine, uint32_t team) {
    return team == 1 ? mine : cooperative_groups::this_cluster().map_shared_rank(mine, 0);
}

__device__ __forceinline__ bool seen_column(const Row &r, uint32_t column) {
    if (!r.seen_any) return false;
    return (seen_bitmap()[column >> 5] >> (column & 31u)) & 1u;
}

// The larger of `best` and a vector's largest finite logit among those the history has not seen.
template <int N>
__device__ __forceinline__ float largest_unseen(const float (&v)[N], uint32_t column, float best) {
    const float most = largest(v);
    if (!(most > best)) return best;
    if (!shared().row.seen_any && !is_nonfinite(most)) return most;
#pragma unroll
    for (int j = 0; j < N; j++)
        if (v[j] > best && !is_nonfinite(v[j]) && !seen_column(shared().row, column + (uint32_t)j)) best = v[j];
    return best;
}

// Raw logits under this cannot reach tau: unseen ones are their own value; of a seen one `most` is
// the most it can be worth, and that grows with the logit.
__device__ __noinline__ float raw_floor(float tau) {
    const Row &r = shared().row;
    const Repetition repetition = make_repetition(r.repetition);
    float at = __fadd_rn(tau, r.flat_offset);
    if (repetition.active) at = at > 0.0f ? __fmul_rn(at, repetition.value) : __fdiv_rn(at, repetition.value);
    at = fminf(at, tau);
    float slack = 1e-6f * fmaxf(fmaxf(fabsf(at), fabsf(tau)), fabsf(r.flat_offset)) + 1e-30f;
    for (int i = 0; i < 24; i++) {
        const float low = at - slack;
        if (penalise_with_offset(low, r.flat_offset, repetition) < tau) return low;
        slack *= 8.0f;
    }
    return __uint_as_float(0xff800000u);
}

// What a bound asks of a raw logit.  An unseen one must be larger than `tau`, or equal to it with an id up
// to `last_id`; a seen one must reach `floor`, which is tau unless penalties may raise it.
struct Gate {
    uint64_t bound;
    float tau, floor;
    __device__ __forceinline__ uint32_t last_id() const { return ~(uint32_t)bound; }
};
__device__ __forceinline__ Gate gate_of(uint64_t bound) {
    Gate g;
    g.bound = bound;
    g.tau = key_to_float((uint32_t)(bound >> 32));
    g.floor = shared().row.raises ? raw_floor(g.tau) : g.tau;
    return g;
}
// What the largest logit of a vector must be for a look at it: `at_least`, or `above` if no id in there is below
// `ties_lose`.  (An infinity is no candidate: greedy rows find it otherwise.)
struct VectorGate {
    float at_least, above;
    uint32_t ties_lose;  // a column of the CTA's
};
__device__ __forceinline__ VectorGate gate_of_vectors(const Gate &g) {
    const Row &r = shared().row;
    constexpr float kLowest = -3.402823466e38f;
    VectorGate v;
    v.at_least = fmaxf(g.floor, kLowest);
    v.above = fmaxf(key_to_float((uint32_t)(g.bound >> 32) + 1u), kLowest);
    const uint32_t last = g.last_id();
    v.ties_lose = r.raises || last >= r.id_base + r.columns ? 0xffffffffu : last < r.id_base ? 0u : last - r.id_base + 1u;
    return v;
}

// NaN, infinities and magnitudes a repetition factor of 2^-40 to 2^40 could push there: greedy rows
// must see them.  (The charge cannot: penalties are 2 at most, so it is less than the last place of such a
// value, and whether the value becomes infinite does not depend on the count.)
__device__ __forceinline__ bool odd_value(float x, uint32_t odd) { return (__float_as_uint(x) & 0x7fffffffu) >= odd; }
template <int N>
__device__ __forceinline__ bool odd_values(const float (&v)[N], uint32_t odd) {
    return !(propagating_max(v[0], v) < __uint_as_float(odd)) || smallest(v) <= -__uint_as_float(odd);
}

// A gate with what else decides over whole vectors, for where a mask, equal logits or a penalty that raises let many
// through: few elements of theirs are left then.
struct Sieve {
    Gate gate;
    uint32_t first_id, odd;
    bool greedy, marked;  // marked: it makes a difference whether the history has seen a column
};
__device__ __forceinline__ Sieve sieve_of(const Gate &gate) {
    const Row &r = shared().row;
    return Sieve{gate, r.id_base, r.odd, r.greedy, r.seen_any && (r.greedy || r.raises)};
}
// Which of a vector's columns the history has seen, a bit each.
template <int N>
__device__ __forceinline__ uint32_t seen_columns(uint32_t column) {
    const uint32_t word = column >> 5, shift = column & 31u;
    const uint32_t *bitmap = seen_bitmap();
    uint32_t seen = bitmap[word] >> shift;
    if (shift + N > 32u) seen |= bitmap[word + 1u] << (32u - shift);  // (the vector ends in there)
    return seen & ((1u << N) - 1u);
}
// Whether any element of a vector may be worth the bound.
template <int N>
__device__ __forceinline__ bool may_pass(const float (&v)[N], uint32_t column, const Sieve &s) {
    const float most = largest(v);
    return s.greedy || most > s.gate.tau || (most == s.gate.tau && s.first_id + column <= s.gate.last_id()) ||
           (s.marked && seen_columns<N>(column) != 0);
}
// Which of them, a bit each.  Greedy rows also look at the first NaN or infinity (the smallest id counts) and at what
// a penalty may turn into one.
template <int N>
__device__ __forceinline__ uint32_t passing(const float (&v)[N], uint32_t column, const Sieve &s) {
    const uint32_t first = s.first_id + column, last = s.gate.last_id(), seen = s.marked ? seen_columns<N>(column) : 0u;
    uint32_t pass = 0, wild = 0;
#pragma unroll
    for (int j = 0; j < N; j++) {
        const bool was_seen = (seen >> j) & 1u, finite = !is_nonfinite(v[j]);
        const bool take = v[j] > s.gate.tau || (v[j] == s.gate.tau && first + (uint32_t)j <= last) ||
                          (was_seen && (v[j] >= s.gate.floor || (s.greedy && odd_value(v[j], s.odd))));
        pass |= (take && finite ? 1u : 0u) << j;
        wild |= (finite ? 0u : 1u) << j;
    }
    if (s.greedy && wild != 0 && first + (uint32_t)__ffs(wild) - 1u < (uint32_t)(peek64(&shared().wild) >> 32))
        pass |= wild & (0u - wild);
    return pass;
}

// Bounds for k lanes' keys: at least k of them are as large.  `largest`: the largest of all lanes' keys.  All
// threads call.
//
// Every warp contributes three more than k / warps, and of all those the k-th largest is taken (k and a few keys are as
// large: worth a step more when much of the row is still to come).  Syncs twice.  One copy for all its users:
// instructions that have not run before come from L2.
__device__ __noinline__ uint2 tight_bound(uint32_t key, uint32_t k) {
    Shared &sh = shared();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t rounds = min((k + kWarps - 1u) / kWarps + 3u, kMostRounds), keys = rounds * kWarps;
    uint32_t found = __reduce_max_sync(kFullMask, key);
    for (uint32_t i = 0;; i++) {
        if (lane == 0) sh.warp_key[i * kWarps + warp] = found;
        if (i + 1u >= rounds) break;
        const unsigned owners = __ballot_sync(kFullMask, key == found);
        if ((int)lane == __ffs(owners) - 1) key = 0;
        found = __reduce_max_sync(kFullMask, key);
    }
    if (tid == 0) sh.tight_key = 0;
    __syncthreads();
    if (tid < keys) {
        // (equal keys are counted together, so that somebody finds the k-th)
        const uint32_t mine = sh.warp_key[tid];
        uint32_t larger = 0, equal = 0;
        for (uint32_t i = 0; i < keys; i += 4) {
            const uint4 four = *reinterpret_cast<const uint4 *>(&sh.warp_key[i]);
            larger += (four.x > mine) + (four.y > mine) + (four.z > mine) + (four.w > mine);
            equal += (four.x == mine) + (four.y == mine) + (four.z == mine) + (four.w == mine);
        }
        if (larger < k && larger + equal >= k) sh.tight_key = mine;
        if (larger == 0) sh.warp_top[0] = mine;
    }
    __syncthreads();
    return make_uint2(sh.tight_key, sh.warp_top[0]);
}

// Every warp's j-th largest, j = ceil(k / warps), of the `warps` first warps; the smallest of them (twice k keys or so
// are as large).  Syncs once, in the middle.
__device__ __forceinline__ uint2 loose_bound(uint32_t key, uint32_t k, uint32_t warps) {
    Shared &sh = shared();
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t found = __reduce_max_sync(kFullMask, key);
    const uint32_t top = found;
    for (uint32_t each = (k + warps - 1u) / warps; each > 1u; each--) {
        const unsigned owners = __ballot_sync(kFullMask, key == found);
        if ((int)lane == __ffs(owners) - 1) key = 0;
        found = __reduce_max_sync(kFullMask, key);
    }
    if (lane == 0) {
        sh.warp_key[warp] = found;
        sh.warp_top[warp] = top;
    }
    __syncthreads();
    uint32_t low = 0xffffffffu, high = 0;
#pragma unroll
    for (uint32_t w = 0; w < (uint32_t)kWarps; w += 4) {
        const uint4 four = *reinterpret_cast<const uint4 *>(&sh.warp_key[w]), tops = *reinterpret_cast<const uint4 *>(&sh.warp_top[w]);
        const uint32_t keys[4] = {four.x, four.y, four.z, four.w};
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) low = w + q < warps ? min(low, keys[q]) : low;
        high = max(max(high, max(tops.x, tops.y)), max(tops.z, tops.w));
    }
    return make_uint2(low, high);
}

// What a logit is worth (src/sampler.c:52-58).
struct Worth {
    uint64_t key;  // 0: not worth the bound
    float value;   // the raw logit if it waits to be counted
    bool waits;
};
__device__ __forceinline__ Worth worth_of(float raw, uint32_t column, uint64_t bound) {
    Shared &sh = shared();
    const Row &r = sh.row;
    const uint32_t id = r.id_base + column;
    Worth w = {0ull, raw, false};
    if (seen_column(r, column)) {
        const Repetition repetition = make_repetition(r.repetition);
        if (r.with_counts && r.counts != nullptr) {
            const uint32_t times = __ldg(&r.counts[column]);  // the session's table holds the exact count
            if (times != 0) w.value = penalise_with_offset(raw, penalty_offset(times, r.presence, r.frequency), repetition);
        } else {
            // (the charge grows with the count: the most the id can be worth)
            w.value = penalise_with_offset(raw, r.flat_offset, repetition);
            w.waits = r.with_counts;
        }
    }
    if (!is_nonfinite(w.value)) {
        w.key = select_key(w.value, id);
        if (w.key < bound) w.key = 0;
    } else if (r.greedy) {
        atomicMin(&sh.wild, ((unsigned long long)id << 32) | __float_as_uint(w.value));  // (for any count: see odd_value)
    }
    if (w.waits) w.value = raw;
    return w;
}
__device__ __forceinline__ bool entry_waits(const Shared &sh, uint32_t i) { return (sh.waiting[i >> 5] >> (i & 31u)) & 1u; }

// Counts the occurrences of the entries that wait for it, and gives them their exact value.  One that
// does not reach the bound is dead.  All threads call; ends synced.  `last`: no id is looked up any more, and the
// bitmap of seen columns becomes one of those that are to be counted, which few tokens pass.
__device__ __noinline__ void settle(bool last) {
    Shared &sh = shared();
    const Row &r = sh.row;
    const uint32_t tid = threadIdx.x;
    const bool waits = tid < min(sh.count, kListCap) && entry_waits(sh, tid);
    const bool need = waits && sh.key[tid] >= peek64(&sh.bound);
    const uint32_t column = need ? sh.column[tid] : 0u, id = r.id_base + column;
    if (waits && !need) sh.key[tid] = 0;
    const bool any = __syncthreads_or(need);
    if (tid < kListCap / 32) sh.waiting[tid] = 0;
    if (any) {
        for (uint32_t i = tid; i < kHashSlots; i += kThreads) {
            sh.hash.id[i] = kPaddingId;
            sh.hash.count[i] = 0;
        }
        uint32_t *bitmap = seen_bitmap();
        if (last) {
            uint4 *words = reinterpret_cast<uint4 *>(bitmap);
            for (uint32_t i = tid; i < (r.columns + 127u) / 128u; i += kThreads) words[i] = make_uint4(0, 0, 0, 0);
        }
        __syncthreads();
        auto first_slot = [](uint32_t of) { return (of * 0x9e3779b1u) >> (32u - kHashBits); };
        uint32_t place = first_slot(id);
        if (need) {
            if (last) atomicOr(&bitmap[column >> 5], 1u << (column & 31u));
            // (at most half the slots are ever taken, and no id twice: the walk ends)
            while (atomicCAS(&sh.hash.id[place], kPaddingId, id) != kPaddingId) place = (place + 1u) & (kHashSlots - 1u);
        }
        __syncthreads();
        constexpr int kBatch = 16;  // tokens per thread and trip, loaded before any is used
        for (uint32_t base = 0; base < r.history_len; base += kBatch * kThreads) {
            uint32_t token[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                const uint32_t at = base + (uint32_t)q * kThreads + tid;
                token[q] = at < r.history_len ? __ldg(&r.tokens[at]) : kPaddingId;
            }
            uint32_t found = 0;
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                const uint32_t local = token[q] - r.id_base;  // wraps for ids below the CTA's columns
                const bool ours = token[q] != kPaddingId && local < r.columns;
                found |= (ours && ((bitmap[ours ? local >> 5 : 0u] >> (local & 31u)) & 1u) ? 1u : 0u) << q;
            }
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                if (((found >> q) & 1u) == 0) continue;
                uint32_t slot = first_slot(token[q]);
                for (;;) {
                    const uint32_t there = sh.hash.id[slot];
                    if (there == kPaddingId) break;
                    if (there == token[q]) {
                        atomicAdd(&sh.hash.count[slot], 1u);
                        break;
                    }
                    slot = (slot + 1u) & (kHashSlots - 1u);
                }
            }
        }
        __syncthreads();
        if (need) {
            const float raw = sh.value[tid];
            const uint32_t times = sh.hash.count[place];
            const float exact = times == 0 ? raw
                : penalise_with_offset(raw, penalty_offset(times, r.presence, r.frequency), make_repetition(r.repetition));
            const uint64_t key = select_key(exact, id);  // (finite, as what it was listed by: see odd_value)
            sh.value[tid] = exact;
            sh.key[tid] = key >= peek64(&sh.bound) ? key : 0ull;
        }
    }
    __syncthreads();
}

// Ranks the first n entries: sh.rank[i] becomes the number of larger keys in sh.order[0 .. n) (keys are
// distinct, 0 is nobody's).  Several threads count for one entry, each over a part of the list.  All threads
// call, with order[] written and rank[] cleared, synced; ends synced.
__device__ __forceinline__ void rank_entries(Shared &sh, uint32_t n) {
    const uint32_t tid = threadIdx.x;
    const uint32_t bits = n <= 32u ? 5u : n <= 64u ? 6u : n <= 128u ? 7u : 8u, parts = kThreads >> bits;
    const uint32_t each = ((n + parts - 1u) / parts + 1u) & ~1u;  // (two keys to a load)
    const uint32_t at = tid & ((1u << bits) - 1u), from = (tid >> bits) * each, to = min(n, from + each);
    if (at < n) {
        const uint64_t key = sh.order[at];
        uint32_t larger = 0;
#pragma unroll 4
        for (uint32_t j = from; j < to; j += 2) {  // (behind the last entry: zero)
            const ulonglong2 two = *reinterpret_cast<const ulonglong2 *>(&sh.order[j]);
            larger += (two.x > key ? 1u : 0u) + (two.y > key ? 1u : 0u);
        }
        if (larger != 0) atomicAdd(&sh.rank[at], larger);
    }
    __syncthreads();
}

// The list is cut: the k-th best of the entries that need not be counted bounds the row, and what does
// not reach that goes.  `hard`: the others are counted first, so that k entries are
// left at most.  All threads call; ends synced.
__device__ __noinline__ void tighten(bool hard) {
    Shared &sh = shared();
    const uint32_t tid = threadIdx.x;
    __syncthreads();
    const uint32_t n = min(sh.count, kListCap), k = sh.row.k;
    if (hard) settle(false);
    sh.order[tid] = tid < n && !entry_waits(sh, tid) ? sh.key[tid] : 0ull;
    sh.rank[tid] = 0;
    __syncthreads();
    rank_entries(sh, n);
    const uint64_t mine = sh.order[tid];
    if (mine != 0 && sh.rank[tid] == k - 1u) atomicMax(&sh.bound, (unsigned long long)mine);
    __syncthreads();
    const uint64_t key = tid < n ? sh.key[tid] : 0ull;
    const bool keep = key != 0 && key >= peek64(&sh.bound);
    const bool waits = keep && entry_waits(sh, tid);
    const float value = keep ? sh.value[tid] : 0.0f;
    const uint32_t column = keep ? sh.column[tid] : 0u;
    __syncthreads();
    if (tid < kListCap / 32) sh.waiting[tid] = 0;
    if (tid == 0) sh.count = 0;
    __syncthreads();
    if (keep) {
        const uint32_t slot = atomicAdd(&sh.count, 1u);
        sh.key[slot] = key;
        sh.value[slot] = value;
        sh.column[slot] = column;
        if (waits) atomicOr(&sh.waiting[slot >> 5], 1u << (slot & 31u));
    }
    __syncthreads();
}

// The vectors of a CTA's columns, kHalf of a thread in half a turn at most (fewer if all of them are one turn's and
// that does not take as many: then they are dealt out to all warps evenly).  In the turn at `base` a thread's
// (h kHalf + u)-th, the u-th of half h, is number(base, h kHalf + u).
template <typename T, int kHalf>
struct Vectors {
    static constexpr int kPer = Lanes<T>::kPer;
    const T *body;    // the CTA's first 16-byte boundary
    uint32_t count;   // vectors from there on
    uint32_t head;    // columns before it
    uint32_t span;    // vectors of a warp in half a turn, a multiple of 32
    bool stuck;       // a wait of this warp has run out
    __device__ __forceinline__ uint32_t turn() const { return 2u * kWarps * span; }
    __device__ __forceinline__ uint32_t first_of(uint32_t base, uint32_t h) const {
        return base + ((threadIdx.x >> 5) * 2u + h) * span;
    }
    __device__ __forceinline__ uint32_t number(uint32_t base, uint32_t u) const {
        return first_of(base, u / kHalf) + u % kHalf * 32u + lane_id();
    }
    // the thread's vectors of a half lie at 0, 32, 64 ... below this, counted from its first
    __device__ __forceinline__ int extent(uint32_t base, uint32_t h) const {
        const uint32_t first = first_of(base, h);
        return (int)min(span, count - min(first, count)) - (int)lane_id();
    }
    __device__ __forceinline__ uint4 fetch(uint32_t number) const {
        return __ldg(reinterpret_cast<const uint4 *>(body) + number);
    }
    __device__ __forceinline__ uint32_t column(uint32_t number) const { return head + number * kPer; }
    __device__ __forceinline__ uint4 *stage(const Params &p, uint32_t h) const {
        return stages(p) + ((threadIdx.x >> 5) * 2u + h) * kHalf * 32u;
    }
    // the warp asks for its vectors of half `h` of the turn at `base`
    __device__ __forceinline__ void ask(const Params &p, uint32_t base, uint32_t h) const {
        const uint32_t first = first_of(base, h);
        if (first >= count || stuck || lane_id() != 0) return;
        if (blockIdx.x == p.withhold_cta && threadIdx.x == 0 && base / turn() * 2u + h == p.withhold_issue) return;
        uint64_t *landed = &shared().landed[threadIdx.x >> 5][h];
        const uint32_t bytes = min(span, count - first) * 16u;
        mbarrier_expect(landed, bytes);
        bulk_copy_to_shared(stage(p, h), reinterpret_cast<const uint4 *>(body) + first, bytes, landed);
    }
    // ... and waits for them; false: there are none to look at.  A warp whose wait runs out sees what else
    // it has asked for land, waits no more and asks for nothing more: the row fails.
    __device__ __forceinline__ bool wait(const Params &p, uint32_t base, uint32_t h, uint32_t parity) {
        if (first_of(base, h) >= count || stuck) return false;
        uint64_t *landed = shared().landed[threadIdx.x >> 5];
        bool done = false;
        for (uint32_t polls = 0; polls < p.wait_polls && !done; polls++) done = mbarrier_try_wait(&landed[h], parity);
        if (__any_sync(kFullMask, !done)) {
            stuck = true;
            poke(&shared().lost, 1u);
            // (the other half: asked for in this turn if it is the second, in the next if the first)
            if (first_of(h == 0 ? base : base + turn(), 1u - h) < count)
                for (uint32_t polls = 0; polls < p.wait_polls; polls++)
                    if (mbarrier_try_wait(&landed[1u - h], h == 0 ? parity : parity ^ 1u)) break;
            return false;
        }
        return true;
    }
};

// The elements of the lanes' vectors (those in `mask`) that are worth the bound go on the list; returns those that
// found no place there.  All lanes call.
template <typename T>
__device__ __forceinline__ uint32_t list_elements(const float (&v)[Lanes<T>::kPer], uint32_t mask, uint32_t column, float floor,
                                                  uint64_t bound, bool greedy) {
    constexpr int kPer = Lanes<T>::kPer;
    Shared &sh = shared();
    const uint32_t lane = lane_id();
    const uint32_t odd = greedy ? sh.row.odd : 0u;
    uint32_t hits = 0, left = 0;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
        bool take = v[j] >= floor;
        if (greedy) take = take || odd_value(v[j], odd);
        hits |= (take ? 1u : 0u) << j;
    }
    hits &= mask;
    while (__any_sync(kFullMask, hits != 0)) {  // (as a rule a lane has one)
        const int j = hits != 0 ? __ffs(hits) - 1 : 0;
        Worth w = {0ull, 0.0f, false};
        if (hits != 0) {
            float x = v[0];
#pragma unroll
            for (int i = 1; i < kPer; i++) x = i == j ? v[i] : x;
            w = worth_of(x, column + (uint32_t)j, bound);
        }
        const uint32_t takers = __ballot_sync(kFullMask, w.key != 0);
        if (takers != 0) {
            uint32_t slot = 0;
            if (lane == 0) slot = atomicAdd(&sh.count, (uint32_t)__popc(takers));
            slot = __shfl_sync(kFullMask, slot, 0) + __popc(takers & ((1u << lane) - 1u));
            if (w.key != 0) {
                if (slot < kListCap) {
                    sh.key[slot] = w.key;
                    sh.value[slot] = w.value;
                    sh.column[slot] = column + (uint32_t)j;
                    if (w.waits) atomicOr(&sh.waiting[slot >> 5], 1u << (slot & 31u));
                } else {
                    left |= 1u << j;
                }
            }
        }
        hits &= hits - 1;
    }
    return left;
}

// Puts a vector into the queue; false when that is full.
__device__ __forceinline__ bool enqueue(Shared &sh, const uint4 &raw, uint32_t column, uint32_t mask) {
    const uint32_t slot = atomicAdd(&sh.queue_count, 1u);
    if (slot >= kQueueCap) return false;
    sh.queue.vector[slot] = raw;
    sh.queue.column[slot] = column;
    sh.queue.mask[slot] = (uint8_t)mask;
    return true;
}

// Elements (`left`) of a vector of every thread go on the list.  What finds no place waits until that has been
// cut and the bound lifted by what is left.  All threads call; ends synced.
template <typename T>
__device__ __forceinline__ void list_all(const uint4 raw, uint32_t left, uint32_t column) {
    constexpr int kPer = Lanes<T>::kPer;
    Shared &sh = shared();
    const Row &r = sh.row;
    float v[kPer];
    Lanes<T>::unpack(raw, v);
    bool hard = false;
    for (;;) {
        const Gate gate = gate_of(peek64(&sh.bound));
        left = list_elements<T>(v, left, column, gate.floor, gate.bound, r.greedy);
        if (!__syncthreads_or(left != 0)) break;
        tighten(hard);
        hard = true;  // (whatever the first cut has left: the next one makes room)
        uint32_t best = 0;
        if (left != 0) {
#pragma unroll
            for (int j = 0; j < kPer; j++)
                if (((left >> j) & 1u) && !is_nonfinite(v[j]) && !seen_column(r, column + (uint32_t)j))
                    best = max(best, float_key(v[j]));
        }
        const uint32_t key = tight_bound(best, r.k).x;
        if (threadIdx.x == 0 && key != 0) atomicMax(&sh.bound, (unsigned long long)key << 32);
        __syncthreads();
    }
}

// What is in the queue goes on the list.  All threads call; ends synced.
template <typename T>
__device__ __noinline__ void work_off() {
    Shared &sh = shared();
    const uint32_t tid = threadIdx.x;
    uint4 raw = make_uint4(0, 0, 0, 0);
    uint32_t column = 0, mask = 0;
    if (tid < min(sh.queue_count, kQueueCap)) {
        raw = sh.queue.vector[tid];
        column = sh.queue.column[tid];
        mask = sh.queue.mask[tid];
    }
    __syncthreads();
    if (tid == 0) sh.queue_count = 0;
    list_all<T>(raw, mask, column);
    if (__syncthreads_or(sh.count > kListLong)) tighten(false);
}

// Vectors of the turn at `base` (`pending`, a bit each) go into the queue if they are still worth a look; returns those
// that found it full.
template <typename T, int kHalf>
__device__ __noinline__ uint32_t refill(const Vectors<T, kHalf> vectors, uint32_t base, uint32_t pending) {
    constexpr int kPer = Lanes<T>::kPer;
    constexpr int kBatch = 4;  // vectors on their way at a time
    Shared &sh = shared();
    const Sieve sieve = sieve_of(gate_of(peek64(&sh.bound)));
    uint32_t left = 0;
#pragma unroll 1
    for (uint32_t rest = pending; rest != 0;) {
        if (peek(&sh.queue_count) >= kQueueCap) return left | rest;
        uint4 raw[kBatch];
        uint32_t bit[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            bit[q] = rest & (0u - rest);
            raw[q] = vectors.fetch(vectors.number(base, (uint32_t)__ffs(rest != 0 ? rest : pending) - 1u));
            rest &= rest - 1u;
        }
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            if (bit[q] == 0) continue;
            const uint32_t column = vectors.column(vectors.number(base, (uint32_t)__ffs(bit[q]) - 1u));
            float v[kPer];
            Lanes<T>::unpack(raw[q], v);
            if (!may_pass(v, column, sieve)) continue;
            const uint32_t mask = passing(v, column, sieve);
            if (mask != 0 && !enqueue(sh, raw[q], column, mask)) left |= bit[q];
        }
    }
    return left;
}

// More than the queue holds is worth a look (`pending`: vectors of the turn at `base`, a bit each): the queue is worked
// off, which lifts the bound, and filled with what still passes, until nothing is left.  After the first turn, whose
// bound comes from all its lanes' largest logits, and if far more than the queue holds was offered, those of the
// pending vectors lift it before that.  All threads call; ends synced.
template <typename T, int kHalf>
__device__ __noinline__ void crowded(const Vectors<T, kHalf> vectors, uint32_t base, uint32_t pending) {
    constexpr int kPer = Lanes<T>::kPer;
    constexpr int kBatch = 4;  // vectors on their way at a time
    Shared &sh = shared();
    if (base != 0 && peek(&sh.queue_count) > 2u * kQueueCap) {  // (what was offered; a few too many need no new bound)
        float best = __uint_as_float(0xff800000u);
#pragma unroll 1
        for (uint32_t rest = pending; rest != 0;) {
            uint4 raw[kBatch];
            uint32_t column[kBatch];
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                const uint32_t number = vectors.number(base, (uint32_t)__ffs(rest != 0 ? rest : pending) - 1u);
                raw[q] = vectors.fetch(number);
                column[q] = vectors.column(number);
                rest &= rest - 1u;
            }
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
                float v[kPer];
                Lanes<T>::unpack(raw[q], v);
                best = largest_unseen(v, column[q], best);
            }
        }
        const uint32_t key = tight_bound(is_nonfinite(best) ? 0u : float_key(best), sh.row.k).x;
        if (threadIdx.x == 0 && key != 0) atomicMax(&sh.bound, (unsigned long long)key << 32);
    }
    do {
        work_off<T>();
        if (pending != 0) pending = refill<T, kHalf>(vectors, base, pending);
    } while (__syncthreads_or(pending != 0));
}

// A warp's half of a turn in which most lanes have found something: what passes goes into the queue.  Returns the
// vectors that found it full, a bit each.  All lanes call.
template <typename T, int kHalf>
__device__ __noinline__ uint32_t sift(const uint4 *stage, uint32_t column, uint32_t hot, const Gate gate) {
    constexpr int kPer = Lanes<T>::kPer;
    const Sieve sieve = sieve_of(gate);
    uint32_t full = 0, rest = 0;
#pragma unroll
    for (uint32_t u = 0; u < (uint32_t)kHalf; u++) {
        float v[kPer];
        Lanes<T>::unpack(stage[u * 32u], v);
        if (((hot >> u) & 1u) && may_pass(v, column + u * 32u * kPer, sieve)) rest |= 1u << u;
    }
#pragma unroll 1
    for (; rest != 0; rest &= rest - 1) {
        const uint32_t u = (uint32_t)__ffs(rest) - 1u, at = column + u * 32u * kPer;
        const uint4 raw = stage[u * 32u];
        float v[kPer];
        Lanes<T>::unpack(raw, v);
        const uint32_t mask = passing(v, at, sieve);
        if (mask != 0 && !enqueue(shared(), raw, at, mask)) full |= 1u << u;
    }
    return full;
}

// The turns of the scan after the first.  The warps run freely; when the queue has become long all stop
// where they are, it is worked off, which lifts the bound, and they go on.
template <typename T, int kHalf, bool kGreedy>
__device__ __forceinline__ void scan(const Params &p, Vectors<T, kHalf> &vectors) {
    constexpr int kPer = Lanes<T>::kPer;
    constexpr uint32_t kTurn = 2u * kHalf * kThreads;  // (more than one turn: whole ones)
    Shared &sh = shared();
    const uint32_t odd = sh.row.odd;
    uint32_t base = kTurn, h = 0, parity = 1;
    for (;;) {
        uint32_t pending = 0;
        const Gate gate = gate_of(peek64(&sh.bound));
        const VectorGate look_at = gate_of_vectors(gate);
        bool stopped = false;  // with a half looked at
        while (vectors.first_of(base, h) < vectors.count && !__any_sync(kFullMask, peek(&sh.queue_count) > kQueueLong)) {
            if (!vectors.wait(p, base, h, parity)) {
                base = vectors.count;  // (the row fails)
                break;
            }
            const uint4 *stage = vectors.stage(p, h) + lane_id();
            const uint32_t first = vectors.number(base, h * kHalf);
            const int here = vectors.extent(base, h);
            const float at_least = vectors.column(vectors.first_of(base, h)) >= look_at.ties_lose ? look_at.above : look_at.at_least;
            uint32_t hot = 0;
#pragma unroll
            for (int u = 0; u < kHalf; u++) {
                float v[kPer];
                Lanes<T>::unpack(stage[u * 32], v);
                bool look = largest(v) >= at_least;
                if (kGreedy) look = look || odd_values(v, odd);
                hot |= (look && u * 32 < here ? 1u : 0u) << u;
            }
            const uint32_t finders = __ballot_sync(kFullMask, hot != 0);
            if (finders != 0) {
                if (__popc(finders) > 16 && __popc(__ballot_sync(kFullMask, (hot & (hot - 1u)) != 0)) > 16) {
                    // (most lanes have found several: not what a row as such has to offer)
                    pending |= sift<T, kHalf>(stage, vectors.column(first), hot, gate) << (h * kHalf);
                } else {
#pragma unroll 1
                    for (; hot != 0; hot &= hot - 1) {
                        const uint32_t u = (uint32_t)__ffs(hot) - 1u;
                        if (!enqueue(sh, stage[u * 32u], vectors.column(first + u * 32u), (1u << kPer) - 1u))
                            pending |= 1u << (h * kHalf + u);
                    }
                }
                __syncwarp();
                stopped = __any_sync(kFullMask, pending != 0);
            }
            vectors.ask(p, base + kTurn, h);
            if (stopped) break;
            if (h != 0) {
                base += kTurn;
                parity ^= 1u;
            }
            h ^= 1u;
        }
        if (!__syncthreads_or(pending != 0 || vectors.first_of(base, h) < vectors.count)) return;
        crowded<T, kHalf>(vectors, base, pending);
        if (stopped) {
            if (h != 0) {
                base += kTurn;
                parity ^= 1u;
            }
            h ^= 1u;
        }
    }
}

// The k best of the lists in the inbox, in order, into the finish buffer.  A warp has a list, which is in
// order.  An entry's place is its own in there and the number of larger ones in every other list, found by
// binary searches side by side (behind a list's last entry lie zeros, which nothing is smaller than).
// All threads call; ends synced.
template <uint32_t kLists>
__device__ __forceinline__ void merge_lists(uint32_t k) {
    static_assert(kLists <= kMostTeam && kLists <= (uint32_t)kWarps, "a warp per list");
    Shared &sh = shared();
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t count = warp < kLists ? sh.inbox_count[warp] : 0u;
    if (warp < kLists) {
#pragma unroll
        for (uint32_t i = lane; i < (uint32_t)kMaxK; i += 32)
            sh.order[warp * kMaxK + i] = i < count ? select_key(sh.inbox_score[warp][i], sh.inbox_id[warp][i]) : 0ull;
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t i = lane; i < count; i += 32) {
        const uint64_t own = sh.order[warp * kMaxK + i];
        uint32_t larger[kLists], place = i;
#pragma unroll
        for (uint32_t o = 0; o < kLists; o++) larger[o] = o * kMaxK;
#pragma unroll
        for (uint32_t step = kMaxK / 2; step != 0; step /= 2) {
            if (step >= 2u * k) continue;  // (no list is that long)
            uint64_t other[kLists];
#pragma unroll
            for (uint32_t o = 0; o < kLists; o++) other[o] = sh.order[larger[o] + step - 1u];
#pragma unroll
            for (uint32_t o = 0; o < kLists; o++) larger[o] += other[o] > own ? step : 0u;
        }
#pragma unroll
        for (uint32_t o = 0; o < kLists; o++) {
            larger[o] += sh.order[larger[o]] > own ? 1u : 0u;
            place += o != warp ? larger[o] - o * kMaxK : 0u;
        }
        if (place < k) {
            sh.fin.score[place] = sh.inbox_score[warp][i];
            sh.fin.id[place] = sh.inbox_id[warp][i];
        }
    }
    __syncthreads();
}

// The CTA's k best, in order, go to the team's first CTA, which ends the row.  All threads call, with the
// list complete, synced.
__device__ __forceinline__ void conclude(const Params &p, uint32_t row, uint32_t rank) {
    Shared &sh = shared();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, team = p.team;
    const uint32_t k = sh.row.k, first_id = sh.row.id_base;
    float uniform = 0.0f;  // (on its way meanwhile; rows that draw nothing may not have one)
    if (rank == 0 && warp == 0 && p.shard_k == 0 && !sh.row.greedy) uniform = __ldg(&p.uniforms[row]);
    const uint32_t total = min(sh.count, kListCap);
    if (sh.row.with_counts && sh.row.counts == nullptr) settle(true);
    const uint64_t mine = tid < total ? sh.key[tid] : 0ull;  // (a thread's own entry)
    sh.order[tid] = mine;
    sh.rank[tid] = 0;
    const uint32_t alive = __syncthreads_count(mine != 0);
    rank_entries(sh, total);
    if (team > 1) team_wait(team);  // the first CTA has begun
    if (mine != 0) {
        const uint32_t place = sh.rank[tid];
        if (place < k) {
            *in_first_cta(&sh.inbox_score[rank][place], team) = sh.value[tid];
            *in_first_cta(&sh.inbox_id[rank][place], team) = first_id + sh.column[tid];
        }
    }
    if (tid == 0) {
        *in_first_cta(&sh.inbox_count[rank], team) = min(alive, k);
        *in_first_cta(&sh.inbox_wild[rank], team) = sh.wild;
        *in_first_cta(&sh.inbox_bad[rank], team) = sh.lost ? kErrLimit : sh.bad_history;
        if (sh.lost) atomicMin(p.out.first_error + 1, 1ull);  // the cause, for the host's message
    }
    team_arrive(team);
    team_wait(team);
    if (rank != 0) return;

    // ---- the first CTA: the k best of all of them in order (one candidate: the largest of the lists' first) ----
    if (k > 1u) {
        if (team == 8u) merge_lists<8>(k);
        else if (team == 4u) merge_lists<4>(k);
        else if (team == 2u) merge_lists<2>(k);
    }
    if (warp != 0) return;
    unsigned long long wild = ~0ull;  // the padding id when nothing was seen
    uint32_t entries = 0, bad = 0;
    if (lane < team) {
        entries = sh.inbox_count[lane];
        wild = sh.inbox_wild[lane];
        bad = sh.inbox_bad[lane];
    }
    RowResult result;
    result.kept = min(__reduce_add_sync(kFullMask, entries), k);
    result.bad_history = __reduce_max_sync(kFullMask, bad);
    result.wild_id = __reduce_min_sync(kFullMask, (uint32_t)(wild >> 32));
    const unsigned owner = __ballot_sync(kFullMask, (uint32_t)(wild >> 32) == result.wild_id);
    result.wild_bits = __shfl_sync(kFullMask, (uint32_t)wild, __ffs(owner) - 1);
    if (k == 1u) {
        const uint64_t own = entries != 0 ? select_key(sh.inbox_score[lane][0], sh.inbox_id[lane][0]) : 0ull;
        const uint32_t high = __reduce_max_sync(kFullMask, (uint32_t)(own >> 32));
        const uint32_t low = __reduce_max_sync(kFullMask, (uint32_t)(own >> 32) == high ? (uint32_t)own : 0u);
        if (own != 0 && (uint32_t)(own >> 32) == high && (uint32_t)own == low) {
            sh.fin.score[0] = sh.inbox_score[lane][0];
            sh.fin.id[0] = sh.inbox_id[lane][0];
        }
    } else if (team == 1) {
        for (uint32_t i = lane; i < result.kept; i += 32) {
            sh.fin.score[i] = sh.inbox_score[0][i];
            sh.fin.id[i] = sh.inbox_id[0][i];
        }
    }
    __syncwarp();
    const SamplerConfig *configs = p.configs;
    asm volatile("" : "+l"(configs));  // (read once more: nobody has to keep them)
    const SamplerConfig cfg = p.config_count > 1 ? configs[row] : p.config0;
    finish_row(p, sh.fin, result, k, sh.row.greedy, cfg, uniform, row);
}

template <typename T, int kHalf>
__global__ void __launch_bounds__(kThreads, 2) team_select_kernel(const __grid_constant__ Params p) {
    constexpr int kPer = Lanes<T>::kPer;
    constexpr int kTokens = 16;  // tokens per thread and trip, loaded before any is used
    Shared &sh = shared();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t team = p.team, row = team == 1 ? blockIdx.x : blockIdx.x / team, rank = blockIdx.x - row * team;
    const SamplerConfig cfg = p.config_count > 1 ? p.configs[row] : p.config0;
    // (the whole team leaves, or none of it)
    const bool raises = can_raise(cfg);
    if ((p.shard_k == 0 && cfg.temperature != 0.0f && cfg.top_k == 0) ||
        (p.which != kAllRows && (p.which == kRaisingRows) != raises)) {
        clear_next_error(p.out);
        return;
    }
    // the logits
    const uint32_t lo = min(p.vocab, rank * p.chunk), n = min(p.chunk, p.vocab - lo);
    const T *columns = static_cast<const T *>(p.logits) + (size_t)row * p.row_stride + lo;
    const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(columns) & 15u);
    Vectors<T, kHalf> vectors;
    vectors.head = min(n, (off ? 16u - off : 0u) / (uint32_t)sizeof(T));
    vectors.count = (n - vectors.head) / kPer;
    vectors.body = columns + vectors.head;
    vectors.span = 32u * min((uint32_t)kHalf, max(1u, (vectors.count + 2u * kThreads - 1u) / (2u * kThreads)));
    vectors.stuck = false;
    if (lane == 0) {
        mbarrier_init(&sh.landed[warp][0], 1);
        mbarrier_init(&sh.landed[warp][1], 1);
        mbarrier_fence_init();
    }
    __syncwarp();
    vectors.ask(p, 0, 0);
    vectors.ask(p, 0, 1);
    if (team > 1) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    clear_next_error(p.out);
    // the row's history
    const bool penalised = penalties_active(cfg);
    const bool listed = p.history_tokens != nullptr && p.bitmap_words != 0 && penalised;
    const bool tabled = p.slot_counts != nullptr && penalised;
    uint32_t session = 0;
    if (tabled) session = __ldg(&p.row_slots[row]);
    uint64_t begin = 0, end = 0;
    if (listed) {
        begin = __ldg(&p.history_offsets[row]);
        end = __ldg(&p.history_offsets[row + 1]);
    }
    const uint32_t first_id = p.vocab_offset + lo;
    if (tid == 32) {
        sh.bad_history = 0;
        sh.lost = 0;
        sh.wild = ~0ull;
        sh.bound = 0;
        sh.count = sh.queue_count = 0;
    }
    if (tid < kListCap / 32) sh.waiting[tid] = 0;
    uint32_t *bitmap = seen_bitmap();
    if (listed) {
        uint4 *words = reinterpret_cast<uint4 *>(bitmap);
        for (uint32_t i = tid; i < p.bitmap_words / 4u; i += kThreads) words[i] = make_uint4(0, 0, 0, 0);
    } else if (tabled) {
        // (the session keeps its bitmap: `lo` is a multiple of 128, a session's words one of 4)
        const uint4 *kept = reinterpret_cast<const uint4 *>(p.slot_bitmaps + (size_t)session * p.slot_bitmap_words + (lo >> 5));
        uint4 *words = reinterpret_cast<uint4 *>(bitmap);
        for (uint32_t i = tid; i < (n + 127u) / 128u; i += kThreads) words[i] = __ldg(&kept[i]);
    }
    const bool too_long = end < begin || end - begin > p.history_max;
    const uint32_t length = listed && !too_long ? (uint32_t)(end - begin) : 0u;
    const uint32_t *tokens = p.history_tokens + begin;
    uint32_t token[kTokens];
    if (length != 0) {
#pragma unroll
        for (int q = 0; q < kTokens; q++) {
            const uint32_t at = (uint32_t)q * kThreads + tid;
            token[q] = at < length ? __ldg(&tokens[at]) : 0u;
        }
    }
    const bool greedy = cfg.temperature == 0.0f;
    const uint32_t k = p.shard_k != 0 ? p.shard_k : (greedy ? 1u : cfg.top_k);
    if (tid == 64) {
        Row &r = sh.row;
        r.greedy = greedy;
        r.k = k;
        r.id_base = first_id;
        r.columns = n;
        r.flat_offset = penalty_offset(1u, cfg.presence_penalty, cfg.frequency_penalty);
        r.presence = cfg.presence_penalty;
        r.frequency = cfg.frequency_penalty;
        r.repetition = cfg.repetition_penalty;
        r.raises = raises;
        r.odd = cfg.repetition_penalty != 1.0f && (length != 0 || tabled) ? kHugeBits : 0x7f800000u;
        r.tokens = tokens;
        r.counts = tabled ? p.slot_counts + (size_t)session * p.vocab_total + lo : nullptr;
        r.history_len = length;
        r.seen_any = length != 0 || r.counts != nullptr;
        r.with_counts = r.seen_any && cfg.frequency_penalty != 0.0f;
    }
    __syncthreads();
    if (tid == 0) {
        // the host sends only rows whose charge grows with the count; a row that slipped through
        // is failed rather than sampled wrongly
        const bool ours = !sh.row.seen_any || (cfg.frequency_penalty >= 0.0f && cfg.repetition_penalty >= 0x1p-40f &&
                                               cfg.repetition_penalty <= 0x1p40f);
        if (listed && too_long) atomicMax(&sh.bad_history, kErrLimit);
        else if (!ours) atomicMax(&sh.bad_history, kErrArgument);
    }

    // ---- the history's bitmap, while the logits are on their way ----
    if (length != 0) {
        for (uint32_t base = 0;;) {
#pragma unroll
            for (int q = 0; q < kTokens; q++) {
                if (base + (uint32_t)q * kThreads + tid >= length) continue;
                if (token[q] >= p.vocab_total) atomicMax(&sh.bad_history, kErrFormat);
                const uint32_t local = token[q] - first_id;  // wraps for ids below the CTA's columns
                if (local < n) {
                    const uint32_t bit = 1u << (local & 31u);
                    if ((bitmap[local >> 5] & bit) == 0) atomicOr(&bitmap[local >> 5], bit);
                }
            }
            base += kTokens * kThreads;
            if (base >= length) break;
#pragma unroll
            for (int q = 0; q < kTokens; q++) {
                const uint32_t at = base + (uint32_t)q * kThreads + tid;
                token[q] = at < length ? __ldg(&tokens[at]) : 0u;
            }
        }
        __syncthreads();
    }

    // ---- the first turn: every thread's largest, and the bound ----
    const float none = __uint_as_float(0xff800000u);
    float most[2 * kHalf];  // the thread's vectors' largest values
    uint32_t odd = 0;
    const uint32_t odd_from = sh.row.odd;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const bool landed = vectors.wait(p, 0, h, 0);
        const uint4 *stage = vectors.stage(p, h) + lane;
        const int here = landed ? vectors.extent(0, h) : 0;
#pragma unroll
        for (int u = 0; u < kHalf; u++) {
            float v[kPer];
            Lanes<T>::unpack(stage[u * 32], v);
            const bool there = u * 32 < here;
            most[h * kHalf + u] = there ? largest(v) : none;  // (a NaN never wins)
            if (greedy && there && odd_values(v, odd_from)) odd |= 1u << (h * kHalf + u);
        }
        __syncwarp();
        if (landed) vectors.ask(p, vectors.turn(), h);
    }
    const float best = largest(most);
    // a vector of the turn: from where it landed, or, if what follows has been asked for over it, once more
    const bool one_turn = vectors.count <= vectors.turn();
    auto vector_of = [&](uint32_t u) {
        return one_turn ? vectors.stage(p, 0)[u * 32u + lane] : vectors.fetch(vectors.number(0, u));  // (the halves' stages adjoin)
    };
    uint32_t key = 0;
    if (!is_nonfinite(best)) {
        key = float_key(best);
        if (sh.row.seen_any) {
            uint32_t where = 0, j = 0;
#pragma unroll
            for (int u = 2 * kHalf - 1; u >= 0; u--) where = most[u] == best ? (uint32_t)u : where;
            float v[kPer];
            Lanes<T>::unpack(vector_of(where), v);
#pragma unroll
            for (int e = kPer - 1; e >= 0; e--)
                if (v[e] == best) j = e;
            if (seen_column(sh.row, vectors.column(vectors.number(0, where)) + j)) key = 0;
        }
    }
    // Where the history has seen so many of the best that the warp's j-th largest key (j = ceil(k / warps)) would lie
    // low, the lanes' largest unseen ones are looked for.  (Rows that it covers so densely are short.)
    if (one_turn && sh.row.seen_any && 2u * __popc(__ballot_sync(kFullMask, key != 0)) < 5u * ((k + kWarps - 1u) / kWarps)) {
        if (key == 0 && best > none) {
            float unseen = none;
#pragma unroll 1
            for (uint32_t u = 0; u < 2u * kHalf; u++) {
                if ((int)(u % kHalf * 32u) >= vectors.extent(0, u / kHalf)) continue;
                float v[kPer];
                Lanes<T>::unpack(vector_of(u), v);
                unseen = largest_unseen(v, vectors.column(vectors.number(0, u)), unseen);
            }
            key = is_nonfinite(unseen) ? 0u : float_key(unseen);
        }
    }
    // (a last warp with less than half a warp's vectors has too few keys to bound the others)
    const uint32_t warps = max(1u, min((uint32_t)kWarps, (vectors.count + vectors.span) / (2u * vectors.span)));
    const bool tight = k > 1u && (!one_turn || (k > kLooseMost && warps == (uint32_t)kWarps));  // (fewer warps have too few keys)
    const uint2 first_bound = tight ? tight_bound(key, k) : loose_bound(key, k, warps);
    uint32_t low = first_bound.x;
    if (k == 1u) {
        low = first_bound.y;
    } else if (!tight && !(key_to_float(first_bound.y) - key_to_float(low) < kFarApart)) {
        __syncthreads();  // (everybody has read what the second bound is made over)
        low = max(low, tight_bound(key, k).x);
    }
    const uint64_t bound = (uint64_t)low << 32;
    if (tid == 0) sh.bound = bound;
    const Gate gate = gate_of(bound);
    // the columns before the first boundary and after the last: one for some threads of two warps
    const uint32_t tail = vectors.column(vectors.count);
    if (vectors.head != 0 || tail < n) {
        uint32_t single = kPaddingId;
        if (tid < vectors.head) single = tid;
        if (tid >= 32u && tail + (tid - 32u) < n) single = tail + (tid - 32u);
        if (single != kPaddingId) {
            const float x = sizeof(T) == 2 ? bf16_bits_to_float((uint32_t)__ldg(columns + single)) : (float)__ldg(columns + single);
            if (x >= gate.floor || (greedy && odd_value(x, sh.row.odd))) {
                const Worth w = worth_of(x, single, bound);
                if (w.key != 0) {
                    const uint32_t slot = atomicAdd(&sh.count, 1u);
                    sh.key[slot] = w.key;
                    sh.value[slot] = w.value;
                    sh.column[slot] = single;
                    if (w.waits) atomicOr(&sh.waiting[slot >> 5], 1u << (slot & 31u));
                }
            }
        }
        __syncthreads();  // (these find the list empty: they have a place)
    }
    {
        // (what finds the list full is for the queue: elements of one vector, which has room there, and the
        // vectors after it)
        uint32_t hot = odd, part = 0, part_of = 0;
#pragma unroll
        for (int u = 0; u < 2 * kHalf; u++) hot |= (most[u] >= gate.floor && most[u] > none ? 1u : 0u) << u;
        // (a flood is not what a row as such has to offer: left to `crowded`, which sifts it)
        const bool flood = __any_sync(kFullMask, odd != 0 || __popc(hot) > kHalf);
        while (!flood && __any_sync(kFullMask, hot != 0) && !__any_sync(kFullMask, part != 0)) {
            part_of = hot != 0 ? (uint32_t)__ffs(hot) - 1u : 0u;
            float v[kPer] = {};
            if (hot != 0) Lanes<T>::unpack(vector_of(part_of), v);
            part = list_elements<T>(v, hot != 0 ? (1u << kPer) - 1u : 0u, vectors.column(vectors.number(0, part_of)), gate.floor, bound,
                                    greedy);
            hot &= hot - 1u;
        }
        if (part != 0) enqueue(sh, vector_of(part_of), vectors.column(vectors.number(0, part_of)), part);
        if (__syncthreads_or(hot != 0 || part != 0)) crowded<T, kHalf>(vectors, 0, hot);
    }

    // ---- the rest ----
    if (!one_turn) {
        if (greedy) scan<T, kHalf, true>(p, vectors);
        else scan<T, kHalf, false>(p, vectors);
    }
    if (sh.queue_count != 0) work_off<T>();
    conclude(p, row, rank);
}

}  // namespace team
}  // namespace fgk

// ------------------------------------------------------------------ host side

using namespace fgk;

// The forms of the kernel: 8 or 10 vectors that a thread asks for at a time, twice.  (Three CTAs to an SM, with 4
// and 80 registers a thread, spill and are slower throughout: 148 rows of 151,936 fp32 logits 41 us
// against 25, 1024 rows 148 against 129.)
static const void *team_kernel(uint32_t dtype, uint32_t form) {
    if (dtype == 1u)
        return form == 1u ? reinterpret_cast<const void *>(team::team_select_kernel<uint16_t, 10>)
                          : reinterpret_cast<const void *>(team::team_select_kernel<uint16_t, 8>);
    return form == 1u ? reinterpret_cast<const void *>(team::team_select_kernel<float, 10>)
                      : reinterpret_cast<const void *>(team::team_select_kernel<float, 8>);
}

static constexpr size_t kTeamShared = 112u * 1024u;  // two CTAs to an SM
static uint32_t team_vectors(uint32_t form) { return (form == 1u ? 20u : 16u) * team::kThreads; }
static size_t team_dynamic(uint32_t form, uint32_t bitmap_words) {
    return sizeof(team::Shared) + (size_t)team_vectors(form) * 16u + (size_t)bitmap_words * 4u;
}

extern "C" int fgk_team_fits(uint32_t form, uint32_t bitmap_words) {
    return form < FGK_TEAM_FORMS && team_dynamic(form, bitmap_words) <= kTeamShared;
}

extern "C" uint32_t fgk_team_turn(uint32_t dtype, uint32_t form) { return team_vectors(form) * (dtype == 1u ? 8u : 4u); }

extern "C" int fgk_team_prepare(void) {
    for (uint32_t i = 0; i < 2u * FGK_TEAM_FORMS; i++) {
        const void *kernel = team_kernel(i & 1u, i / 2u);
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTeamShared);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return (int)e;
    }
    return (int)cudaSuccess;
}

extern "C" int fgk_launch_team_select(const fgk_stream_launch *l, uint32_t team_size, uint32_t chunk, uint32_t form,
                                      uint32_t which, void *stream) {
    if (team_size == 0 || team_size > team::kMostTeam || (team_size & (team_size - 1u)) != 0 || chunk % 128u != 0 ||
        (uint64_t)team_size * chunk < l->vocab || !fgk_team_fits(form, l->bitmap_words))
        return (int)cudaErrorInvalidValue;
    team::Params p;
    memset(&p, 0, sizeof(p));
    p.logits = l->logits;
    p.row_stride = l->row_stride;
    p.rows = l->rows;
    p.vocab = l->vocab;
    p.vocab_offset = l->vocab_offset;
    p.vocab_total = l->vocab_total;
    p.team = team_size;
    p.chunk = chunk;
    p.which = which;
    p.history_tokens = l->history_tokens;
    p.history_offsets = l->history_offsets;
    p.history_max = l->history_max;
    p.bitmap_words = l->bitmap_words;
    p.configs = static_cast<const SamplerConfig *>(l->configs_device);
    static_assert(sizeof(fg_sampler_config) == sizeof(SamplerConfig), "config layout");
    memcpy(&p.config0, &l->config0, sizeof(SamplerConfig));
    p.config_count = l->config_count;
    p.shard_k = l->shard_k;
    p.uniforms = l->uniforms;
    p.shard_scores = l->shard_scores;
    p.shard_ids = l->shard_ids;
    p.shard_stride = l->shard_stride ? l->shard_stride : 1u;
    for (int t = 0; t < 16; t++) p.push.window[t] = static_cast<unsigned char *>(l->push.window[t]);
    p.push.ranks = l->push.ranks;
    p.push.rank = l->push.rank;
    p.push.half = l->push.half;
    p.push.pair_capacity = l->push.pair_capacity;
    p.push.row_capacity = l->push.row_capacity;
    p.slot_counts = l->slot_counts;
    p.slot_bitmaps = l->slot_bitmaps;
    p.row_slots = l->row_slots;
    p.slot_bitmap_words = l->slot_bitmap_words;
    p.wait_polls = l->wait_polls ? l->wait_polls : team::kDefaultPolls;
    p.withhold_cta = l->withhold_armed ? l->withhold_cta : 0xffffffffu;
    p.withhold_issue = l->withhold_issue;
    p.out.tokens = l->out.tokens;
    p.out.token_logits = l->out.token_logits;
    p.out.row_status = l->out.row_status;
    p.out.first_error = reinterpret_cast<unsigned long long *>(l->out.first_error);
    p.out.next_error = reinterpret_cast<unsigned long long *>(l->out.next_error);
    p.out.noted = l->out.noted;
    p.out.dbg_count = l->out.dbg_count;
    p.out.dbg_ids = l->out.dbg_ids;
    p.out.dbg_scores = l->out.dbg_scores;
    p.out.dbg_raw = l->out.dbg_raw;
    p.out.dbg_tempered = l->out.dbg_tempered;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = team_size;
    cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(l->rows * team_size);
    config.blockDim = dim3(team::kThreads);
    config.dynamicSmemBytes = team_dynamic(form, l->bitmap_words);
    config.stream = static_cast<cudaStream_t>(stream);
    config.attrs = &cluster;
    config.numAttrs = 1;
    void *arguments[] = {&p};
    const cudaError_t e = cudaLaunchKernelExC(&config, team_kernel(l->dtype, form), arguments);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}
