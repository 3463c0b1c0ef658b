// Block-level exact selection and the final sampling arithmetic.
//
//  * CandidateBuffer   shared-memory list of (score, id) pairs a CTA collects
//                      while it streams a row.
//  * compact_topk      MSB-first radix select (8-bit digits over the 64-bit
//                      (score, ~id) key) that keeps exactly the k best entries;
//                      the reference does the same job per 1024-tile in
//                      shaders/fg_topk_select.comp:51-77 with 5/6-bit digits.
//  * sort_candidates   rank-by-counting sort of <= 64 survivors into sampling
//                      order (src/sampler.c:88-96 does it by insertion).
//  * finish_select     the select step of src/sampler.c:97-121 with the same
//                      fp64 operations in the same left-to-right order; only
//                      the exp() calls are spread over the lanes of a warp.
#pragma once

#include "fg_device_common.cuh"

namespace fgk {

template <int CAP>
struct CandidateBuffer {
    float score[CAP];
    uint32_t id[CAP];
    uint32_t hist[256];
    unsigned long long min_key;
    uint32_t count;      // slots handed out (may run past CAP; stores beyond CAP are dropped)
    uint32_t out_count;
    uint32_t eq_count;
    uint32_t sel_digit, sel_need, sel_bucket;
    float tau_score;     // current lower bound: k-th best (score, id) seen so far
    uint32_t tau_id;
};

// Sorted survivors and the select step's work arrays.
struct FinishBuffer {
    float score[kMaxK];
    uint32_t id[kMaxK];
    double raw[kMaxK];
    double tempered[kMaxK];
};

// How the threads that share a candidate list meet: the whole CTA by default; a
// kernel whose CTA also holds warps with another job passes a named barrier instead.
struct WholeBlock {
    static __device__ __forceinline__ void sync() { __syncthreads(); }
};

// Keeps the k best of buf[0..n) (n <= CAP) at buf[0..k) in unspecified order,
// sets buf.tau_* to the k-th best and returns the new count.  All THREADS
// threads that meet at Bar (numbered 0 .. THREADS-1 by threadIdx.x) must call it
// with the same n and k.  n <= k is a no-op.
template <int THREADS, int CAP, class Bar = WholeBlock>
__device__ uint32_t compact_topk(CandidateBuffer<CAP> &buf, uint32_t n, uint32_t k) {
    static_assert(CAP % THREADS == 0, "buffer is a whole number of entries per thread");
    constexpr int PER = CAP / THREADS;
    if (n <= k) return n;
    const uint32_t tid = threadIdx.x;
    uint64_t key[PER];
    float score[PER];
    uint32_t id[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const uint32_t at = j * THREADS + tid;
        key[j] = 0;
        score[j] = 0.0f;
        id[j] = kPaddingId;
        if (at < n) {
            score[j] = buf.score[at];
            id[j] = buf.id[at];
            key[j] = select_key(score[j], id[j]);
        }
    }
    uint64_t prefix = 0;
    uint32_t need = k, bucket = 0;
    int shift = 56;
    for (int pass = 0; pass < 8; pass++) {
        if (tid < 256) buf.hist[tid] = 0;
        Bar::sync();
#pragma unroll
        for (int j = 0; j < PER; j++) {
            if (key[j] != 0 && (pass == 0 || (key[j] >> (shift + 8)) == prefix))
                atomicAdd(&buf.hist[(key[j] >> shift) & 255u], 1u);
        }
        Bar::sync();
        if (tid < 32) {
            // lane l owns digits 255-8l .. 248-8l, walked from the top
            uint32_t mine = 0;
#pragma unroll
            for (int b = 0; b < 8; b++) mine += buf.hist[255 - 8 * tid - b];
            uint32_t incl = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t up = __shfl_up_sync(kFullMask, incl, d);
                if (tid >= (uint32_t)d) incl += up;
            }
            const unsigned reached = __ballot_sync(kFullMask, incl >= need);
            const int owner = __ffs(reached) - 1;  // need <= total, so some lane reaches it
            if ((int)tid == owner) {
                uint32_t above = incl - mine;
                for (int b = 0; b < 8; b++) {
                    const uint32_t digit = 255 - 8 * tid - b;
                    const uint32_t here = buf.hist[digit];
                    if (above + here >= need) {
                        buf.sel_digit = digit;
                        buf.sel_need = need - above;
                        buf.sel_bucket = here;
                        break;
                    }
                    above += here;
                }
            }
        }
        Bar::sync();
        prefix = (prefix << 8) | buf.sel_digit;
        need = buf.sel_need;
        bucket = buf.sel_bucket;
        if (bucket == need || shift == 0) break;
        shift -= 8;
    }
    if (tid == 0) {
        buf.out_count = 0;
        buf.eq_count = 0;
        buf.min_key = ~0ull;
    }
    Bar::sync();
#pragma unroll
    for (int j = 0; j < PER; j++) {
        if (key[j] == 0) continue;
        const uint64_t high = key[j] >> shift;
        bool take = high > prefix;
        if (!take && high == prefix) take = bucket == need || atomicAdd(&buf.eq_count, 1u) < need;
        if (take) {
            const uint32_t slot = atomicAdd(&buf.out_count, 1u);
            buf.score[slot] = score[j];
            buf.id[slot] = id[j];
            atomicMin(&buf.min_key, (unsigned long long)key[j]);
        }
    }
    Bar::sync();
    if (tid == 0) {
        buf.tau_score = key_to_float((uint32_t)(buf.min_key >> 32));
        buf.tau_id = ~(uint32_t)(buf.min_key & 0xffffffffull);
        buf.count = buf.out_count;
    }
    Bar::sync();
    return buf.out_count;
}

// buf[0..n), n <= 64, into fin.score/id in sampling order.  Entries that compare
// equal on (score, id) keep their buffer order.  All threads call; ends synced.
template <int CAP, class Bar = WholeBlock>
__device__ void sort_candidates(const CandidateBuffer<CAP> &buf, FinishBuffer &fin, uint32_t n) {
    const uint32_t tid = threadIdx.x;
    if (tid < n) {
        const float s = buf.score[tid];
        const uint32_t id = buf.id[tid];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < n; j++) {
            const float t = buf.score[j];
            const uint32_t tj = buf.id[j];
            if (precedes(t, tj, s, id) || (t == s && tj == id && j < tid)) rank++;
        }
        fin.score[rank] = s;
        fin.id[rank] = id;
    }
    Bar::sync();
}

// The fused exchange of the vocabulary-sharded mode, device side (layout: fg_kernels.h).
struct PushTargets {
    unsigned char *window[16];
    uint32_t ranks, rank, half, pair_capacity, row_capacity;

    // where this rank's pair i of `row` lands in rank t's window
    __device__ __forceinline__ uint2 *pair(uint32_t t, uint32_t row, uint32_t k, uint32_t i) const {
        uint2 *pairs = reinterpret_cast<uint2 *>(window[t]);
        return pairs + ((size_t)half * ranks + rank) * pair_capacity + (size_t)row * k + i;
    }
    __device__ __forceinline__ uint32_t *arrived(uint32_t t, uint32_t row) const {
        uint32_t *counters = reinterpret_cast<uint32_t *>(
            window[t] + (size_t)2 * ranks * pair_capacity * sizeof(uint2));
        return counters + (size_t)half * row_capacity + row;
    }
};

struct SelectOutput {
    uint32_t *tokens;
    float *token_logits;
    uint32_t *row_status;
    unsigned long long *first_error;  // [0]: min over failing rows of (row << 8 | status), [1]: 1 when a wait ran out
    unsigned long long *next_error;   // the next call's two words, set to "none" here (may be null)
    uint32_t *noted;                  // host word: some row failed (may be null)
    uint32_t *dbg_count;
    uint32_t *dbg_ids;
    float *dbg_scores;
    double *dbg_raw;
    double *dbg_tempered;
};

// A row failed: the smallest one's number and status stay in the device's words, and the host,
// which looks at them only then, is told.
__device__ __forceinline__ void note_error(const SelectOutput &out, uint32_t row, uint32_t status) {
    atomicMin(out.first_error, ((unsigned long long)row << 8) | (unsigned long long)status);
    if (out.noted != nullptr) *reinterpret_cast<volatile uint32_t *>(out.noted) = 1u;
}

// Calls use two pairs of error words in turn: the first block of every kernel clears the pair that
// the call after this one will use (its last user has finished: calls are ordered by their stream).
__device__ __forceinline__ void clear_next_error(const SelectOutput &out) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && out.next_error != nullptr) {
        out.next_error[0] = ~0ull;
        out.next_error[1] = ~0ull;
    }
}

__device__ __forceinline__ void report_row(const SelectOutput &out, uint32_t row, uint32_t status,
                                           uint32_t token, float logit) {
    out.tokens[row] = token;
    out.token_logits[row] = logit;
    out.row_status[row] = status;
    if (status != kOk) note_error(out, row, status);
}

// x[i] becomes x[0] + ... + x[i], added from the left with one rounding per addition, as the C
// loops of src/sampler.c:99-111 do; the loads of four terms go ahead of their additions.  Returns
// the sum of all n.  With `limit` it stops soon after a sum that has reached it: later places keep
// their terms.
__device__ __forceinline__ double running_sums(double *x, uint32_t n, const double *limit = nullptr) {
    double sum = 0.0;
    uint32_t i = 0;
    for (; i + 4 <= n; i += 4) {
        const double a = x[i], b = x[i + 1], c = x[i + 2], d = x[i + 3];
        const double s0 = sum + a, s1 = s0 + b, s2 = s1 + c;
        sum = s2 + d;
        x[i] = s0;
        x[i + 1] = s1;
        x[i + 2] = s2;
        x[i + 3] = sum;
        if (limit != nullptr && sum >= *limit) return sum;
    }
    for (; i < n; i++) {
        sum += x[i];
        x[i] = sum;
    }
    return sum;
}

// Inclusive sums over the lanes' terms of up to 64 places (the second 32 only if `two`).
__device__ __forceinline__ void scan_places(double &low, double &high, bool two) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double up = __shfl_up_sync(kFullMask, low, d);
        low += lane >= (uint32_t)d ? up : 0.0;
        if (two) {
            const double up_high = __shfl_up_sync(kFullMask, high, d);
            high += lane >= (uint32_t)d ? up_high : 0.0;
        }
    }
    high += __shfl_sync(kFullMask, low, 31);
}

// Final step for one row; called by one warp of the CTA (all 32 lanes) with the
// candidates already in sampling order in fin.score/id[0..n), n = min(top_k,
// #finite).  Greedy rows never come here.
//
// What bounds it: chains of fp64 operations, 30 cycles each; in the reference's order n additions for
// the raw weights' sum and n more for the quotients' (the tempered weights' running sums are made
// beside the first).  But those sums decide no more than where one of them passes top_p and where the
// draw lands.  So they are first made by a scan over the lanes, and only if one of the two edges lies
// within 1e-13 (of the total) of a sum -- the two ways of adding 64 positive terms differ by 2e-14 at
// most, see below -- or if the quotients are asked for, the chains decide.  (2.2 thousand cycles for 20
// candidates instead of 3.1, 2.9 instead of 4.6 for 50; 256 rows of a shard and their merge 37.4 us before,
// 35.5 now, 1024 rows of 151,936 the same within noise.)  A top_p that keeps all n does not ask for the
// chains: with k = 64, 512 bf16 rows of 151,936 60.9 us with them, 57.0 without.
__device__ inline void finish_select(FinishBuffer &fin, uint32_t n, const SamplerConfig &cfg,
                              float uniform, uint32_t row, const SelectOutput &out) {
    const uint32_t lane = lane_id();
    if (n == 0) {  // src/sampler.c:97 "sampler received no finite candidates"
        if (lane == 0) {
            report_row(out, row, kErrFormat, kPaddingId, 0.0f);
            if (out.dbg_count) out.dbg_count[row] = 0;
        }
        return;
    }
    // Every lane has at most two candidates (n <= 64), whose exponentials -- the raw and the tempered
    // weight of each -- do not wait for one another.
    static_assert(kMaxK <= 64, "two candidates per lane");
    const double top_raw = (double)fin.score[0];
    const double temperature = (double)cfg.temperature;
    const double top_tempered = (double)fin.score[0] / temperature;
    const uint32_t i0 = lane, i1 = lane + 32;
    const double s0 = i0 < n ? (double)fin.score[i0] : top_raw;
    const double s1 = i1 < n ? (double)fin.score[i1] : top_raw;
    double raw0 = exp(s0 - top_raw), tempered0 = exp(s0 / temperature - top_tempered);
    double raw1 = 1.0, tempered1 = 1.0;
    if (n > 32) {
        raw1 = exp(s1 - top_raw);
        tempered1 = exp(s1 / temperature - top_tempered);
    }
    // the first of the 64 places at which something holds; `otherwise` when at none
    auto first_place = [](bool here0, bool here1, uint32_t otherwise) {
        const uint32_t low = __ballot_sync(kFullMask, here0), high = __ballot_sync(kFullMask, here1);
        return low ? (uint32_t)__ffs(low) - 1u : high ? (uint32_t)__ffs(high) + 31u : otherwise;
    };
    float u = uniform;
    if (is_nonfinite(u) || u < 0.0f) u = 0.0f;
    if (u >= 1.0f) u = __uint_as_float(0x3f7fffffu);  // nextafterf(1, 0)
    const double top_p = (double)cfg.top_p;
    if (out.dbg_count == nullptr) {
        // A sum of n <= 64 positive terms added from the left is off by at most n 2^-53 of itself, 7.1e-15,
        // one added by the scan by 8 * 2^-53; the reference compares sums of quotients by such a sum with
        // top_p (1.5e-14 together), and such a sum with a multiple of another (the same).
        constexpr double kMargin = 1e-13;
        double r0 = i0 < n ? raw0 : 0.0, r1 = i1 < n ? raw1 : 0.0;
        double t0 = i0 < n ? tempered0 : 0.0, t1 = i1 < n ? tempered1 : 0.0;
        scan_places(r0, r1, n > 32);
        scan_places(t0, t1, n > 32);
        const double sum = __shfl_sync(kFullMask, r1, 31), edge = top_p * sum, margin = kMargin * sum;
        const uint32_t last = first_place(i0 < n && r0 >= edge, i1 < n && r1 >= edge, n - 1u);
        // (The last place is never in doubt: whether its sum reaches top_p or no sum does, all n are kept.)
        bool near = (i0 + 1u < n && fabs(r0 - edge) <= margin) || (i1 + 1u < n && fabs(r1 - edge) <= margin) ||
                    !(sum > 0.0 && sum < 1e300);
        const double low = __shfl_sync(kFullMask, t0, (int)(last & 31u)), high = __shfl_sync(kFullMask, t1, (int)(last & 31u));
        const double weights = last < 32u ? low : high, draw = (double)u * weights, slack = kMargin * weights;
        near = near || (i0 <= last && fabs(t0 - draw) <= slack) || (i1 <= last && fabs(t1 - draw) <= slack) ||
               !(weights > 0.0 && weights < 1e300);
        if (!__any_sync(kFullMask, near)) {
            const uint32_t picked = first_place(i0 <= last && draw < t0, i1 <= last && draw < t1, last);
            if (lane == 0) report_row(out, row, kOk, fin.id[picked], fin.score[picked]);
            return;
        }
    }
    if (i0 < n) {
        fin.raw[i0] = raw0;
        fin.tempered[i0] = tempered0;
    }
    if (i1 < n) {
        fin.raw[i1] = raw1;
        fin.tempered[i1] = tempered1;
    }
    __syncwarp();
    double raw_sum = 0.0;
    if (lane < 2) raw_sum = running_sums(lane == 0 ? fin.raw : fin.tempered, n);
    raw_sum = __shfl_sync(kFullMask, raw_sum, 0);
    if (!(raw_sum > 0.0) || isinf(raw_sum) || isnan(raw_sum)) {  // "sampler raw softmax failed"
        if (lane == 0) {
            report_row(out, row, kErrFormat, kPaddingId, 0.0f);
            if (out.dbg_count) out.dbg_count[row] = 0;
        }
        return;
    }
    raw0 = raw0 / raw_sum;
    raw1 = raw1 / raw_sum;
    if (i0 < n) fin.raw[i0] = raw0;
    if (i1 < n) fin.raw[i1] = raw1;
    __syncwarp();
    if (lane == 0) running_sums(fin.raw, n, &top_p);  // (the sums grow: the first that reaches it counts)
    __syncwarp();
    const uint32_t cutoff = first_place(i0 < n && fin.raw[i0] >= top_p, i1 < n && fin.raw[i1] >= top_p, n - 1u) + 1u;
    const double weight_sum = fin.tempered[cutoff - 1u];
    if (!(weight_sum > 0.0) || isinf(weight_sum) || isnan(weight_sum)) {  // "sampler temperature softmax failed"
        if (lane == 0) {
            report_row(out, row, kErrFormat, kPaddingId, 0.0f);
            if (out.dbg_count) out.dbg_count[row] = 0;
        }
        return;
    }
    const double draw = (double)u * weight_sum;
    const uint32_t picked = first_place(i0 < cutoff && draw < fin.tempered[i0], i1 < cutoff && draw < fin.tempered[i1],
                                        cutoff - 1u);
    if (lane == 0) report_row(out, row, kOk, fin.id[picked], fin.score[picked]);
    if (out.dbg_count) {
        if (lane == 0) out.dbg_count[row] = n;
        const size_t at = (size_t)row * kMaxK;
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            const uint32_t i = lane + 32 * h;
            const bool live = i < n;
            if (out.dbg_ids) out.dbg_ids[at + i] = live ? fin.id[i] : kPaddingId;
            if (out.dbg_scores) out.dbg_scores[at + i] = live ? fin.score[i] : 0.0f;
            if (out.dbg_raw) out.dbg_raw[at + i] = live ? (h ? raw1 : raw0) : 0.0;
            if (out.dbg_tempered) out.dbg_tempered[at + i] = i < cutoff ? (h ? tempered1 : tempered0) / weight_sum : 0.0;
        }
    }
}

}  // namespace fgk
