// What the two kernels that scan rows against an admission bound share: 128-bit vectors of
// logits, maxima, and a row's result.
#pragma once

#include "fg_block_select.cuh"

namespace fgk {

constexpr uint32_t kHugeBits = 0x6b000000u;  // |x| >= 2^87: a repetition factor of 2^-40 to 2^40 may reach inf

template <typename T>
struct Lanes;
template <>
struct Lanes<float> {
    static constexpr int kPer = 4;  // logits per 128-bit vector
    static __device__ __forceinline__ void unpack(const uint4 &raw, float *v) {
        v[0] = __uint_as_float(raw.x);
        v[1] = __uint_as_float(raw.y);
        v[2] = __uint_as_float(raw.z);
        v[3] = __uint_as_float(raw.w);
    }
};
template <>
struct Lanes<uint16_t> {  // bf16 bit patterns
    static constexpr int kPer = 8;
    static __device__ __forceinline__ void unpack(const uint4 &raw, float *v) {
        v[0] = __uint_as_float(raw.x << 16);
        v[1] = __uint_as_float(raw.x & 0xffff0000u);
        v[2] = __uint_as_float(raw.y << 16);
        v[3] = __uint_as_float(raw.y & 0xffff0000u);
        v[4] = __uint_as_float(raw.z << 16);
        v[5] = __uint_as_float(raw.z & 0xffff0000u);
        v[6] = __uint_as_float(raw.w << 16);
        v[7] = __uint_as_float(raw.w & 0xffff0000u);
    }
};

// Shared words that warps watch while others change them.
__device__ __forceinline__ uint32_t peek(const uint32_t *word) {
    return *reinterpret_cast<const volatile uint32_t *>(word);
}
__device__ __forceinline__ unsigned long long peek64(const unsigned long long *word) {
    return *reinterpret_cast<const volatile unsigned long long *>(word);
}
__device__ __forceinline__ void poke(uint32_t *word, uint32_t value) {
    *reinterpret_cast<volatile uint32_t *>(word) = value;
}

__device__ __forceinline__ uint64_t warp_max_u64(uint64_t v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const uint64_t other = __shfl_xor_sync(kFullMask, v, d);
        v = other > v ? other : v;
    }
    return v;
}
__device__ __forceinline__ uint64_t warp_min_u64(uint64_t v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const uint64_t other = __shfl_xor_sync(kFullMask, v, d);
        v = other < v ? other : v;
    }
    return v;
}

// Largest of three; a NaN loses against a number, as with fmaxf.
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// max(m, v...) that turns NaN as soon as one operand is NaN.
template <int N>
__device__ __forceinline__ float propagating_max(float m, const float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++) asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(v[i]));
    return m;
}

// Smallest of N values; a NaN loses against a number, as with fminf.
template <int N>
__device__ __forceinline__ float smallest(const float (&v)[N]) {
    float m = v[0];
#pragma unroll
    for (int i = 1; i < N; i++) m = fminf(m, v[i]);
    return m;
}

// Largest of N values, three at a time (a short tree instead of a chain of N - 1).
template <int N>
__device__ __forceinline__ float largest(const float (&v)[N]) {
    float level[N];
#pragma unroll
    for (int i = 0; i < N; i++) level[i] = v[i];
    int n = N;
#pragma unroll
    for (int round = 0; round < 6; round++) {
        if (n <= 1) break;
        int m = 0;
#pragma unroll
        for (int i = 0; i < N; i += 3) {
            if (i >= n) break;
            if (i + 2 < n) level[m++] = fmax3(level[i], level[i + 1], level[i + 2]);
            else if (i + 1 < n) level[m++] = fmaxf(level[i], level[i + 1]);
            else level[m++] = level[i];
        }
        n = m;
    }
    return level[0];
}

// What is known about a row, or about a shard's part of it, when its k best are in a
// FinishBuffer in sampling order.
struct RowResult {
    uint32_t kept;         // how many they are
    uint32_t wild_id;      // greedy rows: smallest id holding a NaN/Inf, padding if none
    uint32_t wild_bits;    // its value
    uint32_t bad_history;  // 0, or the fg_status a broken history earns the row
};

// Writes a row's result, or a shard's candidates; called by one warp.  `p`: the kernel's
// parameters (shard_k, shard_scores, shard_ids, shard_stride, push, out).  `uniform`: the row's draw.
template <class Params>
__device__ __forceinline__ void finish_row(const Params &p, FinishBuffer &fin, const RowResult &result, uint32_t k,
                                           bool greedy, const SamplerConfig &cfg, float uniform, uint32_t row) {
    const uint32_t lane = lane_id();
    if (p.shard_k != 0) {
        // a greedy row's NaN/Inf with the smallest id goes first, as the slice's argmax
        // cascade of src/output.c:320-344 would report it; the finite ones follow
        const uint32_t lead = greedy && result.wild_id != kPaddingId ? 1u : 0u;
        for (uint32_t i = lane; i < k; i += 32) {
            const size_t at = ((size_t)row * k + i) * p.shard_stride;
            const bool ok = i >= lead && i - lead < result.kept && !result.bad_history;
            float score = ok ? fin.score[i - lead] : __uint_as_float(0xff800000u);
            uint32_t id = ok ? fin.id[i - lead] : kPaddingId;
            if (lead && i == 0 && !result.bad_history) {
                score = __uint_as_float(result.wild_bits);
                id = result.wild_id;
            }
            if (p.push.ranks != 0) {
                // the fused exchange: the block lands in every rank's window, this one's too
                for (uint32_t t = 0; t < p.push.ranks; t++)
                    *p.push.pair(t, row, k, i) = make_uint2(__float_as_uint(score), id);
            } else {
                p.shard_scores[at] = score;
                p.shard_ids[at] = id;
            }
        }
        if (p.push.ranks != 0) {
            __threadfence_system();  // the pairs are visible on the peers before the arrivals are
            __syncwarp();
            if (lane < p.push.ranks) atomicAdd_system(p.push.arrived(lane, row), 1u);
        }
        if (lane == 0) {
            p.out.row_status[row] = result.bad_history;
            if (result.bad_history) note_error(p.out, row, result.bad_history);
        }
        return;
    }
    if (result.bad_history) {  // "history token ... is outside vocabulary", src/output.c:610-612
        if (lane == 0) {
            report_row(p.out, row, result.bad_history, kPaddingId, 0.0f);
            if (p.out.dbg_count) p.out.dbg_count[row] = 0;
        }
        return;
    }
    if (greedy) {
        if (lane == 0) {
            uint32_t status = kOk, token;
            float logit;
            if (result.wild_id != kPaddingId) {
                // a NaN/Inf beats every finite logit in the argmax order and is then
                // rejected: src/output.c:593 (no penalties) / 737-739 (penalised)
                status = penalties_active(cfg) ? kErrFormat : kErrMismatch;
                token = result.wild_id;
                logit = __uint_as_float(result.wild_bits);
            } else if (result.kept == 0) {
                status = kErrMismatch;
                token = kPaddingId;
                logit = 0.0f;
            } else {
                token = fin.id[0];
                logit = fin.score[0];
            }
            report_row(p.out, row, status, token, logit);
            if (p.out.dbg_count) {
                const bool ok = status == kOk;
                p.out.dbg_count[row] = ok ? 1u : 0u;
                if (p.out.dbg_ids) p.out.dbg_ids[(size_t)row * kMaxK] = ok ? token : kPaddingId;
                if (p.out.dbg_scores) p.out.dbg_scores[(size_t)row * kMaxK] = ok ? logit : 0.0f;
            }
        }
        return;
    }
    finish_select(fin, result.kept, cfg, uniform, row, p.out);
}

}  // namespace fgk
