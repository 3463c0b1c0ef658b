// Sampling without a top-k cut: top-p over the whole vocabulary, then temperature and
// inverse CDF — the reference's select step (src/sampler.c:97-121) with limit = every
// finite logit.  The reference caps candidates at 64; this is the documented
// generalisation for rows whose nucleus spans tens of thousands of tokens.
//
// The vocabulary is never sorted.  A row belongs to a team of one, two, four or eight CTAs (a
// thread-block cluster), each of which takes a range of its columns.
//
// The short way.  One pass over the logits counts the values into 8,192 buckets of three
// widths in shared memory.  A bucket holds the number of its members and the first two moments of
// their distances from its middle, which give its raw and its tempered softmax mass alike
// (a short series); prefix sums over the buckets' masses tell in which bucket the
// cumulative mass reaches top_p and, to within a bucket or two, where the draw lands.  A
// second pass gathers the members of those buckets, a few hundred, which are
// ordered exactly: the element at which top_p is reached, then the element drawn.  (It reads from L2 while the
// rows in flight fit there.  512 fp32 rows of 151,936 with 32,768 tokens each: 296 rows in flight are 180 MB, and the
// launch reads 1,049 MB, the logits being 311.)
//
// The long way, for rows the short one cannot take (heavy ties, very low temperatures, masses that
// would not be good enough): the CTAs of the team work on the penalised row in scratch memory, histogram
// pass by histogram pass, down to an MSB-first radix descent over the 32-bit monotone value key
// and, among equal values, over the id.
//
// Masses are exp(s - max) as 2^-44 (the long way: 2^-40) fixed point in 64-bit integers: integer
// addition is associative, so the result does not depend on the order threads arrive in, and
// the grid is far below one element's weight.  The reference adds doubles left to right; the two
// agree unless the top-p bound or the draw falls within 1e-10 (relative; as a rule 1e-12) of an edge
// of the CDF: see the errors measured below.
#include <cooperative_groups.h>

#include <cstddef>

#include "fg_block_select.cuh"
#include "fg_kernels.h"
#include "fg_nucleus_window.cuh"

namespace fgk {


constexpr int kNucleusThreads = 512;  // two CTAs to an SM: one streams while the other scans and sorts
constexpr int kNucleusWarps = kNucleusThreads / 32;
constexpr int kBuckets = 4096;  // of the long way

struct NucleusParams {
    const void *logits;
    uint32_t dtype;
    uint32_t rows, vocab;
    uint64_t row_stride;
    const SamplerConfig *configs;
    SamplerConfig config0;
    uint32_t config_count;
    const float *uniforms;
    uint32_t team;             // CTAs that share a row (the cluster size): 1, 2, 4 or 8
    float *scratch;            // gridDim.x / team rows of scratch_stride floats, used on the long way
    uint64_t scratch_stride;
    float2 *seen;              // per CTA seen_stride (penalised value, id) pairs
    uint64_t seen_stride;
    // history structures built by history_build_kernel, one per (row, split)
    const uint32_t *history_global;
    uint64_t history_stride_words;
    const void *history_meta;
    uint32_t splits, split_len, bitmap_words, count_capacity, dense_wide;
    SelectOutput out;
};

struct NucleusShared {
    unsigned long long *mass;         // the long way's kBuckets masses and counts
    uint32_t *count;
    double table[64];                 // 2^(j/64)
    unsigned long long scan_mass[kNucleusWarps];
    uint32_t scan_count[kNucleusWarps];
    unsigned long long total_mass;
    float reduce_max[kNucleusWarps];
    float zero;
    // result of a scan
    uint32_t hit_bucket;
    unsigned long long hit_mass_before;
    uint32_t hit_count_before;
    uint32_t hit_found;
};

// exp(x) * 2^bits for x <= 0 as a 64-bit integer (round to nearest): argument reduction
// to n/64 * ln2 + r, |r| <= ln2/128, a 64-entry table of 2^(j/64) and a degree-5
// polynomial (truncation 4e-17).  Below e^-70 the weight is under the fixed-point grid.
__device__ __forceinline__ unsigned long long exp_fixed(double x, const double *table, int bits = 40) {
    if (!(x > -70.0)) return 0ull;
    const double scaled = x * 92.33248261689366;                  // 64 / ln 2
    const double shifted = scaled + 6755399441055744.0;           // 1.5 * 2^52: rounds to nearest
    const int n = __double2loint(shifted);
    const double nd = shifted - 6755399441055744.0;
    double r = fma(nd, -1.0830424696249145e-02, x);               // ln2/64, high part
    r = fma(nd, -3.623510646634843e-19, r);                       // low part
    double p = fma(r, 8.3333333333333332e-03, 4.1666666666666664e-02);
    p = fma(p, r, 1.6666666666666666e-01);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);                                           // 1 + r + r^2/2 + ... + r^5/120
    const int j = n & 63, k = n >> 6;                             // floor division for negative n
    const double scale = __longlong_as_double((long long)(k + bits + 1023) << 52);
    return __double2ull_rn(table[j] * p * scale);
}

// Block-wide: walk the buckets from the top; find the first bucket b where
// before + mass(>= b) reaches `target` (strict: exceeds it).  All threads call.
__device__ void find_crossing(NucleusShared &sh, uint32_t buckets, unsigned long long before,
                              unsigned long long target, bool strict) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t per = (buckets + kNucleusThreads - 1) / kNucleusThreads;
    // thread t owns buckets top-down: indices buckets-1 - (t*per + i)
    unsigned long long mine_mass = 0;
    uint32_t mine_count = 0;
    for (uint32_t i = 0; i < per; i++) {
        const uint32_t at = tid * per + i;
        if (at < buckets) {
            mine_mass += sh.mass[buckets - 1 - at];
            mine_count += sh.count[buckets - 1 - at];
        }
    }
    unsigned long long incl_mass = mine_mass;
    uint32_t incl_count = mine_count;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long up_mass = __shfl_up_sync(kFullMask, incl_mass, d);
        const uint32_t up_count = __shfl_up_sync(kFullMask, incl_count, d);
        if (lane >= (uint32_t)d) {
            incl_mass += up_mass;
            incl_count += up_count;
        }
    }
    if (lane == 31) {
        sh.scan_mass[warp] = incl_mass;
        sh.scan_count[warp] = incl_count;
    }
    if (tid == 0) sh.hit_found = 0;
    __syncthreads();
    unsigned long long prior_mass = before + incl_mass - mine_mass;
    uint32_t prior_count = incl_count - mine_count;
    for (uint32_t w = 0; w < warp; w++) {
        prior_mass += sh.scan_mass[w];
        prior_count += sh.scan_count[w];
    }
    const unsigned long long after = prior_mass + mine_mass;
    const bool was = strict ? prior_mass > target : prior_mass >= target;
    const bool now = strict ? after > target : after >= target;
    if (!was && now) {  // exactly one thread
        for (uint32_t i = 0; i < per; i++) {
            const uint32_t at = tid * per + i;
            if (at >= buckets) break;
            const uint32_t b = buckets - 1 - at;
            const unsigned long long next = prior_mass + sh.mass[b];
            if (strict ? next > target : next >= target) {
                sh.hit_bucket = b;
                sh.hit_mass_before = prior_mass;
                sh.hit_count_before = prior_count;
                sh.hit_found = 1;
                break;
            }
            prior_mass = next;
            prior_count += sh.count[b];
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void clear_histogram(NucleusShared &sh, uint32_t buckets) {
    for (uint32_t b = threadIdx.x; b < buckets; b += kNucleusThreads) {
        sh.mass[b] = 0;
        sh.count[b] = 0;
    }
    __syncthreads();
}

// Walks a scratch row: visit(value, index) for every element.  The next two quads of a thread are on
// their way while it looks at two: a pass over the row is a chain of L2 latencies otherwise.  Rows
// start 16-byte aligned.
template <class Visit>
__device__ __forceinline__ void walk_row(const float *values, uint32_t vocab, Visit visit) {
    const float4 *wide = reinterpret_cast<const float4 *>(values);
    const uint32_t tid = threadIdx.x, quads = vocab / 4u;
    auto visit_quad = [&](const float4 &v, uint32_t i) {
        visit(v.x, i);
        visit(v.y, i + 1u);
        visit(v.z, i + 2u);
        visit(v.w, i + 3u);
    };
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
    uint32_t q = tid;
    if (q < quads) a = wide[q];
    if (q + kNucleusThreads < quads) b = wide[q + kNucleusThreads];
    for (; q < quads; q += 2 * kNucleusThreads) {
        const float4 now_a = a, now_b = b;
        const uint32_t next = q + 2 * kNucleusThreads;
        if (next < quads) a = wide[next];
        if (next + kNucleusThreads < quads) b = wide[next + kNucleusThreads];
        visit_quad(now_a, q * 4u);
        if (q + kNucleusThreads < quads) visit_quad(now_b, (q + kNucleusThreads) * 4u);
    }
    const uint32_t rest = quads * 4u + tid;
    if (rest < vocab) visit(values[rest], rest);
}

// *mass += w in shared memory by two 32-bit adds, the carry between them (a 64-bit one is a loop of
// compare-and-swaps, which many values of one bucket make each other repeat).
__device__ __forceinline__ void add_mass(unsigned long long *mass, unsigned long long w) {
    uint32_t *half = reinterpret_cast<uint32_t *>(mass);
    const uint32_t low = (uint32_t)w, before = atomicAdd(half, low);
    const uint32_t high = (uint32_t)(w >> 32) + (before + low < low ? 1u : 0u);
    if (high != 0) atomicAdd(half + 1, high);
}

// Which elements of the scratch row take part in a descent.
struct Nucleus {
    uint32_t key;     // value key of the last element inside
    uint32_t id;      // ... and its id (ties on the key are ordered by id)
    bool everything;  // no cut yet: every finite value takes part
    __device__ __forceinline__ bool holds(uint32_t k, uint32_t i) const {
        return everything || k > key || (k == key && i <= id);
    }
};

constexpr uint32_t kOrderCap = 2048;   // entries order_members takes

// Entries to be ordered and the memory that takes.
struct OrderWork {
    float *value;
    uint32_t *id;
    float *sorted_value;
    uint32_t *sorted_id;
    unsigned long long *weight;  // of the sorted entries, then their running sum
};

// Like find_crossing but walking the buckets upwards from 0; also leaves the sum of
// all masses in sh.total_mass.  target_of(total) is evaluated once the total is known.
// All threads call.  sh.hit_found == 0 means the total never reaches the target.
template <typename TargetOf>
__device__ unsigned long long find_crossing_up(NucleusShared &sh, TargetOf target_of, bool strict) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    constexpr uint32_t per = kBuckets / kNucleusThreads;
    unsigned long long mine_mass = 0;
    uint32_t mine_count = 0;
#pragma unroll
    for (uint32_t i = 0; i < per; i++) {
        mine_mass += sh.mass[tid * per + i];
        mine_count += sh.count[tid * per + i];
    }
    unsigned long long incl_mass = mine_mass;
    uint32_t incl_count = mine_count;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long up_mass = __shfl_up_sync(kFullMask, incl_mass, d);
        const uint32_t up_count = __shfl_up_sync(kFullMask, incl_count, d);
        if (lane >= (uint32_t)d) {
            incl_mass += up_mass;
            incl_count += up_count;
        }
    }
    if (lane == 31) {
        sh.scan_mass[warp] = incl_mass;
        sh.scan_count[warp] = incl_count;
    }
    if (tid == 0) sh.hit_found = 0;
    __syncthreads();
    unsigned long long prior_mass = incl_mass - mine_mass, total = 0;
    uint32_t prior_count = incl_count - mine_count;
    for (uint32_t w = 0; w < kNucleusThreads / 32; w++) {
        if (w < warp) {
            prior_mass += sh.scan_mass[w];
            prior_count += sh.scan_count[w];
        }
        total += sh.scan_mass[w];
    }
    const unsigned long long target = target_of(total);
    const unsigned long long after = prior_mass + mine_mass;
    const bool was = strict ? prior_mass > target : prior_mass >= target;
    const bool now = strict ? after > target : after >= target;
    if (!was && now) {  // exactly one thread
#pragma unroll
        for (uint32_t i = 0; i < per; i++) {
            const uint32_t b = tid * per + i;
            const unsigned long long next = prior_mass + sh.mass[b];
            if (strict ? next > target : next >= target) {
                sh.hit_bucket = b;
                sh.hit_mass_before = prior_mass;
                sh.hit_count_before = prior_count;
                sh.hit_found = 1;
                break;
            }
            prior_mass = next;
            prior_count += sh.count[b];
        }
    }
    if (tid == 0) sh.total_mass = total;
    __syncthreads();
    return target;
}

struct Position {
    uint32_t key, id;            // the element found
    float value;
    unsigned long long mass;     // cumulative weight up to and including it
    uint32_t rank;               // its 1-based position in the order
    unsigned long long total;    // weight of everything inside
    bool ok;                     // false: fall back to the generic descent
};

// The first `members` entries of the list, those of them that lie `inside`, ordered exactly, and
// among them the first at which the running weight -- `before` plus the weights
// exp((v - top) * inv_t) of the members so far -- reaches `target` (strict: exceeds it); the last
// one when none does or when `clipped`.  ok = false: there is no member inside.  With
// `also_sum` the weights exp((v - top) * also_inv_t) of the members up to and including the
// one found are summed into it.  All threads call.
__device__ __forceinline__ Position order_members(NucleusShared &sh, const OrderWork &list, uint32_t members, double inv_t, float top,
                                  const Nucleus inside, unsigned long long before, uint32_t rank_before,
                                  unsigned long long target, bool strict, bool clipped, double also_inv_t,
                                  unsigned long long *also_sum, int bits) {
    const uint32_t tid = threadIdx.x;
    Position found;
    found.ok = false;
    found.total = 0;
    const uint32_t listed = members;
    // order them by their (value, ~id) keys
    unsigned long long *key = list.weight;
    if (members <= 256u) {
        // an entry's rank is the number of larger keys; several threads count for one entry, each
        // over a part of the list
        uint32_t *rank = list.sorted_id;
        for (uint32_t a = tid; a < members; a += kNucleusThreads) {
            key[a] = select_key(list.value[a], list.id[a]);
            rank[a] = 0;
        }
        __syncthreads();
        const uint32_t parts = members <= 64u ? 8u : members <= 128u ? 4u : 2u;
        const uint32_t abreast = kNucleusThreads / parts, length = (members + parts - 1u) / parts;
        const uint32_t from = tid / abreast * length, to = min(members, from + length), a = tid % abreast;
        const unsigned long long mine = a < members ? key[a] : 0ull;
        if (a < members) {
            uint32_t larger = 0;
#pragma unroll 4
            for (uint32_t b = from; b < to; b++) larger += key[b] > mine ? 1u : 0u;
            atomicAdd(&rank[a], larger);
        }
        __syncthreads();
        const uint32_t place = a < members ? rank[a] : 0u;
        __syncthreads();
        if (a < members && tid < abreast) key[place] = mine;
        __syncthreads();
    } else {
        // a bitonic network, the largest first; zeros fill up to a power of two
        uint32_t size = 512u;
        while (size < members) size *= 2u;
        for (uint32_t a = tid; a < size; a += kNucleusThreads)
            key[a] = a < members ? select_key(list.value[a], list.id[a]) : 0ull;
        for (uint32_t run = 2; run <= size; run <<= 1) {
            for (uint32_t stride = run >> 1; stride > 0; stride >>= 1) {
                __syncthreads();
                for (uint32_t pair = tid; pair < size / 2; pair += kNucleusThreads) {
                    const uint32_t low = ((pair & ~(stride - 1)) << 1) | (pair & (stride - 1)), high = low | stride;
                    const unsigned long long x = key[low], y = key[high];
                    if ((x < y) == ((low & run) == 0)) {
                        key[low] = y;
                        key[high] = x;
                    }
                }
            }
        }
        __syncthreads();
    }
    constexpr int kOwned = kOrderCap / kNucleusThreads;
#pragma unroll
    for (int h = 0; h < kOwned; h++) {
        const uint32_t a = h * kNucleusThreads + tid;
        if (a >= members) continue;
        const unsigned long long mine = key[a];
        const float value = key_to_float((uint32_t)(mine >> 32));  // (-0.0 comes back as +0.0: see below)
        list.sorted_value[a] = value;
        list.sorted_id[a] = ~(uint32_t)mine;
        list.weight[a] = exp_fixed(((double)value - (double)top) * inv_t, sh.table, bits);
    }
    __syncthreads();
    // (what is not inside the nucleus comes last in the order)
    uint32_t held = 0;
    for (uint32_t a = 0; a < members; a += kNucleusThreads) {
        const uint32_t at = a + tid;
        held += __syncthreads_count(at < members && inside.holds(float_key(list.sorted_value[at]), list.sorted_id[at]));
    }
    members = held;
    if (members == 0) return found;
    // running sum: a few entries per thread, then the usual scan
    {
        const uint32_t lane = tid & 31u, warp = tid >> 5;
        unsigned long long sums[kOwned], own = 0;
#pragma unroll
        for (int h = 0; h < kOwned; h++) {
            const uint32_t a = kOwned * tid + h;
            own += a < members ? list.weight[a] : 0ull;
            sums[h] = own;
        }
        unsigned long long incl = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long up = __shfl_up_sync(kFullMask, incl, d);
            if (lane >= (uint32_t)d) incl += up;
        }
        if (lane == 31) sh.scan_mass[warp] = incl;
        __syncthreads();
        unsigned long long prior = before + incl - own;
#pragma unroll
        for (uint32_t w = 0; w < (uint32_t)kNucleusWarps; w++) {
            const unsigned long long sum = sh.scan_mass[w];
            prior += w < warp ? sum : 0ull;
        }
#pragma unroll
        for (int h = 0; h < kOwned; h++) {
            const uint32_t a = kOwned * tid + h;
            if (a < members) list.weight[a] = prior + sums[h];
        }
        if (tid == 0) sh.hit_bucket = kPaddingId;
        __syncthreads();
    }
    // the first entry whose running sum reaches the target (exactly one thread sees the step)
    for (uint32_t a = tid; a < members; a += kNucleusThreads) {
        const unsigned long long here = list.weight[a];
        const unsigned long long prev = a ? list.weight[a - 1] : before;
        const bool was = strict ? prev > target : prev >= target;
        const bool now = strict ? here > target : here >= target;
        if (!clipped && !was && now) sh.hit_bucket = a;
    }
    __syncthreads();
    uint32_t at = sh.hit_bucket;
    if (clipped || at == kPaddingId) at = members - 1;
    found.key = float_key(list.sorted_value[at]);
    found.id = list.sorted_id[at];
    found.value = list.sorted_value[at];
    if (found.value == 0.0f) {  // the zero's own sign, from the unsorted entry
        if (tid == 0) sh.zero = 0.0f;
        __syncthreads();
        for (uint32_t a = tid; a < listed; a += kNucleusThreads)
            if (list.id[a] == found.id) sh.zero = list.value[a];
        __syncthreads();
        found.value = sh.zero;
    }
    found.mass = list.weight[at];
    found.rank = rank_before + at + 1;
    found.ok = true;
    __syncthreads();
    if (also_sum != nullptr) {
        // the other weight of the members up to the one found (order does not matter: integers)
        unsigned long long part = 0;
        for (uint32_t a = tid; a <= at; a += kNucleusThreads)
            part += exp_fixed(((double)list.sorted_value[a] - (double)top) * also_inv_t, sh.table, bits);
        const uint32_t lane = tid & 31u, warp = tid >> 5;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(kFullMask, part, d);
        if (lane == 0) sh.scan_mass[warp] = part;
        __syncthreads();
        unsigned long long sum = 0;
        for (int w = 0; w < kNucleusThreads / 32; w++) sum += sh.scan_mass[w];
        *also_sum = sum;
        __syncthreads();
    }
    return found;
}

// After a crossing search: the bucket it stopped in, or -- when the total never reaches the
// target (top_p = 1, a draw rounded up to the total) -- the last non-empty bucket.  Returns
// whether it was clipped; all threads call.
__device__ bool settle_crossing(NucleusShared &sh) {
    if (sh.hit_found) return false;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long m = 0;
        uint32_t c = 0, last = 0;
        bool any = false;
        for (uint32_t b = 0; b < kBuckets; b++) {
            if (sh.count[b]) {
                if (any) {
                    m += sh.mass[last];
                    c += sh.count[last];
                }
                last = b;
                any = true;
            }
        }
        sh.hit_bucket = last;
        sh.hit_mass_before = m;
        sh.hit_count_before = c;
    }
    __syncthreads();
    return true;
}

// ================================================================== the short way
//
// What bounds it: instruction issue and latency.  The first pass is about twenty instructions and
// two shared-memory adds per logit; masses are not summed per logit, exp() and fp64 appear once
// per bucket.  A row's other steps (scanning the buckets, ordering the candidates) are chains of
// latencies of 20 us, so two CTAs share an SM, one streaming while the other scans and sorts; for
// few rows a row is spread over several CTAs instead.  A CTA per row and SM that added two fp64 weights
// per logit to five shared-memory sums took, per call: 512 rows of 151,936 fp32 logits, histories
// of 32,768 tokens 772 us (now 571), without history 538 (250); 32 rows bf16 410-560 (64).
// With histories the largest part is the seen columns' gather (amend_seen).
//
// A value's place: buckets 1/1024 wide over the top four units of the row's window, 1/256 wide over
// the next eight, 1/64 over the next 32 (all half as wide for temperatures below 0.36, a quarter as
// wide below 0.18, and so on), with their middles on the grid of multiples of the width, so that
// neither the bucket nor the distance f from its middle depends on a subtraction that rounds:
// n = rint(v * 1024) by adding and subtracting 1.5 * 2^23, f = v * 1024 - n in [-1/2, 1/2], both exact
// in fp32.  With w = width * f the members' weights relative to the middle's add up to
//     sum exp(w) = N + c M1 + c^2/2 M2 + c^3/6 M3 + ...,   c = width (times 1/T: tempered)
// M3 is not kept: f^3 is replaced by the nearest multiple of f (0.15 f over a bucket), which
// leaves 0.019 c^3/6 (root mean square) of a member's weight: 3e-12 raw and 2.4e-11 at T = 0.5 in
// the narrow buckets, against 6.7e-11 for weights rounded to 2^-32 of themselves, but 2e-10 and 1.2e-8 raw in
// the wider ones.  So make_plan estimates how far off the masses are (place_error), and a row whose bulk
// lies in wide buckets -- a peak above it placed the window -- is counted again with a window that has
// its top at the 512th value, those above it being kept one by one.  What lies under a window (a cold
// row's reaches only 44 units, halved as often as its buckets) counts as an error too.
//
// Largest error of the cumulative masses over their total against extended precision, this and weights
// rounded to 2^-32 (the long way's): rows of 151,936 logits, spread 0.5 to 4 with and without Gumbel
// noise, one token 6 to 20 above a body, 300 or 2,000 tokens 12 above it, bodies at -4 and -10, each
// as fp32, bf16 and bf16 widened to fp32:
//     T      0.2     0.5     1       1.4     2.5
//     here   1e-11   2e-11   9e-12   3e-11   5e-11
//     2^-32  7e-11   7e-11   7e-11   7e-11   6e-11
//
// A bucket is two 32-bit words that are added to, once each, per member:
//     first    sum of f in units of 2^-22 (the bits of f * 2^22 + 1.5 * 2^23: the constant's
//              share, N times its bits, is taken off afterwards, modulo 2^32)
//     second   low 22 bits: sum of f^2 in units of 2^-14; high 10 bits: N times an odd number
//              (what the bits of the constant leave there), so N modulo 1024
// Neither can overflow up to 1023 members.  A row whose counts do not add up to the number of
// values counted had a bucket with more (a wrap loses 1024 and nothing can make up for it): its
// window is placed anew or it goes the long way.  Rows of raw bf16 logits have at most eight significant
// bits, so f is 0 beyond 128 widths from 0, and many members share a value: they trade precision for
// twelve bits of count.  From 2,049 members at f = +-1/2 on, the sum of f^2 can run into the count there; the
// total of the counts tells that as well (one carry changes a count by the inverse of the odd number).
//
// Slots are xor-swizzled inside their group of 32: bf16 values lie a power of two apart and
// would meet in a few banks otherwise.

constexpr uint32_t kMostTeam = 8;              // CTAs that may share a row
constexpr uint32_t kOverCap = 768;             // values above the window that are kept one by one
constexpr uint32_t kCutCap = 1024, kPickCap = kOrderCap;  // members of the cut's bucket and the draw's
constexpr int kSamples = 4;                    // logits a thread looks at to place the window
constexpr float kPeak = 1.5f;                  // the largest of them is left out if it is that far above the next
constexpr uint32_t kBodyRank = 512;            // a window that is placed anew leaves that many values above it
// Buckets are made narrower, halves at a time, until a narrow one is at most 1/369 of the temperature;
// colder rows than the last go the long way (their window would reach less than 5.5 units down).
constexpr float kWideColdest = 0.36f, kMostSharp = 8.0f;
// How far off the cumulative masses may be beyond what weights rounded to 2^-32 of themselves would
// be, by the estimate of make_plan and as a share of their total: a window that promises more is placed
// anew, and a row that even then promises more than the second goes the long way.  (The estimate is
// up to seven times what is found, where few members decide, and down to a twentieth of it for raw bf16
// rows, whose values tie: they are held to a twentieth.  At 8e-12 two rows in a hundred of 38,016 logits
// of spread 3.8 with Gumbel noise, T = 0.54, were counted twice, 75 us instead of 39, for errors of
// 1e-11; at 4e-11 none, and the errors above are the same.)
constexpr double kMassError = 4e-11, kMostMassError = 6e-11;

constexpr uint32_t inverse_mod(uint32_t a, uint32_t modulus) {  // a odd, modulus a power of two
    uint32_t x = 1;
    for (int i = 0; i < 5; i++) x *= 2 - a * x;
    return x & (modulus - 1);
}

// How a bucket's words are packed: rows of raw bf16 logits, all others.
template <bool kRawBf16>
struct Packing {
    static constexpr bool kCoarser = kRawBf16;
    static constexpr int kCountShift = kRawBf16 ? 20 : 22;
    static constexpr uint32_t kCountMask = (1u << (32 - kCountShift)) - 1u;
    static constexpr float kFirstUnit = kRawBf16 ? 1048576.0f : 4194304.0f;  // 2^20, 2^22
    static constexpr float kSecondUnit = kRawBf16 ? 2048.0f : 16384.0f;      // 2^11, 2^14
    static constexpr float kSecondMagic = kRawBf16 ? 13631488.0f : kMagic;   // bits 0x4b500000: an odd count field
    static constexpr uint32_t kField = (kRawBf16 ? 0x4b500000u : kMagicBits) >> kCountShift;
    static_assert(kField & 1u, "the count can be read back");
    // root mean square of f^3 less 0.15 f
    static constexpr float kThirdError = kRawBf16 ? 0.03f : 0.019f;
    static constexpr uint32_t kInverse = inverse_mod(kField, kCountMask + 1u);

    static __device__ __forceinline__ uint32_t count(uint32_t second) {
        return ((second >> kCountShift) * kInverse) & kCountMask;
    }
    static __device__ __forceinline__ int sum_f(uint32_t first, uint32_t n) { return (int)(first - n * kMagicBits); }
    static __device__ __forceinline__ uint32_t sum_ff(uint32_t second) { return second & ((1u << kCountShift) - 1u); }
};

__device__ __forceinline__ uint32_t swizzled(uint32_t slot) { return slot ^ ((slot >> 5) & 31u); }

// What one CTA knows about its columns after the first pass.
struct Share {
    float best;          // largest finite value
    uint32_t finite;     // how many are finite
    double unseen;       // upper bound of what the values under the window weigh (a share of the largest
                         // value's weight); infinite: a bucket had more members than its words take
};

enum Verdict : uint32_t { kDone, kLongWay, kElsewhere };  // (kElsewhere: with the window placed anew)

// What the team's first CTA has found out: in which buckets the answer lies.
struct Plan {
    uint32_t verdict;
    uint32_t cut;                 // 0: above the window, else 1 + slot
    uint32_t pick_first, pick_last;  // the draw lands in one of these, numbered the same way
    unsigned long long cut_target, cut_before, cut_tempered_before;
    uint32_t cut_rank_before, cut_members;
    unsigned long long pick_before;
    uint32_t pick_members;
    float reference;              // where the window goes next, if the verdict is kElsewhere
};

// Result of looking for a crossing among the 32 slots of a group.
struct SlotHit {
    uint32_t slot, count, count_before;
    unsigned long long raw_before, tempered_before, tempered;
};

// What the first CTA of a team asks of all of them on the long way, and what they need for it.
struct LongStep {
    enum What : uint32_t { kStop, kLargest, kWeighBoth, kWeigh, kWeighAll, kWeighKeys, kCountIds, kListMembers, kFindOnly };
    uint32_t what, bucket, level, prefix, key;
    float top;
    double inv_t;
    Nucleus inside;
};
// the levels of a descent over 32 bits: 12, 12 and 8
__device__ __forceinline__ int descent_bits(uint32_t level) { return level < 2u ? 12 : 8; }
__device__ __forceinline__ int descent_shift(uint32_t level) { return level == 0u ? 20 : level == 1u ? 8 : 0; }
__device__ __forceinline__ uint32_t descent_buckets(uint32_t level) { return 1u << descent_bits(level); }

struct ShortShared {
    Share share;
    Plan plan;
    uint32_t over_count, cut_count, pick_count;   // the first CTA's lists
    int lost, below, above;                       // this CTA: not finite, under the window, over it
    uint32_t counted;                             // sum of the buckets' counts
    uint32_t seen_count;                          // seen columns of this CTA
    uint32_t top_slot;                            // the first bucket that holds anything
    uint32_t cut_place, pick_place[2];
    float sample_max[kNucleusWarps], sample_next[kNucleusWarps];
    unsigned long long scan_raw[kNucleusWarps], scan_tempered[kNucleusWarps];
    uint32_t scan_count[kNucleusWarps];
    float raw_error[kNucleusWarps], tempered_error[kNucleusWarps];
    uint32_t poor;                                // the masses are not good enough
    LongStep step;                                // the first CTA's
    uint32_t only_id;
};

// Dynamic shared memory of the kernel: two CTAs' worth fit an SM.  The long way's memory lies over
// all but the last two parts; the ordering works where the buckets were; the queues of visit_seen
// lie over what is only filled after it (`lists` to `edges`).
struct ShortMemory {
    uint32_t first[kSlots], second[kSlots];
    struct {
        float cut_value[kCutCap];
        uint32_t cut_id[kCutCap];
        float pick_value[kPickCap];
        uint32_t pick_id[kPickCap];
    } lists;                                             // the first CTA's
    unsigned long long raw[kPlaces], tempered[kPlaces];  // masses per place, then their running sums
    uint32_t count[kPlaces];
    double edges[2][kGroups];         // raw, tempered: the weight of a group's first middle, times 2^bits
    double lanes[2][3][32];           // the weights of the 32 slots relative to it, by kind of bucket
    float over_value[kOverCap];
    uint32_t over_id[kOverCap];
    ShortShared state;
    NucleusShared scan;               // what the ordering and the long way share
};

// All of it is reached through this, so that functions of their own know it is shared memory.
__device__ __forceinline__ ShortMemory &short_memory() {
    extern __shared__ __align__(16) unsigned char nucleus_memory[];
    return *reinterpret_cast<ShortMemory *>(nucleus_memory);
}

// The CTAs that share a row.  With one CTA a team's barrier is the block's.
struct Team {
    uint32_t size, rank;
    __device__ __forceinline__ void sync() const {
        if (size == 1) {
            __syncthreads();
        } else {
            asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        }
    }
    // the same variable in another CTA's shared memory
    template <class V>
    __device__ __forceinline__ V *at(V *mine, uint32_t other) const {
        return size == 1 ? mine : cooperative_groups::this_cluster().map_shared_rank(mine, other);
    }
};

// Hands out the rows without a top-k cut in turn.  Every warp walks by itself and comes to the
// same rows: with per-row configs it looks at 32 of them at a time.
struct RowWalk {
    uint32_t base, mask, turn;
    __device__ __forceinline__ explicit RowWalk(uint32_t team) : base(0), mask(0), turn(team) {}
    __device__ __forceinline__ bool next(const NucleusParams &p, uint32_t teams, uint32_t &row) {
        if (p.config_count <= 1) {
            row = turn;
            turn += teams;
            return row < p.rows;
        }
        for (;;) {
            while (mask == 0) {
                if (base >= p.rows) return false;
                const uint32_t mine = base + lane_id();
                bool ours = false;
                if (mine < p.rows) ours = p.configs[mine].temperature != 0.0f && p.configs[mine].top_k == 0;
                mask = __ballot_sync(kFullMask, ours);
                base += 32;
            }
            const uint32_t lowest = (uint32_t)__ffs(mask) - 1u;
            mask &= mask - 1;
            if (turn == 0) {
                turn = teams - 1;
                row = base - 32 + lowest;
                return true;
            }
            turn--;
        }
    }
};

template <typename T>
struct Vector;
template <>
struct Vector<float> {
    static constexpr int kPer = 4;
    static __device__ __forceinline__ float one(const float *p) { return __ldg(p); }
    static __device__ __forceinline__ void unpack(const uint4 &raw, float (&v)[4]) {
        v[0] = __uint_as_float(raw.x);
        v[1] = __uint_as_float(raw.y);
        v[2] = __uint_as_float(raw.z);
        v[3] = __uint_as_float(raw.w);
    }
};
template <>
struct Vector<uint16_t> {  // bf16 bit patterns
    static constexpr int kPer = 8;
    static __device__ __forceinline__ float one(const uint16_t *p) { return bf16_bits_to_float(__ldg(p)); }
    static __device__ __forceinline__ void unpack(const uint4 &raw, float (&v)[8]) {
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

// Walks n logits from `source` on: vectors(v, column) for 128-bit vectors, one(v, column) for the
// ragged ends and for what lies before the first 16-byte boundary.  The next two vectors of a
// thread are on their way while it looks at two.
template <typename T, class Vectors, class One>
__device__ __forceinline__ void walk_logits(const T *source, uint32_t n, Vectors vectors, One one) {
    constexpr int kPer = Vector<T>::kPer;
    const uint32_t tid = threadIdx.x;
    const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(source) & 15u);
    const uint32_t head = min(n, (off ? 16u - off : 0u) / (uint32_t)sizeof(T));
    const uint32_t count = (n - head) / kPer;
    const T *body = source + head;
    if (tid < head) one(Vector<T>::one(source + tid), tid);
    const uint32_t rest = head + count * kPer + tid;
    if (rest < n) one(Vector<T>::one(source + rest), rest);
    uint4 a = make_uint4(0, 0, 0, 0), b = a;
    uint32_t i = tid;
    if (i < count) a = load_stream_128(body + (size_t)i * kPer);
    if (i + kNucleusThreads < count) b = load_stream_128(body + (size_t)(i + kNucleusThreads) * kPer);
    for (; i < count; i += 2 * kNucleusThreads) {
        const uint4 now_a = a, now_b = b;
        const uint32_t next = i + 2 * kNucleusThreads;
        if (next < count) a = load_stream_128(body + (size_t)next * kPer);
        if (next + kNucleusThreads < count) b = load_stream_128(body + (size_t)(next + kNucleusThreads) * kPer);
        float v[kPer];
        Vector<T>::unpack(now_a, v);
        vectors(v, head + i * kPer);
        if (i + kNucleusThreads < count) {
            Vector<T>::unpack(now_b, v);
            vectors(v, head + (i + kNucleusThreads) * kPer);
        }
    }
}

// v[j] for a j that is not known at compile time, without an array in memory
template <int kPer>
__device__ __forceinline__ float pick_element(const float (&v)[kPer], int j) {
    float x = v[0];
#pragma unroll
    for (int i = 1; i < kPer; i++) x = i == j ? v[i] : x;
    return x;
}

// What a pass over one CTA's columns finds out beside the buckets.
struct Findings {
    float best;                     // largest finite value; with penalties, of those outside the window
    int lost, below, above;         // not finite, under the window, over it
};

// Which of a row's columns its history has seen, where that is asked of single columns.
struct SeenBits {
    const uint32_t *bitmap;         // the row's first history structure; null: no penalties
    uint64_t stride;                // words between its splits
    uint32_t split_len;
    __device__ __forceinline__ bool test(uint32_t column) const {
        if (bitmap == nullptr) return false;
        const uint32_t split = column / split_len, local = column - split * split_len;
        return (bitmap[split * stride + (local >> 5)] >> (local & 31u)) & 1u;
    }
};

// The first pass over one CTA's columns: counts into the buckets, values above the window onto
// the first CTA's list.
template <class P, bool kPenalised>
struct Counter {
    const Window window;
    const Team team;
    Findings found;

    __device__ __forceinline__ Counter(const Window &w, const Team &team_) : window(w), team(team_) {
        found.best = -INFINITY;
        found.lost = found.below = found.above = 0;
    }
    // a value inside the window
    __device__ __forceinline__ void count(float v) {
        ShortMemory &m = short_memory();
        float f;
        const uint32_t at = swizzled(window.slot(v, f));
        atomicAdd(&m.first[at], __float_as_uint(__fmaf_rn(f, P::kFirstUnit, kMagic)));
        atomicAdd(&m.second[at], __float_as_uint(__fmaf_rn(__fmul_rn(f, f), P::kSecondUnit, P::kSecondMagic)));
    }
    // A vector's values: as a rule all of them lie inside the window, which its largest (NaN if
    // one is) and its smallest tell.
    template <int kPer>
    __device__ __forceinline__ void take_vector(const float (&v)[kPer], uint32_t column, const SeenBits &skip) {
        float high = v[0], low = v[0];
#pragma unroll
        for (int j = 1; j < kPer; j++) {
            asm("max.NaN.f32 %0, %0, %1;" : "+f"(high) : "f"(v[j]));
            low = fminf(low, v[j]);
        }
        if (high <= window.top && low >= window.bottom) {
            if (!kPenalised) found.best = fmaxf(found.best, high);
#pragma unroll
            for (int j = 0; j < kPer; j++) count(v[j]);
        } else {
#pragma unroll 1
            for (int j = 0; j < kPer; j++) take(pick_element(v, j), column + j, skip);
        }
    }
    // `skip`: columns whose value outside the window is not the row's (a seen id's raw logit)
    __device__ __forceinline__ void take(float v, uint32_t column, const SeenBits &skip) {
        if (v >= window.bottom && v <= window.top) {
            if (!kPenalised) found.best = fmaxf(found.best, v);
            count(v);
        } else if (is_nonfinite(v)) {
            found.lost++;
        } else {
            if (v > window.top) {
                ShortMemory &m = short_memory();
                found.above++;
                if (skip.test(column)) return;
                found.best = fmaxf(found.best, v);
                const uint32_t slot = atomicAdd(team.at(&m.state.over_count, 0), 1u);
                if (slot < kOverCap) {
                    team.at(m.over_value, 0)[slot] = v;
                    team.at(m.over_id, 0)[slot] = column;
                }
            } else {
                found.below++;
                if (v > found.best && !skip.test(column)) found.best = v;
            }
        }
    }
    // takes a counted value back (sums modulo 2^32: nothing of it stays)
    __device__ __forceinline__ void uncount(float v) {
        ShortMemory &m = short_memory();
        float f;
        const uint32_t at = swizzled(window.slot(v, f));
        atomicAdd(&m.first[at], 0u - __float_as_uint(__fmaf_rn(f, P::kFirstUnit, kMagic)));
        atomicAdd(&m.second[at], 0u - __float_as_uint(__fmaf_rn(__fmul_rn(f, f), P::kSecondUnit, P::kSecondMagic)));
    }
    __device__ __forceinline__ void take_back(float v) {
        if (v >= window.bottom && v <= window.top) {
            uncount(v);
        } else if (is_nonfinite(v)) {
            found.lost--;
        } else if (v > window.top) {
            found.above--;
        } else {
            found.below--;
        }
    }
};

template <typename T, class P, bool kPenalised>
__device__ __noinline__ Findings count_logits(const T *columns, uint32_t lo, uint32_t n, const Window window,
                                              const Team team, const SeenBits seen) {
    Counter<P, kPenalised> counter(window, team);
    walk_logits<T>(
        columns + lo, n,
        [&](const float (&v)[Vector<T>::kPer], uint32_t c) { counter.take_vector(v, lo + c, seen); },
        [&](float v, uint32_t c) { counter.take(v, lo + c, seen); });
    return counter.found;
}

// Every column in [lo, lo + n) the row's history has seen: visit(column, raw, penalised, slot),
// slots numbered from 0 (state.seen_count says how many; zeroed by the caller).  A warp takes
// 32 words of the bitmap at a time and lists the columns whose bits are up, so that the lanes
// share them evenly however they lie.  All threads call; the lists' memory holds the queues.
template <typename T, class Visit>
__device__ __forceinline__ void visit_seen(const NucleusParams &p, uint32_t row, const SamplerConfig &cfg, uint32_t lo,
                                           uint32_t n, Visit visit) {
    ShortMemory &m = short_memory();
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    constexpr uint32_t kWarps = kNucleusWarps;
    static_assert(offsetof(ShortMemory, lanes) - offsetof(ShortMemory, lists) >= kWarps * 1024 * sizeof(uint16_t),
                  "a queue of 1024 columns per warp");
    if (n == 0) return;  // (a CTA without columns does not begin at a multiple of 64)
    uint16_t *queue = reinterpret_cast<uint16_t *>(&m.lists) + warp * 1024u;
    const T *columns = static_cast<const T *>(p.logits) + (size_t)row * p.row_stride;
    const Repetition repetition = make_repetition(cfg.repetition_penalty);
    const float flat_offset = penalty_offset(1u, cfg.presence_penalty, cfg.frequency_penalty);
    for (uint32_t split = lo / p.split_len; split < p.splits && split * p.split_len < lo + n; split++) {
        const uint32_t split_lo = split * p.split_len;
        const uint32_t from = max(lo, split_lo), to = min(lo + n, min(split_lo + p.split_len, p.vocab));
        const size_t unit = (size_t)row * p.splits + split;
        const uint32_t flags = reinterpret_cast<const uint2 *>(p.history_meta)[unit].x;
        if (!(flags & 1u)) continue;
        const HistoryView history = make_history_view(
            const_cast<uint32_t *>(p.history_global) + unit * p.history_stride_words, p.bitmap_words,
            p.count_capacity, p.dense_wide != 0);
        // (`from` is a multiple of 64 columns, and so is where a split begins)
        const uint32_t word_end = (to - split_lo + 31u) / 32u;
        uint32_t word = (from - split_lo) / 32u + warp * 32u + lane;
        uint32_t bits = word < word_end ? history.bitmap[word] : 0u;
        uint32_t next_rank = flags & 2u ? history.running[min(word - lane, word_end - 1u)] : 0u;
        for (uint32_t base = (from - split_lo) / 32u + warp * 32u; base < word_end; base += kWarps * 32u) {
            const uint32_t ahead = word + kWarps * 32u;
            const uint32_t next_bits = ahead < word_end ? history.bitmap[ahead] : 0u;
            const uint32_t rank0 = next_rank;
            if (flags & 2u) next_rank = history.running[min(base + kWarps * 32u, word_end - 1u)];
            const uint32_t mine = __popc(bits);
            uint32_t incl = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t up = __shfl_up_sync(kFullMask, incl, d);
                if (lane >= (uint32_t)d) incl += up;
            }
            const uint32_t total = __shfl_sync(kFullMask, incl, 31);
            uint32_t slot0 = 0;
            if (lane == 0 && total != 0) slot0 = atomicAdd(&m.state.seen_count, total);
            slot0 = __shfl_sync(kFullMask, slot0, 0);
            for (uint32_t rest = bits, at = incl - mine; rest != 0; rest &= rest - 1)
                queue[at++] = (uint16_t)(lane * 32u + (uint32_t)__ffs(rest) - 1u);
            __syncwarp();
            constexpr int kBatch = 8;  // columns per lane and trip, loaded before any is used
            const uint32_t column0 = split_lo + base * 32u;
            for (uint32_t i0 = lane; i0 < total; i0 += 32 * kBatch) {
                uint32_t times[kBatch];
                float raw[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; q++) {
                    const uint32_t i = i0 + 32 * q;
                    raw[q] = 0.0f;
                    times[q] = 1;
                    if (i < total) {
                        raw[q] = Vector<T>::one(columns + column0 + queue[i]);
                        if (flags & 2u) {
                            const uint32_t at = min(rank0 + i, history.capacity - 1u);
                            times[q] = history.wide ? static_cast<const uint32_t *>(history.dense)[at]
                                                    : static_cast<const uint16_t *>(history.dense)[at];
                        }
                    }
                }
#pragma unroll
                for (int q = 0; q < kBatch; q++) {
                    const uint32_t i = i0 + 32 * q;
                    if (i >= total) break;
                    const float offset = flags & 2u ? penalty_offset(times[q], cfg.presence_penalty, cfg.frequency_penalty)
                                                    : flat_offset;
                    visit(column0 + queue[i], raw[q], penalise_with_offset(raw[q], offset, repetition), slot0 + i);
                }
            }
            __syncwarp();
            word = ahead;
            bits = next_bits;
        }
    }
}

// Largest value under `bottom` among the CTA's columns, raw or (the `listed` seen ones) penalised:
// a seen column's raw logit may be the one.  All threads call.
template <typename T>
__device__ __noinline__ float largest_under(const T *columns, uint32_t lo, uint32_t n, float bottom, const float2 *seen,
                                            uint32_t listed) {
    ShortShared &ss = short_memory().state;
    float best = __uint_as_float(0xff800000u);
    auto look = [&](float v) { best = v < bottom ? fmaxf(best, v) : best; };
    walk_logits<T>(
        columns + lo, n,
        [&](const float (&v)[Vector<T>::kPer], uint32_t) {
#pragma unroll
            for (int j = 0; j < Vector<T>::kPer; j++) look(v[j]);
        },
        [&](float v, uint32_t) { look(v); });
    for (uint32_t i = threadIdx.x; i < listed; i += kNucleusThreads) look(seen[i].x);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) best = fmaxf(best, __shfl_xor_sync(kFullMask, best, d));
    __syncthreads();
    if (lane_id() == 0) ss.sample_max[threadIdx.x >> 5] = best;
    __syncthreads();
    for (uint32_t w = 0; w < (uint32_t)kNucleusWarps; w++) best = fmaxf(best, ss.sample_max[w]);
    return best;
}

// After the raw logits have been counted: every seen column's raw value is taken back and its
// penalised value counted instead, and kept with its column for the second pass.
template <typename T, class P>
__device__ __noinline__ Findings amend_seen(const NucleusParams &p, uint32_t row, const SamplerConfig cfg, uint32_t lo,
                                            uint32_t n, float2 *seen, const Window window, const Team team) {
    Counter<P, true> counter(window, team);
    const SeenBits all_listed = {nullptr, 0, 1};
    visit_seen<T>(p, row, cfg, lo, n, [&](uint32_t column, float raw, float penalised, uint32_t slot) {
        if (fmaxf(raw, penalised) <= window.top && fminf(raw, penalised) >= window.bottom && raw == raw && penalised == penalised) {
            counter.uncount(raw);
            counter.count(penalised);
        } else {
            counter.take_back(raw);
            counter.take(penalised, column, all_listed);
        }
        seen[slot] = make_float2(penalised, __uint_as_float(column));
    });
    return counter.found;
}

// The penalised row in scratch memory, for the long way.  Returns the thread's largest finite raw logit.
template <typename T>
__device__ __noinline__ float write_scratch(const NucleusParams &p, uint32_t row, const SamplerConfig cfg, uint32_t lo,
                                           uint32_t n, bool penalised, float *values) {
    const T *columns = static_cast<const T *>(p.logits) + (size_t)row * p.row_stride;
    constexpr int kPer = Vector<T>::kPer;
    float best = __uint_as_float(0xff800000u);
    walk_logits<T>(
        columns + lo, n,
        [&](const float (&v)[kPer], uint32_t c) {
            float *to = values + lo + c;
#pragma unroll
            for (int j = 0; j < kPer; j++) best = is_nonfinite(v[j]) ? best : fmaxf(best, v[j]);
            if ((c & 3u) == 0) {  // (`lo` is a multiple of 64)
#pragma unroll
                for (int j = 0; j < kPer; j += 4) *reinterpret_cast<float4 *>(to + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < kPer; j++) to[j] = v[j];
            }
        },
        [&](float v, uint32_t c) {
            values[lo + c] = v;
            best = is_nonfinite(v) ? best : fmaxf(best, v);
        });
    __syncthreads();
    if (penalised)
        visit_seen<T>(p, row, cfg, lo, n, [&](uint32_t column, float, float value, uint32_t) { values[column] = value; });
    return best;
}

// Sum over the warp of masses below 2^60 (4,095 members of 2^44 weigh less than 2^57).
__device__ __forceinline__ unsigned long long warp_sum_mass(unsigned long long mass) {
    const uint32_t low = __reduce_add_sync(kFullMask, (uint32_t)mass & 0xfffffu);
    const uint32_t middle = __reduce_add_sync(kFullMask, (uint32_t)(mass >> 20) & 0xfffffu);
    const uint32_t high = __reduce_add_sync(kFullMask, (uint32_t)(mass >> 40));
    return ((unsigned long long)high << 40) + ((unsigned long long)middle << 20) + low;
}

// The factors of the moments in a bucket's masses, by kind of bucket.
template <class P>
struct MomentFactors {
    double raw1, raw2, tempered1, tempered2;
    __device__ __forceinline__ MomentFactors(const Window &window, uint32_t slot, double inv_t) {
        float width;
        window.middle_of(slot, width);
        const double c = (double)width, ct = c * inv_t;
        raw1 = c * (1.0 + c * c * 0.025) / (double)P::kFirstUnit;  // 0.15 / 6
        tempered1 = ct * (1.0 + ct * ct * 0.025) / (double)P::kFirstUnit;
        raw2 = 0.5 * c * c / (double)P::kSecondUnit;
        tempered2 = 0.5 * ct * ct / (double)P::kSecondUnit;
    }
};
__device__ __forceinline__ uint32_t kind_of_group(uint32_t group) {
    return group < kFineSlots / 32 ? 0u : group < (kFineSlots + kMiddleSlots) / 32 ? 1u : 2u;
}

struct SlotMass {
    unsigned long long raw, tempered;
    uint32_t count;
};
// `raw_weight`, `tempered_weight`: the weights of the slot's middle, times 2^bits.
template <class P>
__device__ __forceinline__ SlotMass slot_mass(uint32_t first, uint32_t second, const MomentFactors<P> &k,
                                              double raw_weight, double tempered_weight) {
    SlotMass s;
    s.count = P::count(second);
    const double n = (double)s.count, f = (double)P::sum_f(first, s.count), ff = (double)P::sum_ff(second);
    // (an empty bucket: three zeros)
    s.raw = __double2ull_rn(fma(k.raw2, ff, fma(k.raw1, f, n)) * raw_weight);
    s.tempered = __double2ull_rn(fma(k.tempered2, ff, fma(k.tempered1, f, n)) * tempered_weight);
    return s;
}

// Masses of the short way are 2^-44 fixed point (every one of 8,192 buckets is rounded to it, which
// at 2^-40 was the largest error for peaked rows), unless a row has so many columns that their sum
// might not fit: then 2^-40.
constexpr uint32_t kFinestVocab = 1u << 18;

// Masses and counts of this CTA's groups into m.raw, m.tempered, m.count (place 1 + group), and the
// weights they are made with into m.edges, m.lanes; state.counted gets the sum of all counts.  All
// threads call; ends synced.
template <class P>
__device__ __noinline__ void group_masses(const Window window, double best, double inv_t, int bits) {
    ShortMemory &m = short_memory();
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    constexpr uint32_t kWarps = kNucleusWarps;
    static_assert(kNucleusThreads == 2 * kGroups && kGroups == 16 * kWarps, "an exponential per thread, 16 groups per warp");
    static_assert(kFineSlots == 8 * 32 * kWarps && kMiddleSlots == 4 * 32 * kWarps, "four groups abreast are of one kind");
    {
        const uint32_t group = tid % kGroups, tempered = tid / kGroups;
        const double x = window.middle(group * 32u) - best;
        m.edges[tempered][group] = exp(tempered ? x * inv_t : x) * (double)(1ull << bits);
        if (tid < 192u) {
            const uint32_t kind = tid / 32u % 3u;
            float width;
            window.middle_of(kind == 0 ? 0u : kind == 1 ? kFineSlots : kFineSlots + kMiddleSlots, width);
            const double away = -(double)lane * (double)width;
            m.lanes[tid / 96u][kind][lane] = exp(tid < 96u ? away : away * inv_t);
        }
    }
    __syncthreads();
    uint32_t counted = 0;
    // four groups abreast: their chains of conversions and reductions overlap
#pragma unroll 1
    for (uint32_t j = 0; j < 16; j += 4) {
        const uint32_t group0 = j * kWarps + warp, kind = kind_of_group(group0);
        uint32_t first[4], second[4], any = 0;
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) {
            const uint32_t at = swizzled((group0 + q * kWarps) * 32u + lane);
            first[q] = m.first[at];
            second[q] = m.second[at];
            any |= second[q];
        }
        any = __any_sync(kFullMask, any != 0);
        if (!any) {
            if (lane < 4) {
                const uint32_t place = 1 + group0 + lane * kWarps;
                m.raw[place] = m.tempered[place] = 0;
                m.count[place] = 0;
            }
            continue;
        }
        const MomentFactors<P> k(window, group0 * 32u, inv_t);
        const double raw_lane = m.lanes[0][kind][lane], tempered_lane = m.lanes[1][kind][lane];
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) {
            const uint32_t group = group0 + q * kWarps;
            const SlotMass s = slot_mass<P>(first[q], second[q], k, m.edges[0][group] * raw_lane, m.edges[1][group] * tempered_lane);
            const unsigned long long raw = warp_sum_mass(s.raw), tempered = warp_sum_mass(s.tempered);
            const uint32_t count = __reduce_add_sync(kFullMask, s.count);
            if (lane == 0) {
                m.raw[1 + group] = raw;
                m.tempered[1 + group] = tempered;
                m.count[1 + group] = count;
            }
            counted += count;
        }
    }
    if (lane == 0) atomicAdd(&m.state.counted, counted);
    __syncthreads();
}

// Among the 32 slots of a group, summed over the team: the first at which the running raw (or
// tempered) mass reaches `target` (strict: exceeds it); the last with members when none does.
// One warp calls.
template <class P>
__device__ __noinline__ SlotHit find_slot(const Team team, const Window window, uint32_t group,
                                          double inv_t, unsigned long long raw_before,
                                          unsigned long long tempered_before, uint32_t count_before,
                                          unsigned long long target, bool tempered, bool strict) {
    ShortMemory &m = short_memory();
    const uint32_t lane = lane_id();
    const MomentFactors<P> k(window, group * 32u, inv_t);
    const uint32_t kind = kind_of_group(group);
    const double raw_weight = m.edges[0][group] * m.lanes[0][kind][lane];
    const double tempered_weight = m.edges[1][group] * m.lanes[1][kind][lane];
    const uint32_t at = swizzled(group * 32u + lane);
    SlotMass mine;
    mine.raw = mine.tempered = 0;
    mine.count = 0;
    uint32_t far_first[kMostTeam], far_second[kMostTeam];
#pragma unroll
    for (uint32_t r = 0; r < kMostTeam; r++) {
        far_first[r] = r < team.size ? *team.at(&m.first[at], r) : 0u;
        far_second[r] = r < team.size ? *team.at(&m.second[at], r) : 0u;
    }
#pragma unroll
    for (uint32_t r = 0; r < kMostTeam; r++) {
        if (r >= team.size) break;
        const SlotMass s = slot_mass<P>(far_first[r], far_second[r], k, raw_weight, tempered_weight);
        mine.raw += s.raw;
        mine.tempered += s.tempered;
        mine.count += s.count;
    }
    unsigned long long raw = mine.raw, other = mine.tempered;
    uint32_t count = mine.count;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long up_raw = __shfl_up_sync(kFullMask, raw, d), up_other = __shfl_up_sync(kFullMask, other, d);
        const uint32_t up_count = __shfl_up_sync(kFullMask, count, d);
        if (lane >= (uint32_t)d) {
            raw += up_raw;
            other += up_other;
            count += up_count;
        }
    }
    const unsigned long long here = tempered ? tempered_before + other : raw_before + raw;
    const uint32_t reached = __ballot_sync(kFullMask, strict ? here > target : here >= target);
    const uint32_t peopled = __ballot_sync(kFullMask, mine.count != 0);
    const int lead = reached ? __ffs(reached) - 1 : (peopled ? 31 - __clz(peopled) : 0);
    SlotHit hit;
    hit.slot = group * 32u + (uint32_t)lead;
    hit.count = __shfl_sync(kFullMask, mine.count, lead);
    hit.count_before = count_before + __shfl_sync(kFullMask, count - mine.count, lead);
    hit.raw_before = raw_before + __shfl_sync(kFullMask, raw - mine.raw, lead);
    hit.tempered = __shfl_sync(kFullMask, mine.tempered, lead);
    hit.tempered_before = tempered_before + __shfl_sync(kFullMask, other - mine.tempered, lead);
    return hit;
}

// cumulative / sum >= top_p  <=>  cumulative >= top_p * sum
__device__ __forceinline__ unsigned long long mass_target_of(double top_p, unsigned long long total) {
    const unsigned long long t = (unsigned long long)ceil(top_p * (double)total);
    return t > total ? total : t;
}
// the first element whose cumulative weight exceeds draw = u * sum
__device__ __forceinline__ unsigned long long draw_target_of(double draw_at, unsigned long long total) {
    return (unsigned long long)floor(draw_at * (double)total);
}

// The window goes where all but a few hundred values lie under its top, those above it being kept
// one by one.  First CTA, with the running sums of the counts; all its threads call.
__device__ __noinline__ void place_anew(const Window window, bool sensible) {
    Plan &plan = short_memory().state.plan;
    const uint32_t tid = threadIdx.x;
    const uint32_t places = __syncthreads_count(tid < kPlaces && short_memory().count[tid] <= kBodyRank);  // (the first ones)
    if (tid == 0) {
        float top = window.top;
        if (places > 0 && places < kPlaces) top = window.highest((places - 1) * 32u);
        plan.reference = top - kWindowMargin / window.sharp;
        plan.verdict = sensible ? kElsewhere : kLongWay;
    }
    __syncthreads();
}

// What a place (not the first) adds to the square of the masses' error, less what weights rounded to
// 2^-32 of themselves would: its members are off independently of one another, each by its weight
// times the error of a bucket that is c wide.  `mass`: its running sums over the places.  `middle`:
// that of the place's first bucket, in widths -- raw bf16 values have at most eight significant bits
// and lie on their bucket's middle unless they are within 128 widths of 0.  (A row's largest weight
// is no rounded one, and is left out.)
template <class P>
__device__ __forceinline__ float place_error(uint32_t place, float c, int middle, const unsigned long long *mass, float largest) {
    constexpr float kSecond = 0.5f * 0x1p-14f * 0.28867513f, kThird = P::kThirdError / 6.0f, kWeight = 0x1p-32f * 0.28867513f;
    const uint32_t *counts = short_memory().count;
    const uint32_t before = place ? counts[place - 1] : 0u, count = counts[place] - before;
    const float weight = __ull2float_rn(mass[place] - (place ? mass[place - 1] : 0ull));
    const float second = c * c * kSecond, third = c * c * c * kThird;
    const bool exact = P::kCoarser && (middle < -128 || middle > 128 + 31);
    const float off = count && !exact ? (second * second + third * third) * weight * weight / (float)count : 0.0f;
    const float others = before ? weight : weight - largest, rest = (float)(before ? count : count - 1u);
    return off - (others > 0.0f && rest > 0.0f ? kWeight * kWeight * others * others / rest : 0.0f);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFullMask, v, d);
    return v;
}

// The first CTA adds the team's masses up and finds the buckets the answer lies in.  `error`: how
// far off the masses may be.  All its threads call; ends synced.
template <class P>
__device__ __noinline__ void make_plan(const Team team, const Window window, float best, double top_p, double inv_t,
                                       double draw_at, int bits, double error) {
    ShortMemory &m = short_memory();
    ShortShared &ss = m.state;
    const NucleusShared &sh = m.scan;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t over = min(ss.over_count, kOverCap);
    double unseen = 0.0;
    for (uint32_t r = 0; r < team.size; r++) unseen += team.at(&ss.share, r)->unseen;
    const bool crowded = !(unseen < INFINITY);
    // place 0: the values above the window, each with its own weights
    if (warp == kNucleusWarps - 1) {
        unsigned long long raw = 0, tempered = 0;
        for (uint32_t i = lane; i < over; i += 32) {
            const double x = (double)m.over_value[i] - (double)best;
            raw += exp_fixed(x, sh.table, bits);
            tempered += exp_fixed(x * inv_t, sh.table, bits);
        }
        raw = warp_sum_mass(raw);
        tempered = warp_sum_mass(tempered);
        if (lane == 0) {
            m.raw[0] = raw;
            m.tempered[0] = tempered;
            m.count[0] = over;
        }
    }
    __syncthreads();
    unsigned long long raw = 0, tempered = 0;
    uint32_t count = 0;
    if (tid < kPlaces) {
        raw = m.raw[tid];
        tempered = m.tempered[tid];
        count = m.count[tid];
        unsigned long long far_raw[kMostTeam], far_tempered[kMostTeam];  // (all on their way before one is used)
        uint32_t far_count[kMostTeam];
#pragma unroll
        for (uint32_t r = 1; r < kMostTeam; r++) {
            const bool there = tid > 0 && r < team.size;
            far_raw[r] = there ? *team.at(&m.raw[tid], r) : 0ull;
            far_tempered[r] = there ? *team.at(&m.tempered[tid], r) : 0ull;
            far_count[r] = there ? *team.at(&m.count[tid], r) : 0u;
        }
#pragma unroll
        for (uint32_t r = 1; r < kMostTeam; r++) {
            raw += far_raw[r];
            tempered += far_tempered[r];
            count += far_count[r];
        }
    }
    const unsigned long long own_raw = raw, own_tempered = tempered;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long up_raw = __shfl_up_sync(kFullMask, raw, d), up_tempered = __shfl_up_sync(kFullMask, tempered, d);
        const uint32_t up_count = __shfl_up_sync(kFullMask, count, d);
        if (lane >= (uint32_t)d) {
            raw += up_raw;
            tempered += up_tempered;
            count += up_count;
        }
    }
    if (lane == 31) {
        ss.scan_raw[warp] = raw;
        ss.scan_tempered[warp] = tempered;
        ss.scan_count[warp] = count;
    }
    __syncthreads();
    unsigned long long total_raw = 0;
    constexpr uint32_t kScanWarps = (kPlaces + 31) / 32;
#pragma unroll
    for (uint32_t w = 0; w < kScanWarps; w++) {
        const unsigned long long more = ss.scan_raw[w], more_tempered = ss.scan_tempered[w];
        const uint32_t more_count = ss.scan_count[w];
        total_raw += more;
        raw += w < warp ? more : 0ull;
        tempered += w < warp ? more_tempered : 0ull;
        count += w < warp ? more_count : 0u;
    }
    const unsigned long long cut_target = mass_target_of(top_p, total_raw);
    if (tid < kPlaces) {
        m.raw[tid] = raw;
        m.tempered[tid] = tempered;
        m.count[tid] = count;
        if (raw - own_raw < cut_target && raw >= cut_target) ss.cut_place = tid;  // exactly one thread when there is any mass
    }
    __syncthreads();
    if (crowded || total_raw == 0) {
        place_anew(window, crowded && !P::kCoarser);  // (the other packing takes fewer members)
        return;
    }
    const uint32_t cut_place = ss.cut_place;
    constexpr uint32_t kErrorWarp = 2, kErrorWarps = kScanWarps;
    static_assert(kErrorWarp + kErrorWarps <= (uint32_t)kNucleusWarps, "a thread per place beside the warps that look for slots");
    if (warp >= kErrorWarp && warp < kErrorWarp + kErrorWarps) {
        // meanwhile: how far off are the masses?
        const uint32_t place = (warp - kErrorWarp) * 32 + lane;
        const float largest = (float)(1ull << bits);
        float width = 0.0f, raw_error = 0.0f, tempered_error = 0.0f;
        const int middle = place != 0 ? window.middle_of((place - 1) * 32u, width) : 0;
        if (place < kPlaces) raw_error = place_error<P>(place, width, middle, m.raw, largest);
        if (place <= cut_place) tempered_error = place_error<P>(place, width * (float)inv_t, middle, m.tempered, largest);
        raw_error = warp_sum(raw_error);
        tempered_error = warp_sum(tempered_error);
        if (lane == 0) {
            ss.raw_error[warp - kErrorWarp] = raw_error;
            ss.tempered_error[warp - kErrorWarp] = tempered_error;
        }
    }
    if (warp == 0) {
        SlotHit cut;
        cut.slot = 0;
        cut.count = over;
        cut.count_before = 0;
        cut.raw_before = cut.tempered_before = 0;
        cut.tempered = m.tempered[0];
        if (cut_place != 0)
            cut = find_slot<P>(team, window, cut_place - 1, inv_t, m.raw[cut_place - 1],
                               m.tempered[cut_place - 1], m.count[cut_place - 1], cut_target, false, false);
        if (lane == 0) {
            ss.plan.cut = cut_place == 0 ? 0u : 1u + cut.slot;
            ss.plan.cut_target = cut_target;
            ss.plan.cut_before = cut.raw_before;
            ss.plan.cut_tempered_before = cut.tempered_before;
            ss.plan.cut_rank_before = cut.count_before;
            ss.plan.cut_members = cut.count;
            ss.plan.pick_before = cut.tempered;  // (handed on to the next step)
            ss.pick_place[0] = ss.pick_place[1] = cut_place;
        }
    }
    __syncthreads();
    // The nucleus weighs at least what lies above the cut's bucket and at most that and the
    // bucket: the draw lands between the two targets.
    const unsigned long long least = ss.plan.cut_tempered_before, most = least + ss.plan.pick_before;
    const unsigned long long target_first = draw_target_of(draw_at, least), target_last = draw_target_of(draw_at, most);
    if (tid < kPlaces && tid < cut_place) {
        const unsigned long long before = tempered - own_tempered;
        if (before <= target_first && tempered > target_first) ss.pick_place[0] = tid;
        if (before <= target_last && tempered > target_last) ss.pick_place[1] = tid;
    }
    __syncthreads();
    __shared__ uint32_t ends[2], ends_count[2];
    __shared__ unsigned long long ends_before;
    if (warp == 2) {
        // Are the masses good enough?  (Squares are compared; the nucleus weighs `most`, tempered.
        // Values of raw bf16 rows tie, and ties are off by the same.)
        float raw_off = 0.0f, tempered_off = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < kErrorWarps; w++) {
            raw_off += ss.raw_error[w];
            tempered_off += ss.tempered_error[w];
        }
        if (P::kCoarser) error *= 0.05;
        const double raw_allowed = error * (double)total_raw, tempered_allowed = error * (double)most;
        if (lane == 0)
            ss.poor = (double)raw_off > raw_allowed * raw_allowed ||
                      (double)tempered_off > tempered_allowed * tempered_allowed ||
                      unseen * (double)(1ull << bits) > raw_allowed;
    }
    if (warp < 2) {
        const uint32_t place = ss.pick_place[warp];
        const unsigned long long target = warp == 0 ? target_first : target_last;
        uint32_t at = 0, edge = warp == 0 ? 0u : over;
        unsigned long long before = 0;
        if (place != 0) {
            const SlotHit hit = find_slot<P>(team, window, place - 1, inv_t, m.raw[place - 1],
                                             m.tempered[place - 1], m.count[place - 1], target, true, true);
            at = 1u + hit.slot;
            before = hit.tempered_before;
            edge = warp == 0 ? hit.count_before : hit.count_before + hit.count;
            if (at > ss.plan.cut) {  // (nothing below the cut takes part)
                at = ss.plan.cut;
                before = ss.plan.cut_tempered_before;
                edge = warp == 0 ? ss.plan.cut_rank_before : ss.plan.cut_rank_before + ss.plan.cut_members;
            }
        }
        if (lane == 0) {
            ends[warp] = at;
            ends_count[warp] = edge;
            if (warp == 0) ends_before = before;
        }
    }
    __syncthreads();
    if (ss.poor) {
        place_anew(window, true);
        return;
    }
    if (tid == 0) {
        ss.plan.pick_first = ends[0];
        ss.plan.pick_last = ends[1];
        ss.plan.pick_before = ends_before;
        ss.plan.pick_members = ends_count[1] - ends_count[0];
        ss.plan.verdict = (ss.plan.cut != 0 && ss.plan.cut_members > kCutCap) || ss.plan.pick_members > kPickCap ? kLongWay : kDone;
    }
    __syncthreads();
}

// The second pass: the members of the plan's buckets onto the first CTA's two lists.
struct Gatherer {
    const Team team;
    float cut_low, cut_high, pick_low, pick_high;  // whole buckets, both ends included

    __device__ __forceinline__ Gatherer(const Team &team_, const Window &w) : team(team_) {
        const Plan *plan = team.at(&short_memory().state.plan, 0);
        cut_low = pick_low = __uint_as_float(0x7f800000u);  // nothing
        cut_high = pick_high = __uint_as_float(0xff800000u);
        if (plan->cut != 0) {
            cut_low = w.lowest(plan->cut - 1);
            cut_high = w.highest(plan->cut - 1);
        }
        if (plan->pick_last != 0) {
            pick_low = w.lowest(plan->pick_last - 1);
            pick_high = plan->pick_first != 0 ? w.highest(plan->pick_first - 1) : w.top;
        }
    }
    __device__ __forceinline__ bool wanted(float v) const {
        return (v >= cut_low && v <= cut_high) || (v >= pick_low && v <= pick_high);
    }
    // `skip`: columns that do not count
    __device__ __forceinline__ void put(float v, uint32_t column, const SeenBits &skip) const {
        if (skip.test(column)) return;
        ShortMemory &m = short_memory();
        if (v >= cut_low && v <= cut_high) {
            const uint32_t slot = atomicAdd(team.at(&m.state.cut_count, 0), 1u);
            if (slot < kCutCap) {
                team.at(m.lists.cut_value, 0)[slot] = v;
                team.at(m.lists.cut_id, 0)[slot] = column;
            }
        }
        if (v >= pick_low && v <= pick_high) {
            const uint32_t slot = atomicAdd(team.at(&m.state.pick_count, 0), 1u);
            if (slot < kPickCap) {
                team.at(m.lists.pick_value, 0)[slot] = v;
                team.at(m.lists.pick_id, 0)[slot] = column;
            }
        }
    }
    template <int kPer>
    __device__ __forceinline__ void take_vector(const float (&v)[kPer], uint32_t column, const SeenBits &skip) const {
        uint32_t hits = 0;
#pragma unroll
        for (int j = 0; j < kPer; j++) hits |= wanted(v[j]) ? 1u << j : 0u;
#pragma unroll 1
        for (; hits != 0; hits &= hits - 1) {
            const int j = __ffs(hits) - 1;
            put(pick_element(v, j), column + j, skip);
        }
    }
};

// (`listed` seen columns with their penalised values; their raw logits do not count)
template <typename T>
__device__ __noinline__ void gather_members(const T *columns, uint32_t lo, uint32_t n, const Window window, const Team team,
                                            const SeenBits bits, const float2 *seen, uint32_t listed) {
    const Gatherer gather(team, window);
    walk_logits<T>(
        columns + lo, n, [&](const float (&v)[Vector<T>::kPer], uint32_t c) { gather.take_vector(v, lo + c, bits); },
        [&](float v, uint32_t c) {
            if (gather.wanted(v)) gather.put(v, lo + c, bits);
        });
    const SeenBits all_listed = {nullptr, 0, 1};
    constexpr int kBatch = 4;
    for (uint32_t i0 = threadIdx.x; i0 < listed; i0 += kBatch * kNucleusThreads) {
        float2 pair[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
            const uint32_t i = i0 + q * kNucleusThreads;
            pair[q] = i < listed ? seen[i] : make_float2(__uint_as_float(0x7fc00000u), 0.0f);
        }
#pragma unroll
        for (int q = 0; q < kBatch; q++)
            if (gather.wanted(pair[q].x)) gather.put(pair[q].x, __float_as_uint(pair[q].y), all_listed);
    }
}

// The first CTA orders the gathered members and reports the row; leaves the verdict in the plan.
// All its threads call; ends synced.
__device__ __noinline__ void finish_short(float best, double inv_t, double draw_at, int bits, uint32_t row,
                                          const SelectOutput &out) {
    ShortMemory &m = short_memory();
    ShortShared &ss = m.state;
    NucleusShared &sh = m.scan;
    const uint32_t tid = threadIdx.x;
    const Plan plan = ss.plan;
    const uint32_t over = min(ss.over_count, kOverCap);
    // (the lists hold what the plan has counted, or the row is not this way's to answer)
    const uint32_t cut_listed = plan.cut == 0 ? over : ss.cut_count;
    const uint32_t pick_listed = ss.pick_count + (plan.pick_first == 0 ? over : 0u);
    if (cut_listed != plan.cut_members || pick_listed != plan.pick_members) {
        __syncthreads();
        if (tid == 0) ss.plan.verdict = kLongWay;
        __syncthreads();
        return;
    }
    // the ordering's work arrays lie where the buckets were
    OrderWork work;
    work.weight = reinterpret_cast<unsigned long long *>(m.first);
    work.sorted_value = reinterpret_cast<float *>(work.weight + kOrderCap);
    work.sorted_id = reinterpret_cast<uint32_t *>(work.sorted_value + kOrderCap);
    static_assert(kOrderCap * 16 <= sizeof(m.first) + sizeof(m.second), "the ordering fits over the buckets");
    work.value = plan.cut == 0 ? m.over_value : m.lists.cut_value;
    work.id = plan.cut == 0 ? m.over_id : m.lists.cut_id;
    Nucleus nucleus;
    nucleus.everything = true;
    nucleus.key = nucleus.id = 0;
    unsigned long long tempered_inside = 0;
    // (one copy of the ordering's code for both turns)
    Position cut, pick;
    cut.ok = pick.ok = false;
    unsigned long long weight_sum = 0;
    uint32_t members = plan.cut == 0 ? over : min(ss.cut_count, kCutCap);
#pragma unroll 1
    for (int turn = 0; turn < 2; turn++) {
        const Position found = order_members(sh, work, members, turn == 0 ? 1.0 : inv_t, best, nucleus,
                                             turn == 0 ? plan.cut_before : plan.pick_before,
                                             turn == 0 ? plan.cut_rank_before : 0u,
                                             turn == 0 ? plan.cut_target : draw_target_of(draw_at, weight_sum), turn != 0,
                                             false, inv_t, turn == 0 ? &tempered_inside : nullptr, bits);
        if (turn != 0) {
            pick = found;
            break;
        }
        cut = found;
        if (!cut.ok) break;
        nucleus.everything = false;
        nucleus.key = cut.key;
        nucleus.id = cut.id;
        weight_sum = plan.cut_tempered_before + tempered_inside;
        members = min(ss.pick_count, kPickCap);
        work.value = m.lists.pick_value;
        work.id = m.lists.pick_id;
        if (plan.pick_first == 0) {  // what lies above the window takes part
            const uint32_t more = min(over, kPickCap - members);
            for (uint32_t i = tid; i < more; i += kNucleusThreads) {
                m.lists.pick_value[members + i] = m.over_value[i];
                m.lists.pick_id[members + i] = m.over_id[i];
            }
            members += more;
        }
        __syncthreads();
    }
    const bool done = cut.ok && pick.ok && weight_sum != 0;
    if (done && tid == 0) {
        report_row(out, row, kOk, pick.id, pick.value);
        if (out.dbg_count) out.dbg_count[row] = cut.rank;  // nucleus size; the list itself is not dumped
    }
    if (tid == 0) ss.plan.verdict = done ? kDone : kLongWay;
    __syncthreads();
}

// One row's second half: masses, plan, gather, order.  All CTAs of the team call, with the
// buckets filled; returns the verdict.
template <typename T, class P>
__device__ __forceinline__ uint32_t locate_and_pick(const NucleusParams &p, const Team &team, const Window &window,
                                                    uint32_t row, uint32_t lo, uint32_t n, uint32_t counted,
                                                    const SeenBits &bits, const float2 *seen, float best, double top_p,
                                                    double inv_t, double draw_at, double error) {
    ShortShared &ss = short_memory().state;
    const int grid = p.vocab <= kFinestVocab ? 44 : 40;
    group_masses<P>(window, (double)best, inv_t, grid);
    if (threadIdx.x == 0 && ss.counted != counted) ss.share.unseen = INFINITY;
    team.sync();
    if (team.rank == 0) make_plan<P>(team, window, best, top_p, inv_t, draw_at, grid, error);
    team.sync();
    if (team.at(&ss.plan, 0)->verdict == kDone) {
        gather_members<T>(static_cast<const T *>(p.logits) + (size_t)row * p.row_stride, lo, n, window, team, bits, seen,
                          ss.seen_count);
        team.sync();
        if (team.rank == 0) finish_short(best, inv_t, draw_at, grid, row, p.out);
        team.sync();
    }
    return team.at(&ss.plan, 0)->verdict;
}

// ================================================================== the long way
//
// For rows the short way cannot take: the row with its penalties applied lies in the team's scratch
// memory, and every CTA of the team goes over its own columns again and again, step by step as the
// first CTA asks; what the steps leave (histograms, members of a bucket) the first CTA adds up.
//
// Buckets of equal width in the value itself, 1/256 wide and counted down from the row's maximum
// (bucket 0 holds the largest values; everything 16 below the maximum, where weights are below
// 2^-23, shares the last bucket).  Unlike the top bits of the float key this spreads real logit rows
// over hundreds of buckets, which keeps the shared-memory atomics apart.  One pass fills the
// histograms of both phases, a prefix sum finds the bucket in which the target is reached, a second
// pass gathers that bucket's members, which are ordered exactly.  A bucket too crowded for that
// is taken apart by its members' keys, and equal keys by their ids (descend).
//
// What bounds it: the passes' instruction issue, and latency where a row has one CTA.  Measured with 1 /
// 32 / 148 / 512 rows of 151,936 bf16 logits N(-10, 1.5^2), whose ties fill buckets: 381 / 572 / 1278 /
// 4181 us.  By the first CTA alone, one value in flight per thread in the descents and 64-bit adds in
// shared memory: 1887 / 1974 / 2146 / 6413; by a CTA of 1,024 threads a row: 1032 / 1270 / 1342 / 4522.
// Continuous rows of spread 0.03 315 / 366 / 828 / 2838 (1136 / 1150 / 1442 / 4492; 846 / 860 / 880 / 3423).

// Which values share a bucket.  (fp32 arithmetic: the bucket edges need not be exact, only the same
// in every pass and monotone in v, which one rounded subtraction and an exact scaling are.)
__device__ __forceinline__ uint32_t value_bucket(float v, float top) {
    const float below = __fmul_rn(__fsub_rn(top, v), 256.0f);  // >= 0
    return below >= (float)(kBuckets - 1) ? (uint32_t)(kBuckets - 1) : (uint32_t)below;
}

constexpr uint32_t kListCap = kOrderCap;  // members of a bucket that are ordered in shared memory

// Lies over the short way's memory; the ordering works where the masses were.
struct LongMemory {
    unsigned long long mass[kBuckets], other_mass[kBuckets];  // raw and tempered, or the one asked for
    uint32_t count[kBuckets];
    float value[kListCap];  // the first CTA's list
    uint32_t id[kListCap];
};
static_assert(sizeof(LongMemory) <= offsetof(ShortMemory, state), "the long way fits over the short way's memory");
static_assert(kOrderCap * 16 <= sizeof(LongMemory::mass), "the ordering fits over the masses");

// exp(x) for |x| <= 1/64 by its series to the sixth power (the next term is below 1e-16).
__device__ __forceinline__ double exp_small(double x) {
    double p = fma(x, 1.0 / 720.0, 1.0 / 120.0);
    p = fma(p, x, 1.0 / 24.0);
    p = fma(p, x, 1.0 / 6.0);
    p = fma(p, x, 0.5);
    p = fma(p, x, 1.0);
    return fma(p, x, 1.0);
}

// One CTA's part of a row in scratch memory.
struct LongWay {
    const Team team;
    const float *const values;  // of its columns
    const uint32_t lo, n;
    __device__ __forceinline__ LongMemory &memory() const { return *reinterpret_cast<LongMemory *>(&short_memory()); }

    template <class Visit>
    __device__ __forceinline__ void walk(Visit visit) const {
        const uint32_t first = lo;
        walk_row(values, n, [&](float v, uint32_t i) { visit(v, first + i); });
    }
    // The largest of the threads' values, into the CTA's share.
    __device__ __forceinline__ void share_largest(float best) const {
        ShortShared &ss = short_memory().state;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) best = fmaxf(best, __shfl_xor_sync(kFullMask, best, d));
        if (lane_id() == 0) ss.sample_max[threadIdx.x >> 5] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 0; w < kNucleusWarps; w++) best = fmaxf(best, ss.sample_max[w]);
            ss.share.best = best;
        }
    }
    __device__ __noinline__ void largest() const {
        float best = -INFINITY;
        walk([&](float v, uint32_t) {
            if (!is_nonfinite(v)) best = fmaxf(best, v);
        });
        share_largest(best);
    }
    // Per value bucket the count, the raw weights exp(v - top) and the tempered weights
    // exp((v - top) * inv_t) of its members.  A member's weight is taken relative to the bucket's
    // upper edge -- an argument of at most 1/256 (times inv_t), a short series instead of a full
    // exp() -- as 2^-32 fixed point, and summed in two 16-bit halves with 32-bit shared-memory adds
    // (a bucket of up to 65,535 members cannot overflow them; integer sums do not depend on the
    // order of arrival).  The rounding of one member is 2^-33 of a member's weight.  The last bucket
    // (everything 16 below the maximum) and the tempered weights for inv_t > 4 take the full exp().  A bucket with
    // more members than the sums take (heavy ties) is noted in the CTA's share.
    __device__ __noinline__ void weigh_both(const LongStep &step) const {
        LongMemory &m = memory();
        const NucleusShared &sh = short_memory().scan;
        const uint32_t tid = threadIdx.x;
        // the two mass arrays, seen as four arrays of 32-bit sums
        uint32_t *raw_low = reinterpret_cast<uint32_t *>(m.mass), *raw_high = raw_low + kBuckets;
        uint32_t *tempered_low = reinterpret_cast<uint32_t *>(m.other_mass), *tempered_high = tempered_low + kBuckets;
        for (uint32_t b = tid; b < kBuckets; b += kNucleusThreads) {
            m.mass[b] = 0;
            m.other_mass[b] = 0;
            m.count[b] = 0;
        }
        if (tid == 0) short_memory().state.share.unseen = 0.0;
        __syncthreads();
        const float top = step.top;
        const double inv_t = step.inv_t, top_d = (double)top;
        // (65,535 members 40 temperatures below the maximum weigh less than half a unit of the row's
        // 2^-40 fixed point: what they weigh tempered need not be known)
        const uint32_t weightless = (uint32_t)fmin(ceil(40.0 * 256.0 / inv_t), (double)kBuckets);
        const bool series = inv_t <= 4.0;  // (1/256) * inv_t <= 1/64
        constexpr double kOne = 4294967296.0;  // 2^32
        walk([&](float v, uint32_t) {
            if (is_nonfinite(v)) return;
            const uint32_t b = value_bucket(v, top);
            // v - (top - b/256): at most a bucket's width (and a rounding of the bucket's number) from 0
            const double x = ((double)v - top_d) + (double)b * (1.0 / 256.0);
            // (a weight of 1 and a rounding above it saturate at 2^32 - 1: half a unit, like any rounding)
            const bool last = b == (uint32_t)(kBuckets - 1);
            const uint32_t r = (uint32_t)min(last ? (exp_fixed(x, sh.table) + 128ull) >> 8
                                                  : __double2ull_rn(exp_small(x) * kOne), 0xffffffffull);
            atomicAdd(&raw_low[b], r & 0xffffu);
            atomicAdd(&raw_high[b], r >> 16);
            if (b < weightless) {
                const uint32_t t = (uint32_t)min(last || !series ? (exp_fixed(x * inv_t, sh.table) + 128ull) >> 8
                                                                 : __double2ull_rn(exp_small(x * inv_t) * kOne), 0xffffffffull);
                atomicAdd(&tempered_low[b], t & 0xffffu);
                atomicAdd(&tempered_high[b], t >> 16);
            }
            atomicAdd(&m.count[b], 1u);
        });
        __syncthreads();
        // the halves back together (every thread reads the sums of its buckets before any of them is
        // overwritten: the 64-bit masses take the place of the 32-bit sums)
        constexpr int kOwn = kBuckets / kNucleusThreads;
        unsigned long long raw[kOwn], tempered[kOwn];
#pragma unroll
        for (int j = 0; j < kOwn; j++) {
            const uint32_t b = j * kNucleusThreads + tid;
            raw[j] = ((unsigned long long)raw_high[b] << 16) + raw_low[b];
            tempered[j] = ((unsigned long long)tempered_high[b] << 16) + tempered_low[b];
            if (m.count[b] > 65535u) short_memory().state.share.unseen = INFINITY;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kOwn; j++) {
            const uint32_t b = j * kNucleusThreads + tid;
            m.mass[b] = raw[j];
            m.other_mass[b] = tempered[j];
        }
    }
    // The weights exp((v - top) * inv_t) inside `step.inside`, per value bucket.
    __device__ __noinline__ void weigh(const LongStep &asked) const {
        const LongStep step = asked;
        LongMemory &m = memory();
        const NucleusShared &sh = short_memory().scan;
        clear_histogram(short_memory().scan, kBuckets);
        walk([&](float v, uint32_t i) {
            if (is_nonfinite(v) || !step.inside.holds(float_key(v), i)) return;
            const unsigned long long w = exp_fixed(((double)v - (double)step.top) * step.inv_t, sh.table);
            const uint32_t b = value_bucket(v, step.top);
            add_mass(&m.mass[b], w);
            atomicAdd(&m.count[b], 1u);
        });
    }
    // ... all of them together
    __device__ __noinline__ void weigh_all(const LongStep &asked) const {
        const LongStep step = asked;
        NucleusShared &sh = short_memory().scan;
        unsigned long long sum = 0;
        walk([&](float v, uint32_t i) {
            if (!is_nonfinite(v) && step.inside.holds(float_key(v), i))
                sum += exp_fixed(((double)v - (double)step.top) * step.inv_t, sh.table);
        });
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(kFullMask, sum, d);
        if (lane_id() == 0) sh.scan_mass[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < kNucleusWarps; w++) sum += sh.scan_mass[w];
            sh.total_mass = sum;
        }
    }
    // One level of a descent over the keys: those that begin with `step.prefix`, by their next bits.
    __device__ __noinline__ void weigh_keys(const LongStep &asked) const {
        const LongStep step = asked;
        LongMemory &m = memory();
        const NucleusShared &sh = short_memory().scan;
        const int shift = descent_shift(step.level);
        const uint32_t buckets = descent_buckets(step.level);
        clear_histogram(short_memory().scan, buckets);
        walk([&](float v, uint32_t i) {
            if (is_nonfinite(v)) return;
            const uint32_t key = float_key(v);
            if (step.level > 0 && (key >> (shift + descent_bits(step.level))) != step.prefix) return;
            if (!step.inside.holds(key, i)) return;
            const unsigned long long w = exp_fixed((double)v * step.inv_t - (double)step.top * step.inv_t, sh.table);
            const uint32_t b = (key >> shift) & (buckets - 1);
            add_mass(&m.mass[b], w);
            atomicAdd(&m.count[b], 1u);
        });
    }
    // One level of a descent over the ids of the values with key `step.key`, small ones first: the
    // buckets are numbered backwards.
    __device__ __noinline__ void count_ids(const LongStep &asked) const {
        const LongStep step = asked;
        LongMemory &m = memory();
        const int shift = descent_shift(step.level);
        const uint32_t buckets = descent_buckets(step.level);
        clear_histogram(short_memory().scan, buckets);
        walk([&](float v, uint32_t i) {
            if (is_nonfinite(v) || float_key(v) != step.key || !step.inside.holds(step.key, i)) return;
            if (step.level > 0 && (i >> (shift + descent_bits(step.level))) != step.prefix) return;
            const uint32_t b = buckets - 1 - ((i >> shift) & (buckets - 1));
            atomicAdd(&m.count[b], 1u);
            add_mass(&m.mass[b], 1ull);
        });
    }
    // The members of a value bucket inside `step.inside` onto the first CTA's list.
    __device__ __noinline__ void list_members(const LongStep &asked) const {
        const LongStep step = asked;
        LongMemory &m = memory();
        ShortShared &ss = short_memory().state;
        walk([&](float v, uint32_t i) {
            // (a NaN or an infinity has no bucket: the conversion sends them to the last one or to
            // bucket 0, so they are looked at, and dropped, only there)
            if (value_bucket(v, step.top) != step.bucket) return;
            if (is_nonfinite(v) || !step.inside.holds(float_key(v), i)) return;
            const uint32_t slot = atomicAdd(team.at(&ss.cut_count, 0), 1u);
            if (slot < kListCap) {
                team.at(m.value, 0)[slot] = v;
                team.at(m.id, 0)[slot] = i;
            }
        });
    }
    // The id of the one value with key `step.key`.
    __device__ __noinline__ void find_only(const LongStep &asked) const {
        const LongStep step = asked;
        ShortShared &ss = short_memory().state;
        walk([&](float v, uint32_t i) {
            if (!is_nonfinite(v) && float_key(v) == step.key && step.inside.holds(step.key, i)) *team.at(&ss.only_id, 0) = i;
        });
    }
    __device__ __forceinline__ void take(const LongStep &step) const {
        switch (step.what) {
        case LongStep::kLargest: largest(); break;
        case LongStep::kWeighBoth: weigh_both(step); break;
        case LongStep::kWeigh: weigh(step); break;
        case LongStep::kWeighAll: weigh_all(step); break;
        case LongStep::kWeighKeys: weigh_keys(step); break;
        case LongStep::kCountIds: count_ids(step); break;
        case LongStep::kListMembers: list_members(step); break;
        case LongStep::kFindOnly: find_only(step); break;
        default: break;
        }
    }

    // ---- the other CTAs of the team: whatever the first one asks for ----
    __device__ __forceinline__ void follow() const {
        for (;;) {
            team.sync();
            const LongStep step = *team.at(&short_memory().state.step, 0);
            if (step.what == LongStep::kStop) return;
            take(step);
            team.sync();
        }
    }
    // ---- the first CTA; all its threads call these ----
    __device__ __forceinline__ void stop() const {
        if (threadIdx.x == 0) short_memory().state.step.what = LongStep::kStop;
        team.sync();
    }
    __device__ __noinline__ void all(const LongStep step) const {
        __syncthreads();
        if (threadIdx.x == 0) short_memory().state.step = step;
        team.sync();
        take(step);
        team.sync();
    }
    // the team's histograms added up in the first CTA's
    __device__ __noinline__ void add_up(uint32_t buckets, bool both) const {
        LongMemory &m = memory();
        for (uint32_t b = threadIdx.x; b < buckets; b += kNucleusThreads) {
            unsigned long long mass = m.mass[b], other = both ? m.other_mass[b] : 0ull;
            uint32_t count = m.count[b];
#pragma unroll
            for (uint32_t r = 1; r < kMostTeam; r++) {
                if (r >= team.size) break;
                mass += *team.at(&m.mass[b], r);
                if (both) other += *team.at(&m.other_mass[b], r);
                count += *team.at(&m.count[b], r);
            }
            m.mass[b] = mass;
            if (both) m.other_mass[b] = other;
            m.count[b] = count;
        }
        __syncthreads();
    }
    // Both phases' masses as 2^-40 fixed point, scaled by the weight of the bucket's edge,
    // exp(-b/256) (and its power inv_t): 2^-32 -> 2^-40 is a factor 256.  false: a bucket holds
    // too many members for its sums.
    __device__ __noinline__ bool fill_both(double inv_t, float top) const {
        LongMemory &m = memory();
        LongStep step;
        step.what = LongStep::kWeighBoth;
        step.inv_t = inv_t;
        step.top = top;
        all(step);
        add_up(kBuckets, true);
        for (uint32_t b = threadIdx.x; b < kBuckets; b += kNucleusThreads) {
            const uint32_t members = m.count[b];
            const double edge = -(double)b * (1.0 / 256.0);
            m.mass[b] = members ? __double2ull_rn((double)m.mass[b] * 256.0 * exp(edge)) : 0ull;
            m.other_mass[b] = members ? __double2ull_rn((double)m.other_mass[b] * 256.0 * exp(edge * inv_t)) : 0ull;
        }
        double unseen = 0.0;
        for (uint32_t r = 0; r < team.size; r++) unseen += team.at(&short_memory().state.share, r)->unseen;
        __syncthreads();
        return unseen == 0.0;
    }
    // The members of one value bucket (restricted to `inside`), then order_members.  ok = false: the
    // bucket is empty or holds more than the list takes.
    __device__ __noinline__ Position resolve_bucket(double inv_t, float top, const Nucleus inside, uint32_t bucket,
                                                    uint32_t members, unsigned long long before, uint32_t rank_before,
                                                    unsigned long long target, bool strict, bool clipped,
                                                    double also_inv_t, unsigned long long *also_sum) const {
        LongMemory &m = memory();
        ShortShared &ss = short_memory().state;
        Position found;
        found.ok = false;
        found.total = 0;
        if (members == 0 || members > kListCap) return found;  // (heavy ties)
        if (threadIdx.x == 0) ss.cut_count = 0;
        LongStep step;
        step.what = LongStep::kListMembers;
        step.top = top;
        step.inside = inside;
        step.bucket = bucket;
        all(step);
        members = min(ss.cut_count, kListCap);  // (inside may hold fewer of the bucket than the histogram counted)
        if (members == 0) return found;
        OrderWork work;
        work.weight = m.mass;
        work.sorted_value = reinterpret_cast<float *>(work.weight + kOrderCap);
        work.sorted_id = reinterpret_cast<uint32_t *>(work.sorted_value + kOrderCap);
        work.value = m.value;
        work.id = m.id;
        return order_members(short_memory().scan, work, members, inv_t, top, inside, before, rank_before, target, strict,
                             clipped, also_inv_t, also_sum, 40);
    }
    // One phase: among the elements `inside`, weights exp((v - top) * inv_t), find the first
    // element of the (value descending, id ascending) order at which the running weight reaches
    // target_of(total) (strict: exceeds it); if it never does, the last element inside.
    template <typename TargetOf>
    __device__ __forceinline__ Position locate(double inv_t, float top, const Nucleus inside, TargetOf target_of,
                                               bool strict) const {
        NucleusShared &sh = short_memory().scan;
        LongStep step;
        step.what = LongStep::kWeigh;
        step.inv_t = inv_t;
        step.top = top;
        step.inside = inside;
        all(step);
        add_up(kBuckets, false);
        const unsigned long long target = find_crossing_up(sh, target_of, strict);
        const unsigned long long total = sh.total_mass;
        const bool clipped = settle_crossing(sh);
        const uint32_t bucket = sh.hit_bucket;
        const unsigned long long before = sh.hit_mass_before;
        const uint32_t rank_before = sh.hit_count_before;
        const uint32_t members = sh.count[bucket];
        __syncthreads();
        Position found = resolve_bucket(inv_t, top, inside, bucket, members, before, rank_before, target, strict, clipped,
                                        0.0, nullptr);
        found.total = total;
        return found;
    }
    __device__ __noinline__ unsigned long long total(double inv_t, float top, const Nucleus inside) const {
        LongStep step;
        step.what = LongStep::kWeighAll;
        step.inv_t = inv_t;
        step.top = top;
        step.inside = inside;
        all(step);
        unsigned long long sum = 0;
        for (uint32_t r = 0; r < team.size; r++) sum += *team.at(&short_memory().scan.total_mass, r);
        __syncthreads();
        return sum;
    }
    // One radix descent.  Weights are exp(value * inv_t - top * inv_t); finds the first element of
    // the (key descending, id ascending) order, restricted to `inside`, at which the cumulative
    // weight reaches `target` (strict: exceeds it).  When even the total does not, the last element
    // inside is returned.  Outputs the element's key and id, the cumulative weight up to and
    // including it and its rank.
    __device__ __noinline__ void descend(double inv_t, float top, const Nucleus inside, unsigned long long target,
                                         bool strict, uint32_t *out_key, uint32_t *out_id,
                                         unsigned long long *out_mass, uint32_t *out_rank) const {
        NucleusShared &sh = short_memory().scan;
        ShortShared &ss = short_memory().state;
        const uint32_t tid = threadIdx.x;
        unsigned long long before = 0;
        uint32_t rank_before = 0;
        unsigned long long weight_of_key = 0;
        uint32_t same_key = 0;
        bool clipped = false;  // target beyond the total: steer to the last element inside
        LongStep step;
        step.what = LongStep::kWeighKeys;
        step.inv_t = inv_t;
        step.top = top;
        step.inside = inside;
        step.prefix = 0;  // key bits fixed so far
        for (step.level = 0; step.level < 3; step.level++) {
            const uint32_t buckets = descent_buckets(step.level);
            all(step);
            add_up(buckets, false);
            if (!clipped) {
                find_crossing(sh, buckets, before, target, strict);
                // the total stays below the target (rounding of the draw, or top_p = 1): the
                // answer is the last element inside, i.e. the lowest non-empty bucket from here on
                if (!sh.hit_found) clipped = true;
                __syncthreads();
            }
            if (clipped) {
                // lowest non-empty bucket: scan by thread 0 (rare path)
                if (tid == 0) {
                    unsigned long long m = before;
                    uint32_t c = 0, last = 0;
                    bool any = false;
                    for (uint32_t at = 0; at < buckets; at++) {
                        const uint32_t b = buckets - 1 - at;
                        if (sh.count[b]) {
                            if (any) {
                                m += sh.mass[last];
                                c += sh.count[last];
                            }
                            last = b;
                            any = true;
                        }
                    }
                    sh.hit_bucket = last;
                    sh.hit_mass_before = m;
                    sh.hit_count_before = c;
                    sh.hit_found = any ? 1u : 0u;
                }
                __syncthreads();
            }
            const uint32_t b = sh.hit_bucket;
            before = sh.hit_mass_before;
            rank_before += sh.hit_count_before;
            weight_of_key = sh.mass[b];
            same_key = sh.count[b];
            step.prefix = (step.prefix << descent_bits(step.level)) | b;
        }
        // the prefix is now a full key; same_key elements share it, each weighing the same
        step.key = step.prefix;
        const unsigned long long each = same_key ? weight_of_key / same_key : 0;
        uint32_t need = same_key;  // how many of the equal-valued elements it takes, 1-based
        if (!clipped && each > 0) {
            // smallest j with before + j*each reaching the target
            const unsigned long long gap = target > before ? target - before : 0;
            unsigned long long j = strict ? gap / each + 1 : (gap + each - 1) / each;
            if (j < 1) j = 1;
            if (j < need) need = (uint32_t)j;
        }
        // the need-th smallest id among the elements with this key that are inside
        step.prefix = 0;
        if (same_key > 1) {
            uint32_t id_rank = need;
            step.what = LongStep::kCountIds;
            for (step.level = 0; step.level < 3; step.level++) {
                const uint32_t buckets = descent_buckets(step.level);
                all(step);
                add_up(buckets, false);
                find_crossing(sh, buckets, 0, id_rank, false);
                id_rank -= (uint32_t)sh.hit_mass_before;
                step.prefix = (step.prefix << descent_bits(step.level)) | (buckets - 1 - sh.hit_bucket);
            }
            *out_id = step.prefix;
        } else {
            step.what = LongStep::kFindOnly;
            if (tid == 0) ss.only_id = kPaddingId;
            all(step);
            *out_id = ss.only_id;
        }
        *out_key = step.key;
        *out_mass = before + (unsigned long long)need * each;
        *out_rank = rank_before + need;
        __syncthreads();
    }

    __device__ __noinline__ void sample(const SamplerConfig cfg, float u, const float *row_values, uint32_t vocab,
                                        uint32_t row, bool penalised, const SelectOutput &out) const {
        NucleusShared &sh = short_memory().scan;
        LongMemory &m = memory();
        const uint32_t tid = threadIdx.x;
        if (penalised) {  // (otherwise the raw logits' maximum has been shared)
            LongStep step;
            step.what = LongStep::kLargest;
            all(step);
        }
        float best = -INFINITY;
        for (uint32_t r = 0; r < team.size; r++) best = fmaxf(best, team.at(&short_memory().state.share, r)->best);
        if (best == -INFINITY) {  // src/sampler.c:97 "sampler received no finite candidates"
            if (tid == 0) {
                report_row(out, row, kErrFormat, kPaddingId, 0.0f);
                if (out.dbg_count) out.dbg_count[row] = 0;
            }
            return;
        }
        // ---- top-p on the un-tempered softmax: where does the mass reach top_p? ----
        Nucleus everything;
        everything.everything = true;
        everything.key = 0;
        everything.id = 0;
        const double top_p = (double)cfg.top_p, inv_t = 1.0 / (double)cfg.temperature, draw_at = (double)u;
        auto mass_target = [top_p](unsigned long long total) { return mass_target_of(top_p, total); };
        auto draw_target = [draw_at](unsigned long long total) { return draw_target_of(draw_at, total); };
        Nucleus nucleus;
        nucleus.everything = false;
        unsigned long long raw_sum, mass_at_cut;
        uint32_t size;
        uint32_t picked_id = kPaddingId;
        unsigned long long weight_sum = 0;

        // ---- the usual way: one pass fills both histograms, each phase then looks into one bucket ----
        bool done = false;
        {
            const bool filled = fill_both(inv_t, best);
            const unsigned long long cut_target = find_crossing_up(sh, mass_target, false);
            raw_sum = sh.total_mass;
            const bool cut_clipped = settle_crossing(sh);
            const uint32_t cut_bucket = sh.hit_bucket;
            const unsigned long long cut_before = sh.hit_mass_before;
            const uint32_t cut_rank_before = sh.hit_count_before;
            const uint32_t cut_members = sh.count[cut_bucket];
            __syncthreads();
            unsigned long long tempered_inside = 0;  // tempered weight of the bucket's members inside the nucleus
            Position cut;
            cut.ok = false;
            if (filled)
                cut = resolve_bucket(1.0, best, everything, cut_bucket, cut_members, cut_before, cut_rank_before, cut_target,
                                     false, cut_clipped, inv_t, &tempered_inside);
            if (cut.ok) {
                nucleus.key = cut.key;
                nucleus.id = cut.id;
                mass_at_cut = cut.mass;
                size = cut.rank;
                // the tempered masses of the nucleus: whole buckets above the cut's, that bucket as
                // far as the nucleus reaches into it, nothing below
                for (uint32_t b = tid; b < kBuckets; b += kNucleusThreads) {
                    m.mass[b] = b < cut_bucket ? m.other_mass[b] : b == cut_bucket ? tempered_inside : 0ull;
                    if (b > cut_bucket) m.count[b] = 0;
                }
                __syncthreads();
                const unsigned long long pick_target = find_crossing_up(sh, draw_target, true);
                weight_sum = sh.total_mass;
                const bool pick_clipped = settle_crossing(sh);
                const uint32_t pick_bucket = sh.hit_bucket;
                const unsigned long long pick_before = sh.hit_mass_before;
                const uint32_t pick_members = sh.count[pick_bucket];
                __syncthreads();
                const Position pick = resolve_bucket(inv_t, best, nucleus, pick_bucket, pick_members, pick_before, 0u,
                                                     pick_target, true, pick_clipped, 0.0, nullptr);
                if (pick.ok) {
                    picked_id = pick.id;
                    done = true;
                }
            }
        }
        if (!done) {
            // ---- a bucket too crowded to order in shared memory: phase by phase, with the exact descent ----
            const Position cut = locate(1.0, best, everything, mass_target, false);
            if (cut.ok) {
                nucleus.key = cut.key;
                nucleus.id = cut.id;
                raw_sum = cut.total;
                mass_at_cut = cut.mass;
                size = cut.rank;
            } else {
                raw_sum = total(1.0, best, everything);
                descend(1.0, best, everything, mass_target(raw_sum), false, &nucleus.key, &nucleus.id, &mass_at_cut, &size);
            }
            // ---- temperature weights of the nucleus, then the draw ----
            const Position pick = locate(inv_t, best, nucleus, draw_target, true);
            if (pick.ok) {
                picked_id = pick.id;
                weight_sum = pick.total;
            } else {
                weight_sum = total(inv_t, best, nucleus);
                uint32_t picked_key, picked_rank;
                unsigned long long picked_mass;
                descend(inv_t, best, nucleus, draw_target(weight_sum), true, &picked_key, &picked_id, &picked_mass,
                        &picked_rank);
            }
        }
        if (tid == 0) {
            if (weight_sum == 0 || raw_sum == 0 || picked_id >= vocab) {
                report_row(out, row, kErrFormat, kPaddingId, 0.0f);
            } else {
                // (from L2: another CTA may have written it)
                report_row(out, row, kOk, picked_id, __ldcg(row_values + picked_id));
            }
            if (out.dbg_count) out.dbg_count[row] = size;  // nucleus size; the list itself is not dumped
        }
        __syncthreads();
    }
};

// The largest of a few logits spread evenly over the row, NaN, infinities and seen columns left
// out (so that the row's own maximum is no smaller): where the window goes.  The second largest if
// the largest is a peak well above it, which would leave the bulk of the row to wide buckets.  (With the
// largest, or peaks of 4 units as the limit, the masses of 1 to 3 % of the rows whose maximum is in the
// sample are estimated to be off by more than 1e-11; with this of none of 1,440.)
// All threads call.
struct TopTwo {
    float first, second;
    __device__ __forceinline__ void join(float a, float b) {  // (a >= b)
        second = fmaxf(fminf(first, a), fmaxf(second, b));
        first = fmaxf(first, a);
    }
};
template <typename T>
__device__ __forceinline__ float sample_row(const T *columns, uint32_t vocab, const SeenBits &seen, float sharp) {
    ShortShared &ss = short_memory().state;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const float none = __uint_as_float(0xff800000u);
    TopTwo best = {none, none};
#pragma unroll
    for (int j = 0; j < kSamples; j++) {
        const uint32_t at = (uint32_t)(((uint64_t)(j * kNucleusThreads + tid) * vocab) / (kSamples * kNucleusThreads));
        const float v = Vector<T>::one(columns + at);
        if (!is_nonfinite(v) && !seen.test(at)) best.join(v, none);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        best.join(__shfl_xor_sync(kFullMask, best.first, d), __shfl_xor_sync(kFullMask, best.second, d));
    if (lane == 0) {
        ss.sample_max[warp] = best.first;
        ss.sample_next[warp] = best.second;
    }
    __syncthreads();
    best = {ss.sample_max[lane % kNucleusWarps], ss.sample_next[lane % kNucleusWarps]};
#pragma unroll
    for (int d = kNucleusWarps / 2; d > 0; d >>= 1)
        best.join(__shfl_xor_sync(kFullMask, best.first, d), __shfl_xor_sync(kFullMask, best.second, d));
    return best.second > none && (best.first - best.second) * sharp > kPeak ? best.second : best.first;
}

// One row the long way; all CTAs of its team call.
template <typename T>
__device__ __noinline__ void go_the_long_way(const NucleusParams &p, const Team team, uint32_t row, const SamplerConfig cfg,
                                             uint32_t lo, uint32_t n, bool penalised, float u) {
    ShortMemory &m = short_memory();
    if (threadIdx.x == 0) {
        m.state.seen_count = 0;
        m.scan.mass = reinterpret_cast<LongMemory *>(&m)->mass;
        m.scan.count = reinterpret_cast<LongMemory *>(&m)->count;
    }
    __syncthreads();
    float *values = p.scratch + (size_t)(blockIdx.x / p.team) * p.scratch_stride;
    const float largest = write_scratch<T>(p, row, cfg, lo, n, penalised, values);
    const LongWay way = {team, values + lo, lo, n};
    way.share_largest(largest);
    team.sync();
    if (team.rank == 0) {
        way.sample(cfg, u, values, p.vocab, row, penalised, p.out);
        way.stop();
    } else {
        way.follow();
    }
}

template <typename T>
__global__ void __launch_bounds__(kNucleusThreads, 2) nucleus_select_kernel(const __grid_constant__ NucleusParams p) {
    constexpr bool kBf16 = sizeof(T) == 2;
    ShortMemory &m = short_memory();
    ShortShared &ss = m.state;
    NucleusShared &sh = m.scan;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    Team team;
    team.size = p.team;
    team.rank = blockIdx.x % p.team;
    const uint32_t teams = gridDim.x / p.team, team_index = blockIdx.x / p.team;
    clear_next_error(p.out);
    if (tid < 64) sh.table[tid] = exp2((double)tid / 64.0);
    if (tid == 0) {
        ss.over_count = ss.cut_count = ss.pick_count = 0;
    }
    float2 *seen = p.seen + (size_t)blockIdx.x * p.seen_stride;
    // the CTA's columns: ranges of a multiple of 64, so that every CTA's first column lies as
    // the row's does to a 16-byte boundary
    const uint32_t chunk = ((p.vocab + p.team - 1) / p.team + 63u) / 64u * 64u;
    const uint32_t lo = min(p.vocab, team.rank * chunk);
    const uint32_t n = min(chunk, p.vocab - lo);
    team.sync();  // every CTA's lists are there before anybody adds to them

    RowWalk walk(team_index);
    uint32_t row;
    while (walk.next(p, teams, row)) {
        const SamplerConfig cfg = p.config_count > 1 ? p.configs[row] : p.config0;
        const T *columns = static_cast<const T *>(p.logits) + (size_t)row * p.row_stride;
        bool penalised = false;  // some column may be
        uint32_t bad = 0;        // status a broken history earns the row
        for (uint32_t split = 0; p.history_meta != nullptr && split < p.splits; split++) {
            const uint2 meta = reinterpret_cast<const uint2 *>(p.history_meta)[(size_t)row * p.splits + split];
            penalised = penalised || (meta.x & 1u);
            if (meta.y) bad = meta.y;
        }
        if (bad) {  // src/output.c:610-612
            if (tid == 0 && team.rank == 0) {
                report_row(p.out, row, bad, kPaddingId, 0.0f);
                if (p.out.dbg_count) p.out.dbg_count[row] = 0;
            }
            continue;
        }
        const double inv_t = 1.0 / (double)cfg.temperature, top_p = (double)cfg.top_p;
        float u = p.uniforms[row];
        if (is_nonfinite(u) || u < 0.0f) u = 0.0f;
        if (u >= 1.0f) u = __uint_as_float(0x3f7fffffu);
        const double draw_at = (double)u;

        // (as many structures as splits in a row, one after the other)
        const SeenBits bits = {penalised ? p.history_global + (size_t)row * p.splits * p.history_stride_words : nullptr,
                               p.history_stride_words, p.split_len};
        float sharp = 1.0f;
        while (cfg.temperature * sharp < kWideColdest && sharp <= kMostSharp) sharp *= 2.0f;
        const bool counting = sharp <= kMostSharp;
        uint32_t finite = 1, verdict = kLongWay;
        float reference = 0.0f;
        if (counting) reference = sample_row(columns, p.vocab, bits, sharp);
        // (nothing finite among the samples, or nothing but a mask's value: any window will do, and the
        // pass finds the true maximum)
        if (is_nonfinite(reference) || !Window(reference, sharp).usable) reference = 0.0f;
        // The window is placed by the sample; if that said little, by the true maximum; if the masses
        // it gives are not good enough, by the bulk of the values.
        bool by_sample = true, by_bulk = false;
        while (counting) {
            const Window window(reference, sharp);
            if (!window.usable) break;
            uint4 *words = reinterpret_cast<uint4 *>(m.first);
            for (uint32_t i = tid; i < 2 * kSlots / 4; i += kNucleusThreads) words[i] = make_uint4(0, 0, 0, 0);
            if (tid == 0) {
                ss.lost = ss.below = ss.above = 0;
                ss.counted = ss.seen_count = 0;
                ss.top_slot = kSlots;
            }
            __syncthreads();
            // ---- first pass ----
            const bool raw_form = kBf16 && !penalised;
            Findings found = penalised  ? count_logits<T, Packing<false>, true>(columns, lo, n, window, team, bits)
                             : raw_form ? count_logits<T, Packing<kBf16>, false>(columns, lo, n, window, team, bits)
                                        : count_logits<T, Packing<false>, false>(columns, lo, n, window, team, bits);
            if (penalised) {
                __syncthreads();
                const Findings more = amend_seen<T, Packing<false>>(p, row, cfg, lo, n, seen, window, team);
                found.lost += more.lost;
                found.below += more.below;
                found.above += more.above;
                __syncthreads();
                // the raw maximum may have been a seen column's: the first bucket that holds anything
                // now stands for it
                uint32_t slot = tid;
                while (slot < kSlots && m.second[swizzled(slot)] == 0) slot += kNucleusThreads;
                slot = __reduce_min_sync(kFullMask, min(slot, kSlots));
                if (lane == 0) atomicMin(&ss.top_slot, slot);
                __syncthreads();
                found.best = fmaxf(found.best, more.best);
                if (ss.top_slot < kSlots) found.best = fmaxf(found.best, window.highest(ss.top_slot));
            }
            float my_best = found.best;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) my_best = fmaxf(my_best, __shfl_xor_sync(kFullMask, my_best, d));
            const int lost = __reduce_add_sync(kFullMask, found.lost);
            const int below = __reduce_add_sync(kFullMask, found.below);
            const int above = __reduce_add_sync(kFullMask, found.above);
            if (lane == 0) {
                ss.sample_max[tid >> 5] = my_best;
                if (lost) atomicAdd(&ss.lost, lost);
                if (below) atomicAdd(&ss.below, below);
                if (above) atomicAdd(&ss.above, above);
            }
            __syncthreads();
            if (tid < 32) {
                my_best = ss.sample_max[lane % kNucleusWarps];
#pragma unroll
                for (int d = kNucleusWarps / 2; d > 0; d >>= 1) my_best = fmaxf(my_best, __shfl_xor_sync(kFullMask, my_best, d));
                if (lane == 0) {
                    ss.share.best = my_best;
                    ss.share.unseen = 0.0;
                    ss.share.finite = n - (uint32_t)ss.lost;
                }
            }
            const uint32_t counted = n - (uint32_t)(ss.lost + ss.below + ss.above);
            team.sync();
            float best = -INFINITY;
            finite = 0;
            for (uint32_t r = 0; r < team.size; r++) {
                const Share *share = team.at(&ss.share, r);
                best = fmaxf(best, share->best);
                finite += share->finite;
            }
            const uint32_t over = *team.at(&ss.over_count, 0);
            if (finite == 0) break;
            if (by_sample && !by_bulk && (over > kOverCap || best < reference)) {
                // the sample said little: the window once more, from the true maximum
                team.sync();
                if (tid == 0) ss.over_count = 0;
                reference = best;
                by_sample = false;
                team.sync();
                continue;
            }
            if (over > kOverCap) break;
            if (sharp > 1.0f && ss.below > 0) {
                // (a window of more than 40 units needs no look at what lies under it)
                const float under = largest_under<T>(columns, lo, n, window.bottom, seen, ss.seen_count);
                if (tid == 0) ss.share.unseen = (double)ss.below * exp((double)under - (double)best);
            }
            const double error = by_bulk ? kMostMassError : kMassError;
            verdict = raw_form ? locate_and_pick<T, Packing<kBf16>>(p, team, window, row, lo, n, counted, bits, seen, best,
                                                                    top_p, inv_t, draw_at, error)
                               : locate_and_pick<T, Packing<false>>(p, team, window, row, lo, n, counted, bits, seen, best,
                                                                    top_p, inv_t, draw_at, error);
            if (verdict != kElsewhere || by_bulk) break;
            const float elsewhere = team.at(&ss.plan, 0)->reference;
            if (elsewhere >= reference) break;
            reference = elsewhere;
            by_bulk = true;
            team.sync();
            if (tid == 0) ss.over_count = ss.cut_count = ss.pick_count = 0;
            team.sync();
        }
        if (finite == 0) {
            // src/sampler.c:97 "sampler received no finite candidates"
            if (tid == 0 && team.rank == 0) {
                report_row(p.out, row, kErrFormat, kPaddingId, 0.0f);
                if (p.out.dbg_count) p.out.dbg_count[row] = 0;
            }
        } else if (verdict != kDone) {
            go_the_long_way<T>(p, team, row, cfg, lo, n, penalised, u);
        }
        // the row's lists are empty again before any CTA adds to them
        if (tid == 0) ss.over_count = ss.cut_count = ss.pick_count = 0;
        team.sync();
    }
}

}  // namespace fgk

using namespace fgk;


static constexpr size_t kNucleusDynamic = sizeof(ShortMemory);
static_assert(sizeof(ShortMemory) + 64 <= 113 * 1024, "two CTAs to an SM");

static const void *nucleus_kernel(uint32_t dtype) {
    return dtype == 1u ? reinterpret_cast<const void *>(nucleus_select_kernel<uint16_t>)
                       : reinterpret_cast<const void *>(nucleus_select_kernel<float>);
}

static cudaLaunchConfig_t nucleus_config(uint32_t ctas, uint32_t team, cudaLaunchAttribute *cluster, cudaStream_t stream) {
    cluster->id = cudaLaunchAttributeClusterDimension;
    cluster->val.clusterDim.x = team;
    cluster->val.clusterDim.y = 1;
    cluster->val.clusterDim.z = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(ctas);
    config.blockDim = dim3(kNucleusThreads);
    config.dynamicSmemBytes = kNucleusDynamic;
    config.stream = stream;
    config.attrs = cluster;
    config.numAttrs = 1;
    return config;
}

extern "C" int fgk_nucleus_prepare(uint32_t most_teams[FGK_NUCLEUS_TEAM_SIZES]) {
    cudaError_t e = cudaSuccess;
    for (uint32_t i = 0; i < FGK_NUCLEUS_TEAM_SIZES; i++) most_teams[i] = 0xffffffffu;
    for (uint32_t dtype = 0; dtype < 2u && e == cudaSuccess; dtype++) {
        e = cudaFuncSetAttribute(nucleus_kernel(dtype), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNucleusDynamic);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(nucleus_kernel(dtype), cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared);
        for (uint32_t i = 0; i < FGK_NUCLEUS_TEAM_SIZES && e == cudaSuccess; i++) {
            cudaLaunchAttribute cluster;
            const cudaLaunchConfig_t config = nucleus_config(1u << i, 1u << i, &cluster, nullptr);
            int teams = 0;
            e = cudaOccupancyMaxActiveClusters(&teams, nucleus_kernel(dtype), &config);
            if (e == cudaSuccess && (uint32_t)teams < most_teams[i]) most_teams[i] = (uint32_t)teams;
        }
    }
    return (int)e;
}

extern "C" int fgk_launch_nucleus_select(const fgk_nucleus_launch *l, void *stream) {
    NucleusParams p;
    p.logits = l->logits;
    p.dtype = l->dtype;
    p.rows = l->rows;
    p.vocab = l->vocab;
    p.row_stride = l->row_stride;
    p.configs = reinterpret_cast<const SamplerConfig *>(l->configs_device);
    p.config0.temperature = l->config0.temperature;
    p.config0.top_p = l->config0.top_p;
    p.config0.top_k = l->config0.top_k;
    p.config0.presence_penalty = l->config0.presence_penalty;
    p.config0.frequency_penalty = l->config0.frequency_penalty;
    p.config0.repetition_penalty = l->config0.repetition_penalty;
    p.config0.min_p = l->config0.min_p;
    p.config0.pad_ = 0;
    p.config0.seed = l->config0.seed;
    p.config_count = l->config_count;
    p.uniforms = l->uniforms;
    p.team = l->team;
    p.scratch = l->scratch;
    p.scratch_stride = l->scratch_stride;
    p.seen = static_cast<float2 *>(l->seen);
    p.seen_stride = l->seen_stride;
    p.history_global = l->history_global;
    p.history_stride_words = l->history_stride_words;
    p.history_meta = l->history_meta;
    p.splits = l->splits;
    p.split_len = l->split_len;
    p.bitmap_words = l->bitmap_words;
    p.count_capacity = l->count_capacity;
    p.dense_wide = l->dense_wide;
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
    const cudaLaunchConfig_t config = nucleus_config(l->ctas, l->team, &cluster, static_cast<cudaStream_t>(stream));
    void *arguments[] = {&p};
    const cudaError_t e = cudaLaunchKernelExC(&config, nucleus_kernel(l->dtype), arguments);
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}
