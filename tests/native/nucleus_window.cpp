// fg_nucleus_window.cuh on the host: for windows all over the range of logits, every bucket's
// lowest and highest values lie in it, the floats next to them outside do not, and a value's
// distance from its bucket's middle is exact.  Prints the number of buckets checked.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

#define __device__
#define __forceinline__ inline
static inline uint32_t __float_as_uint(float v) { uint32_t u; std::memcpy(&u, &v, 4); return u; }
static inline float __uint_as_float(uint32_t u) { float v; std::memcpy(&v, &u, 4); return v; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline int __float2int_rn(float v) { return (int)std::nearbyint(v); }
using std::fabs;
namespace fgk {
// order-preserving bits of a float, both zeros alike, and back
inline uint32_t float_key(float v) {
    const uint32_t bits = v == 0.0f ? 0u : __float_as_uint(v);
    return bits >> 31 ? ~bits : bits | 0x80000000u;
}
inline float key_to_float(uint32_t key) { return __uint_as_float(key >> 31 ? key & 0x7fffffffu : ~key); }
}  // namespace fgk
#include "fg_nucleus_window.cuh"
using namespace fgk;

static int fail(const char *what, const Window &w, uint32_t at, float v) {
    std::printf("%s: slot %u value %.9g (window %.9g..%.9g, sharp %g)\n", what, at, v, w.bottom, w.top, w.sharp);
    return 1;
}

static int check(const Window &w) {
    if (!w.usable) return 0;
    for (uint32_t at = 0; at < kSlots; at++) {
        const float low = w.lowest(at), high = w.highest(at);
        float f, width;
        if (!(low <= high)) return fail("empty", w, at, low);
        for (const float v : {low, high}) {
            if (v < w.bottom || v > w.top) return fail("end outside the window", w, at, v);
            if (w.slot(v, f) != at) return fail("end outside its slot", w, at, v);
            const int n = w.middle_of(at, width);
            if ((double)f != (double)v / width - n) return fail("distance not exact", w, at, v);
        }
        const float under = std::nextafterf(low, -INFINITY), over = std::nextafterf(high, INFINITY);
        if (under >= w.bottom && w.slot(under, f) == at) return fail("lowest is not the lowest", w, at, under);
        if (over <= w.top && w.slot(over, f) == at) return fail("highest is not the highest", w, at, over);
    }
    return 0;
}

int main() {
    uint32_t checked = 0, state = 1;
    for (const float sharp : {1.0f, 2.0f, 4.0f, 8.0f, 16.0f, 128.0f})
        for (int i = 0; i < 300; i++) {
            state = state * 1664525u + 1013904223u;
            const float reach = i < 150 ? 40.0f : 3800.0f;
            const Window w(((float)(state >> 8) * 0x1p-23f - 1.0f) * reach, sharp);
            if (check(w)) return 1;
            checked += w.usable ? kSlots : 0u;
        }
    for (const float reference : {0.0f, -0.0f, 3899.9f, -3899.9f, 9.3f})
        if (check(Window(reference, 1.0f))) return 1;
    std::printf("%u\n", checked);
    return 0;
}
