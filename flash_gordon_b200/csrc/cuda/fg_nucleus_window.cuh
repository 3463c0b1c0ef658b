// The value buckets of a row without a top-k cut: how many of each width, and which values each
// takes.  (Included after fg_device_common.cuh, whose float_key and key_to_float it uses.)
#pragma once

#include <cstdint>

namespace fgk {

constexpr uint32_t kFineSlots = 4096, kMiddleSlots = 2048, kCoarseSlots = 2048;
constexpr uint32_t kSlots = kFineSlots + kMiddleSlots + kCoarseSlots;
constexpr uint32_t kGroups = kSlots / 32;      // the slots a warp looks at side by side
constexpr uint32_t kPlaces = kGroups + 1;      // place 0: the values above the window
constexpr float kFineScale = 1024.0f, kMiddleScale = 256.0f, kCoarseScale = 64.0f;
constexpr float kMagic = 12582912.0f;          // 1.5 * 2^23: adding it rounds to a whole number
constexpr uint32_t kMagicBits = 0x4b400000u;
constexpr float kWindowMargin = 0.5f;          // how far the window reaches above the sample's maximum
constexpr float kWindowLimit = 3900.0f;        // |v| * 1024 must stay below 2^22

// The window of a row: which values have a bucket, and which.
struct Window {
    float sharp;                          // 1, or a larger power of two for buckets that much narrower
    float top, first_edge, second_edge;   // narrow buckets: [first_edge, top], middle: [second_edge, first_edge),
    float bottom;                         // wide: [bottom, second_edge)
    int fine_top, middle_top, coarse_top; // the middle of the topmost bucket of each kind, in widths
    bool usable;

    __device__ __forceinline__ Window(float reference, float sharp_) : sharp(sharp_) {
        usable = fabsf(reference) * sharp < kWindowLimit;
        const float at = usable ? reference * sharp : 0.0f, unit = 1.0f / sharp;
        // a kind's lowest bucket begins where the next kind's highest ends
        constexpr int kRatio = (int)(kMiddleScale / kCoarseScale), kMiddleSpan = kRatio / 2 + (int)kMiddleSlots - 1;
        constexpr int kSpan = 4 * kMiddleSpan + 2 + (int)kFineSlots - 1;
        static_assert(kFineScale == 4.0f * kMiddleScale && kRatio % 2 == 0, "buckets of one kind end in the middle of the next narrower one");
        coarse_top = __float2int_rn(((at + kWindowMargin) * kFineScale - (float)kSpan) / (float)(4 * kRatio));
        middle_top = kRatio * coarse_top + kMiddleSpan;
        fine_top = 4 * kRatio * coarse_top + kSpan;
        top = (float)fine_top * (1.0f / kFineScale) * unit;
        first_edge = ((float)middle_top + 0.5f) * (1.0f / kMiddleScale) * unit;
        second_edge = ((float)coarse_top + 0.5f) * (1.0f / kCoarseScale) * unit;
        bottom = (float)(coarse_top - (int)(kCoarseSlots - 1)) * (1.0f / kCoarseScale) * unit;
    }
    // the bucket of a value in [bottom, top], and its distance from the middle in widths
    __device__ __forceinline__ uint32_t slot(float v, float &f) const {
        float scale = kCoarseScale * sharp;
        uint32_t base = kMagicBits + kFineSlots + kMiddleSlots + (uint32_t)coarse_top;
        if (v >= second_edge) {
            scale = kMiddleScale * sharp;
            base = kMagicBits + kFineSlots + (uint32_t)middle_top;
        }
        if (v >= first_edge) {
            scale = kFineScale * sharp;
            base = kMagicBits + (uint32_t)fine_top;
        }
        const float shifted = __fmaf_rn(v, scale, kMagic);
        f = __fmaf_rn(v, scale, -__fsub_rn(shifted, kMagic));
        return base - __float_as_uint(shifted);
    }
    // a slot's middle in widths, and the width
    __device__ __forceinline__ int middle_of(uint32_t slot, float &width) const {
        if (slot < kFineSlots) {
            width = 1.0f / (kFineScale * sharp);
            return fine_top - (int)slot;
        }
        if (slot < kFineSlots + kMiddleSlots) {
            width = 1.0f / (kMiddleScale * sharp);
            return middle_top - (int)(slot - kFineSlots);
        }
        width = 1.0f / (kCoarseScale * sharp);
        return coarse_top - (int)(slot - kFineSlots - kMiddleSlots);
    }
    __device__ __forceinline__ double middle(uint32_t slot) const {
        float width;
        const int n = middle_of(slot, width);
        return (double)n * (double)width;
    }
    // the largest and the smallest value in the slot (half-way between two middles the even one takes it)
    __device__ __forceinline__ float highest(uint32_t at) const {
        float width, f;
        const int n = middle_of(at, width);
        const float edge = fminf(((float)n + 0.5f) * width, top);
        return slot(edge, f) == at ? edge : key_to_float(float_key(edge) - 1u);
    }
    __device__ __forceinline__ float lowest(uint32_t at) const {
        float width, f;
        const int n = middle_of(at, width);
        // (a kind's last bucket ends at its middle: what lies below has a bucket of the next kind)
        const float end = at == kFineSlots - 1 ? first_edge : at == kFineSlots + kMiddleSlots - 1 ? second_edge : bottom;
        const float edge = fmaxf(((float)n - 0.5f) * width, end);
        return slot(edge, f) == at ? edge : key_to_float(float_key(edge) + 1u);
    }
};

}  // namespace fgk
