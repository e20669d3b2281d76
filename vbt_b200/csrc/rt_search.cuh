// rt_search.cuh -- device-side decode of render-temporal control streams from the payload
// (the reference search, one control at one frame).
//
// A control stream is [desc u32 x C][bins u8 x C*B, pad 4][keyframes, pad 4].  Decoding one
// control at one frame follows src/render_temporal_decode.cpp:79-131 (decodeFromSequence):
// clamp the frame, take the bin hint as the predecessor key, fall back to key 0 when the hint
// overshoots, take the next bin's hint + 1 as the upper bracket (fallback: the last key), binary
// search inside the bracket, then lerp v0 + a*(v1 - v0).  Every float operation uses the _rn
// intrinsics so nvcc cannot contract a multiply and an add into an FMA: the result is bit-equal
// to the reference CPU decoder, which rounds after every operation.
//
// All reads go through the payload as aligned 32-bit words (the leaf block is 4-byte aligned);
// byte fields are extracted with funnel shifts.  Bounds were validated once by the payload walker
// (kernel a), so no read here can leave the leaf: keyframe indices stay in [keyStart,
// keyStart + keyCount) and keyStart + keyCount <= keyframe count was checked for every control.
#pragma once
#include <cuda_fp16.h>

#include "vbt_format.cuh"

namespace vbtb {

__device__ __forceinline__ uint32_t ldw(const uint32_t* __restrict__ words, uint32_t word_index)
{
    return __ldg(words + word_index);
}

// Byte at absolute byte offset `b` of the payload.
__device__ __forceinline__ uint32_t ld_byte(const uint32_t* __restrict__ pw, uint64_t b)
{
    return (ldw(pw, (uint32_t)(b >> 2)) >> ((uint32_t)(b & 3u) * 8u)) & 0xFFu;
}

// Three bytes (b, b+1, b+2) as the low 24 bits: frame byte and fp16 value of an FP16 keyframe.
__device__ __forceinline__ uint32_t ld_key24(const uint32_t* __restrict__ pw, uint64_t b)
{
    const uint32_t w = (uint32_t)(b >> 2);
    const uint32_t sh = (uint32_t)(b & 3u) * 8u;
    const uint32_t lo = ldw(pw, w);
    if (sh <= 8u) return (lo >> sh) & 0xFFFFFFu;
    const uint32_t hi = ldw(pw, w + 1u);
    return __funnelshift_r(lo, hi, sh) & 0xFFFFFFu;
}

struct StreamRef {
    uint64_t base;    // absolute payload byte offset of the stream (4-byte aligned)
    uint32_t controls;
    uint32_t bins;    // 8 (coarse / fine) or 4 (Mode2 shell)
    uint32_t kf;      // keyframe count of the stream
    uint32_t codec;   // 1 = FP32 keyframes, otherwise FP16
};

__device__ __forceinline__ uint64_t stream_key_base(const StreamRef& s)
{
    return s.base + (uint64_t)s.controls * 4u + align4(s.controls * s.bins);
}

// Frame index of key i (absolute index inside the stream's keyframe pool).
__device__ __forceinline__ int key_frame(const uint32_t* __restrict__ pw, uint64_t kb, uint32_t codec, uint32_t i)
{
    if (codec == 1u) return (int)(ldw(pw, (uint32_t)((kb + 8ull * i) >> 2)) & 0xFFFFu);
    return (int)ld_byte(pw, kb + 3ull * i);
}

// Value of key i.
__device__ __forceinline__ float key_value(const uint32_t* __restrict__ pw, uint64_t kb, uint32_t codec, uint32_t i)
{
    if (codec == 1u) return __uint_as_float(ldw(pw, (uint32_t)((kb + 8ull * i + 4u) >> 2)));
    return half_bits_to_float(ld_key24(pw, kb + 3ull * i) >> 8);
}

// Frame and value of key i in one read.
__device__ __forceinline__ void key_read(const uint32_t* __restrict__ pw, uint64_t kb, uint32_t codec, uint32_t i,
                                         int& frame, float& value)
{
    if (codec == 1u) {
        const uint32_t w = (uint32_t)((kb + 8ull * i) >> 2);
        frame = (int)(ldw(pw, w) & 0xFFFFu);
        value = __uint_as_float(ldw(pw, w + 1u));
    } else {
        const uint32_t k = ld_key24(pw, kb + 3ull * i);
        frame = (int)(k & 0xFFu);
        value = half_bits_to_float(k >> 8);
    }
}

// Time bin for a clamped frame: min(bins-1, frame*bins / max(1, total)).
__device__ __forceinline__ uint32_t time_bin(int frame, uint32_t bins, int total)
{
    if (bins == 0u) return 0u;
    const uint32_t n = (uint32_t)(total > 1 ? total : 1);
    // 0 <= frame < total: the product fits 32 bits for any real frame count (bins <= 8)
    const uint32_t q = n < (1u << 28) ? (uint32_t)frame * bins / n : (uint32_t)(((long long)frame * bins) / n);
    return q < bins - 1u ? q : bins - 1u;
}

__device__ __forceinline__ int clamp_frame(int frame_index, int total)
{
    const int tmax = total - 1 > 0 ? total - 1 : 0;
    return frame_index < 0 ? 0 : (frame_index > tmax ? tmax : frame_index);
}

// Decode control c of stream s at clamped frame `frame` (bin = time_bin(frame, s.bins, total)).
__device__ __forceinline__ float decode_control(const uint32_t* __restrict__ pw, const StreamRef& s, uint32_t c,
                                                int frame, uint32_t bin)
{
    const uint32_t desc = ldw(pw, (uint32_t)((s.base + 4ull * c) >> 2));
    const uint32_t kc = (desc >> 16) & 0xFFu;
    // bin row: bins bytes at base + 4C + c*bins (4-byte aligned for bins = 4 or 8)
    const uint64_t row = s.base + 4ull * s.controls + (uint64_t)c * s.bins;
    const uint32_t w0 = ldw(pw, (uint32_t)((row + (bin & ~3u)) >> 2));
    // keyCount 0 decodes to 0; a key range past the pool only occurs for Mode2 shell controls of
    // voxels outside a boundary leaf's extent, which are never sampled (the walker validated all
    // others), so it is not read either.
    if (kc == 0u || (desc & 0xFFFFu) + kc > s.kf) return 0.0f;
    const uint32_t ks = desc & 0xFFFFu;
    const uint32_t last = kc - 1u;
    const uint64_t kb = stream_key_base(s) ;
    const uint32_t hb = (w0 >> ((bin & 3u) * 8u)) & 0xFFu;
    uint32_t lo = hb < last ? hb : last;
    int f0;
    float v0;
    key_read(pw, kb, s.codec, ks + lo, f0, v0);
    if (f0 > frame) {
        lo = 0u;
        key_read(pw, kb, s.codec, ks, f0, v0);
    }
    if (f0 >= frame || lo == last) return v0;
    uint32_t hi = last;
    if (bin + 1u < s.bins) {
        const uint32_t nb = bin + 1u;
        const uint32_t wn = (nb & ~3u) == (bin & ~3u) ? w0 : ldw(pw, (uint32_t)((row + (nb & ~3u)) >> 2));
        const uint32_t h = ((wn >> ((nb & 3u) * 8u)) & 0xFFu) + 1u;
        hi = h < last ? h : last;
    }
    if (hi < lo + 1u) hi = lo + 1u;
    int f1;
    float v1;
    key_read(pw, kb, s.codec, ks + hi, f1, v1);
    if (f1 < frame) {
        hi = last;
        key_read(pw, kb, s.codec, ks + hi, f1, v1);
    }
    if (f1 <= frame) return v1;
    bool moved_lo = false, moved_hi = false;
    while (hi > lo + 1u) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        const int fm = key_frame(pw, kb, s.codec, ks + mid);
        if (fm < frame) {
            lo = mid;
            f0 = fm;
            moved_lo = true;
        } else {
            hi = mid;
            f1 = fm;
            moved_hi = true;
        }
    }
    if (moved_hi) v1 = key_value(pw, kb, s.codec, ks + hi);
    if (f1 == frame) return v1;
    if (moved_lo) v0 = key_value(pw, kb, s.codec, ks + lo);
    const float alpha = __fdiv_rn((float)(frame - f0), (float)(f1 - f0));
    return __fadd_rn(v0, __fmul_rn(alpha, __fsub_rn(v1, v0)));
}

// binary16 -> binary32 with the hardware conversion; NaNs keep their payload bits exactly as
// src/render_temporal_decode.cpp:167-199 maps them.
__device__ __forceinline__ float half_to_float_exact(uint32_t h)
{
    const float f = __half2float(__ushort_as_half((unsigned short)h));
    const bool nan = (h & 0x7C00u) == 0x7C00u && (h & 0x3FFu) != 0u;
    return nan ? __uint_as_float(((h & 0x8000u) << 16) | 0x7F800000u | ((h & 0x3FFu) << 13)) : f;
}

// A control stream by its byte offset inside a leaf (32-bit offsets from the leaf's first word).
struct LeafStream {
    const uint32_t* __restrict__ w;   // the leaf block
    uint32_t base, controls, bins, kf;
};

// Controls of FP16 streams whose key frames strictly increase, at a clamped frame: the value
// decode_control's search gives (for such keys the canonical one: the first key's value before it,
// the last key's after it, the key's on an exact hit, else the lerp of the pair around the frame;
// see the head of rt_staged.cuh).  Four keys (12 bytes from the hinted one on) are taken at a time
// as independent word reads and the pair is selected in registers: a time bin rarely spans more, so
// a control is two dependent steps (descriptor and hint, keys) where the search's halving makes
// four to seven.  The payload's 16-byte tail padding covers the words past the last key.  The steps
// are apart so that a lane can have the reads of several controls in flight.
struct KeyWindow {
    uint32_t kb, kc, lo;      // byte offset of the control's first key, its keys, the window's first
    uint32_t x0, x1, x2, x3;  // words from the window's first byte on
};

__device__ __forceinline__ void key_window(const uint32_t* __restrict__ lw, KeyWindow& k)
{
    const uint32_t* w = lw + ((k.kb + 3u * k.lo) >> 2);
    k.x0 = __ldg(w);
    k.x1 = __ldg(w + 1);
    k.x2 = __ldg(w + 2);
    k.x3 = __ldg(w + 3);
}

// The window a control's descriptor and hint word name; kc 0 where it decodes to 0 (see decode_control).
__device__ __forceinline__ KeyWindow key_start(const LeafStream& s, uint32_t desc, uint32_t hints, uint32_t bin)
{
    const uint32_t kc = (desc >> 16) & 0xFFu, ks = desc & 0xFFFFu, hb = (hints >> ((bin & 3u) * 8u)) & 0xFFu;
    KeyWindow k{};
    k.kc = ks + kc > s.kf ? 0u : kc;
    k.kb = s.base + s.controls * 4u + align4(s.controls * s.bins) + 3u * ks;
    k.lo = hb + 1u < kc ? hb : kc - 1u;
    return k;
}

// a / b for 0 <= a <= b <= 255, correctly rounded: the product with the approximate reciprocal and one
// fused remainder step (P. Markstein, IBM J. Res. Dev. 34(1), 1990).  A quotient of such integers is at
// least 2^-9 of a unit in the last place away from a rounding boundary, far more than the reciprocal's
// error moves the corrected one.  vbt_selftest_key_division checks every pair.
__device__ __forceinline__ float div_u8_rn(float a, float b)
{
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(b));
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
}

// An integer below 2^23 as a float, without the conversion unit.
__device__ __forceinline__ float small_to_float(uint32_t x)
{
    return __fsub_rn(__uint_as_float(x | 0x4B000000u), 8388608.0f);
}

// The value at `frame`, moving the window where the pair lies elsewhere.  PLAIN: no key is a NaN
// (kFlagHalfPlain).  About 60 instructions, of which a move repeats a quarter.
template <bool PLAIN>
__device__ __forceinline__ float key_value_at(const uint32_t* __restrict__ lw, KeyWindow k, int frame)
{
    if (k.kc == 0u) return 0.0f;
    uint32_t a0, a1, a2, left;
    for (;; key_window(lw, k)) {
        const uint32_t sh = ((k.kb + 3u * k.lo) & 3u) * 8u;
        a0 = __funnelshift_r(k.x0, k.x1, sh);
        a1 = __funnelshift_r(k.x1, k.x2, sh);
        a2 = __funnelshift_r(k.x2, k.x3, sh);
        left = k.kc - k.lo;   // keys from lo on
        if ((int)(a0 & 0xFFu) > frame && k.lo != 0u) k.lo = 0u;                        // the hint overshot
        else if (left > 4u && (int)((a2 >> 8) & 0xFFu) <= frame) k.lo += 3u;   // the pair may lie further on
        else break;
    }
    // keys 0..3 of the window: frame in the low byte, value above it; p1..p3: key i is there and not past the frame
    const uint32_t k1 = __byte_perm(a0, a1, 0x0543), k2 = __byte_perm(a1, a2, 0x0432), k3 = a2 >> 8;
    const bool p1 = left > 1u && (int)(a0 >> 24) <= frame, p2 = left > 2u && (int)(k2 & 0xFFu) <= frame,
               p3 = left > 3u && (int)(k3 & 0xFFu) <= frame;
    const uint32_t lower = p3 ? k3 : p2 ? k2 : p1 ? k1 : a0, upper = p2 ? k3 : p1 ? k2 : k1;
    const bool end = left == (p3 ? 4u : p2 ? 3u : p1 ? 2u : 1u);   // no key after the lower one
    const int ahead = frame - (int)(lower & 0xFFu);                // below 0: before the first key
    auto value = [](uint32_t key) {
        const uint32_t h = (key >> 8) & 0xFFFFu;
        return PLAIN ? __half2float(__ushort_as_half((unsigned short)h)) : half_to_float_exact(h);
    };
    const float vp = value(lower);
    if (end || ahead <= 0) return vp;   // past the last key, an exact hit, before the first key
    const float vn = value(upper);
    const float alpha = div_u8_rn(small_to_float((uint32_t)ahead), small_to_float((upper & 0xFFu) - (lower & 0xFFu)));
    return __fadd_rn(vp, __fmul_rn(alpha, __fsub_rn(vn, vp)));
}

__device__ __forceinline__ uint32_t hint_word(const LeafStream& s, uint32_t c, uint32_t bin)
{
    return __ldg(s.w + ((s.base + 4u * s.controls + c * s.bins + bin) >> 2));
}

template <bool PLAIN>
__device__ __forceinline__ float control_sorted(const LeafStream& s, uint32_t c, int frame, uint32_t bin)
{
    const uint32_t desc = __ldg(s.w + (s.base >> 2) + c);
    KeyWindow k = key_start(s, desc, hint_word(s, c, bin), bin);
    if (k.kc == 0u) return 0.0f;
    key_window(s.w, k);
    return key_value_at<PLAIN>(s.w, k, frame);
}

// The reference's search as a call of its own (leaves with unordered keys or FP32 keys).
__device__ __noinline__ static float control_searched(const uint32_t* w, uint32_t base, uint32_t controls, uint32_t bins,
                                                      uint32_t kf, uint32_t codec, uint32_t c, int frame, uint32_t bin)
{
    return decode_control(w, StreamRef{base, controls, bins, kf, codec}, c, frame, bin);
}

// Control c at clamped frame `frame`; sorted: the leaf's kFlagSorted.
__device__ __forceinline__ float control_at(const LeafStream& s, uint32_t codec, uint32_t c, int frame, uint32_t bin,
                                            bool sorted)
{
    if (sorted && codec != 1u) return control_sorted<false>(s, c, frame, bin);
    return control_searched(s.w, s.base, s.controls, s.bins, s.kf, codec, c, frame, bin);
}

// a*(1-t) + b*t with the reference's rounding (two products, one sum; 1-t precomputed exactly).
__device__ __forceinline__ float lerp_ref(float a, float b, float t, float omt)
{
    return __fadd_rn(__fmul_rn(a, omt), __fmul_rn(b, t));
}

}  // namespace vbtb
