// Device functions shared by the codec kernels: group abs-max, alignment-agnostic payload accesses,
// scale staging and the 16-element encode / decode steps.
//
// Math parity with the reference kernels: quantization/quant_pack_kernel.cu:84-163 (the stored scale is
// rounded to the source dtype before use), quantization/dequant_reduce_kernel.cu:38-69 (scale / L decode).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace lbc {

template <int G>
__device__ __forceinline__ float group_max(float v) {
    constexpr int lanes = G / kElemsPerThread;
#pragma unroll
    for (int off = lanes / 2; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off, lanes));
    return v;
}

// Magnitudes of two 16-bit elements per word (the signs that come out mean nothing; NaN wins).
template <typename T>
__device__ __forceinline__ uint32_t abs_max2(uint32_t a, uint32_t b) {
    uint32_t r;
    if constexpr (std::is_same<T, __half>::value)
        asm("max.NaN.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else
        asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {      // NaN wins
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Calls `step` with the distances of a butterfly over a group's `lanes` threads (no loop, no width: the partner of a thread
// of an aligned group is in it anyway).
template <typename Step>
__device__ __forceinline__ void over_group(int lanes, const Step& step) {
    if (lanes >= 4) step(2);
    if (lanes >= 2) step(1);
}

// The largest magnitude of a group, NaN if one is in it: two 16-bit elements (three fp32 ones) to an instruction.
template <typename T, int G>
__device__ __forceinline__ float group_top(const Raw16<T>& p) {
    constexpr int lanes = G / kElemsPerThread;
    if constexpr (sizeof(T) == 2) {
        const uint32_t(&w)[8] = p.part[0].w;
        const uint32_t best = abs_max2<T>(abs_max2<T>(abs_max2<T>(w[0], w[1]), abs_max2<T>(w[2], w[3])),
                                          abs_max2<T>(abs_max2<T>(w[4], w[5]), abs_max2<T>(w[6], w[7])));
        uint32_t top = max(best >> 16 & 0x7fffu, best & 0x7fffu);
        over_group(lanes, [&](int off) { top = max(top, __shfl_xor_sync(0xffffffffu, top, off)); });
        return Src<T>::up(uint16_t(top));
    } else {
        float v[16];
        up16<T>(p, v);
        float top = fabsf(v[0]);
#pragma unroll
        for (int i = 1; i + 1 < 16; i += 2) top = max_nan(top, fabsf(v[i]), fabsf(v[i + 1]));
        top = max_nan(top, fabsf(v[15]));
        over_group(lanes, [&](int off) { top = max_nan(top, __shfl_xor_sync(0xffffffffu, top, off)); });
        return top;
    }
}
// Is the scale of every group of the warp one that limit_over takes?  Then no group holds an infinity or a NaN, no value is above
// its scale, |value * (L / scale)| rounds to L at most, and the codes need no clamp.
constexpr float kNearScale = 1.0e30f;
__device__ __forceinline__ bool scales_near(float top) { return __all_sync(0xffffffffu, top < kNearScale); }
// LIM / s, correctly rounded for every s from 1e-6 to 1e30 (all were tried): the quotient through the reciprocal with one Newton
// correction by its exact remainder (Markstein, see over_limit), without the branch of the division.
template <int LIM>
__device__ __forceinline__ float limit_over(float s) {
    const float inverse = __frcp_rn(s);
    const float q = __fmul_rn(float(LIM), inverse);
    return __fmaf_rn(__fmaf_rn(-q, s, float(LIM)), inverse, q);
}

// Alignment-agnostic store of `n` bytes (n = 8 or 16) held in `v`.
__device__ __forceinline__ void store_codes(uint8_t* p, uint4 v, int n) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    if (n == 16 && (a & 15) == 0) {
        st16(p, v);
    } else if ((a & 7) == 0 && n == 8) {
        *reinterpret_cast<uint2*>(p) = make_uint2(v.x, v.y);
    } else if ((a & 3) == 0) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        for (int i = 0; i < n / 4; ++i) reinterpret_cast<uint32_t*>(p)[i] = w[i];
    } else {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        for (int i = 0; i < n / 2; ++i)
            reinterpret_cast<uint16_t*>(p)[i] = uint16_t(w[i / 2] >> (16 * (i & 1)));
    }
}

__device__ __forceinline__ uint4 load_codes(const uint8_t* p, int n) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    if (n == 16 && (a & 15) == 0) return ld16(p);
    uint32_t w[4] = {0, 0, 0, 0};
    if ((a & 3) == 0) {
        for (int i = 0; i < n / 4; ++i) w[i] = reinterpret_cast<const uint32_t*>(p)[i];
    } else {
        for (int i = 0; i < n / 2; ++i)
            w[i / 2] |= uint32_t(reinterpret_cast<const uint16_t*>(p)[i]) << (16 * (i & 1));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// A warp's records of the compact layout: 512 elements are a multiple of 16 bytes whatever the group size, k and code,
// so a warp's span starts on a 16-byte boundary when the payload does, although its records do not.  The span is built
// (or read) in shared memory and moves as vectors; 2- and 4-byte accesses to the records took one instruction per word.
constexpr int kWarpSpan = 1024;      // at most: 512 code bytes and 32 groups of 16 metadata bytes
constexpr int span_bytes(int group, int record) { return 32 * kElemsPerThread / group * record; }

__device__ __forceinline__ void span_to_global(uint8_t* dst, const uint8_t* span, int bytes, int wlane) {
    for (int o = wlane * 16; o + 16 <= bytes; o += 32 * 16) st16(dst + o, *reinterpret_cast<const uint4*>(span + o));
    for (int o = (bytes & ~15) + wlane * 2; o < bytes; o += 64)
        *reinterpret_cast<uint16_t*>(dst + o) = *reinterpret_cast<const uint16_t*>(span + o);
}
// Code words to and from records that start on any even address (shared memory).
template <int CB>
__device__ __forceinline__ void span_put_codes(uint8_t* p, const uint32_t (&w)[4]) {
    constexpr int words = CB / 4;
    if ((reinterpret_cast<uintptr_t>(p) & 3) == 0) {
#pragma unroll
        for (int i = 0; i < words; ++i) reinterpret_cast<uint32_t*>(p)[i] = w[i];
    } else {
        *reinterpret_cast<uint16_t*>(p) = uint16_t(w[0]);
#pragma unroll
        for (int i = 0; i + 1 < words; ++i)
            *reinterpret_cast<uint32_t*>(p + 2 + 4 * i) = __funnelshift_r(w[i], w[i + 1], 16);
        *reinterpret_cast<uint16_t*>(p + 4 * words - 2) = uint16_t(w[words - 1] >> 16);
    }
}
template <int CB>
__device__ __forceinline__ void span_get_codes(const uint8_t* p, uint32_t (&w)[4]) {
    constexpr int words = CB / 4;
    w[2] = w[3] = 0u;
    if ((reinterpret_cast<uintptr_t>(p) & 3) == 0) {
#pragma unroll
        for (int i = 0; i < words; ++i) w[i] = reinterpret_cast<const uint32_t*>(p)[i];
    } else {
        uint32_t mid[words + 1];
        mid[0] = uint32_t(*reinterpret_cast<const uint16_t*>(p)) << 16;
#pragma unroll
        for (int i = 0; i + 1 < words; ++i) mid[i + 1] = *reinterpret_cast<const uint32_t*>(p + 2 + 4 * i);
        mid[words] = *reinterpret_cast<const uint16_t*>(p + 4 * words - 2);
#pragma unroll
        for (int i = 0; i < words; ++i) w[i] = __funnelshift_r(mid[i], mid[i + 1], 16);
    }
}

template <typename T>
__device__ __forceinline__ void store_scale(uint8_t* p, float stored) {
    if constexpr (sizeof(T) == 2)
        *reinterpret_cast<uint16_t*>(p) = Src<T>::down(stored);
    else
        *reinterpret_cast<float*>(p) = stored;
}

template <typename T>
__device__ __forceinline__ float load_scale(const uint8_t* p) {
    if constexpr (sizeof(T) == 2)
        return Src<T>::up(*reinterpret_cast<const uint16_t*>(p));
    else
        return *reinterpret_cast<const float*>(p);
}

// Scales of planar payloads are written as 16-byte vectors, eight (fp32: four) groups at a
// time: one thread per group storing 2 or 4 bytes turns into one partial-sector write per
// group, which over NVLink costs a whole packet each and was measured to halve the push rate.
// The warp parks its scales in shared memory and a few lanes write them out.  Conditions
// (checked once per kernel): planar layout, layout and group offsets multiples of 8 groups,
// 16-byte aligned destinations; an 8-group unit then never straddles two shards.
struct ScaleStage {
    unsigned char bytes[kThreads / 32][32 * 4];
};

template <typename T>
__device__ __forceinline__ void park_scale(ScaleStage& stage, int group_in_warp, float stored) {
    unsigned char* slot = stage.bytes[threadIdx.x >> 5] + group_in_warp * sizeof(T);
    if constexpr (sizeof(T) == 2)
        *reinterpret_cast<uint16_t*>(slot) = Src<T>::down(stored);
    else
        *reinterpret_cast<float*>(slot) = stored;
}

__device__ __forceinline__ bool dsts_aligned16(uint8_t* const* dst, int n) {
    uintptr_t bits = 0;
    for (int d = 0; d < n; ++d) bits |= reinterpret_cast<uintptr_t>(dst[d]);
    return (bits & 15) == 0;
}

// Quantizes 16 rounded values with the group's stored scale; returns packed codes.
template <typename T, int BIT>
__device__ __forceinline__ uint4 encode16(const float (&vals)[16], float stored_scale, float (*decoded)[16]) {
    constexpr int lim = BIT == 8 ? 127 : 7;
    const float safe = fmaxf(stored_scale, 1.0e-6f);
    const float mul = float(lim) / safe;
    uint32_t b[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) b[i] = quant_bits<lim>(vals[i], mul);
    if (decoded != nullptr) {
        // this rank's own quantization error, one rounding: fma(-code, step, value)
        const float step = stored_scale / float(lim);
#pragma unroll
        for (int i = 0; i < 16; ++i) (*decoded)[i] = __fmaf_rn(-float(code_of_bits(b[i])), step, vals[i]);
    }
    if constexpr (BIT == 8) {
        return pack16_low_bytes<sizeof(T)>(b);
    } else {
        const uint2 h = pack16_low_nibbles<sizeof(T)>(b);
        return make_uint4(h.x, h.y, 0, 0);
    }
}

// The same for a warp of scales_near, half the instructions: no clamp, no branch in the quotient, products and sums two to an
// instruction (the product as a multiply-add with zero: a packed product before a packed sum is contracted).
template <typename T, int BIT>
__device__ __forceinline__ uint4 encode16_near(const float (&vals)[16], float stored_scale, float (*decoded)[16]) {
    constexpr int lim = BIT == 8 ? 127 : 7;
    float t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = vals[i];
    fma16(t, limit_over<lim>(fmaxf(stored_scale, 1.0e-6f)), 0.0f);
    add16(t, kRoundMagic);
    if (decoded != nullptr) {
        const float step = over_limit<lim>(stored_scale);
#pragma unroll
        for (int i = 0; i < 16; ++i) (*decoded)[i] = __fmaf_rn(-(t[i] - kRoundMagic), step, vals[i]);
    }
    uint32_t b[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) b[i] = __float_as_uint(t[i]);
    if constexpr (BIT == 8) {
        return pack16_low_bytes<sizeof(T)>(b);
    } else {
        const uint2 h = pack16_low_nibbles<sizeof(T)>(b);
        return make_uint4(h.x, h.y, 0, 0);
    }
}

// Unpacks 16 codes to their integer values (as floats); the caller multiplies by the step.
template <typename T, int BIT>
__device__ __forceinline__ void codes16(uint4 codes, float (&out)[16]) {
    if constexpr (BIT == 8) {
        unpack16_i8_fast<sizeof(T)>(codes, out);
    } else {
        unpack16_i4_fast<sizeof(T)>(make_uint2(codes.x, codes.y), out);
    }
}

// Picks the instantiation of a launcher for a call's dtype, group size and code width.
template <template <typename, int, int> class Launcher, typename P>
static cudaError_t dispatch_profile(const P* p, cudaStream_t stream) {
#define LBC_CASE(TT, GG, BB)                                                        \
    if (p->group_size == GG && p->bit == BB) return Launcher<TT, GG, BB>::run(p, stream);
#define LBC_TYPE(TT)                                                                \
    LBC_CASE(TT, 64, 8) LBC_CASE(TT, 32, 8) LBC_CASE(TT, 16, 8)                     \
    LBC_CASE(TT, 64, 4) LBC_CASE(TT, 32, 4) LBC_CASE(TT, 16, 4)
    switch (p->dtype) {
        case LBC_BF16: LBC_TYPE(__nv_bfloat16) break;
        case LBC_FP16: LBC_TYPE(__half) break;
        case LBC_FP32: LBC_TYPE(float) break;
        default: break;
    }
#undef LBC_TYPE
#undef LBC_CASE
    return cudaErrorInvalidValue;
}

}  // namespace lbc
