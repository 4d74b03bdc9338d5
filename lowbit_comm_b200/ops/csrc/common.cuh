// Device-side building blocks shared by every sm_100a kernel of the library:
// source-dtype traits, 128/256-bit global accesses, wire-order byte packing,
// system-scope signalling and bounded waits.
//
// Wire format facts used here (reference: csrc/quantization/quant_kernel.cuh:131-146,
// quant_pack_kernel.cu:101-144, dequant_reduce_kernel.cu:27-36): a payload word is
// as wide as the source element and holds its quantized elements most
// significant first, so inside a little-endian word the byte (int8) or nibble
// pair (int4) order is reversed.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "lbc_api.h"

namespace lbc {

constexpr int kMaxRanks = 16;
constexpr int kThreads = 256;
constexpr int kElemsPerThread = 16;  // one 16-byte vector of int8 codes per thread

// ---------------------------------------------------------------------------
// status word written by a kernel whose bounded wait ran out
// ---------------------------------------------------------------------------
struct DeviceStatus {
    unsigned int code;      // 0 = ok, 1 = wait timed out
    unsigned int phase;     // which kernel/phase gave up
    unsigned int peer;      // flag index that never arrived
    unsigned int seen;      // last value read
    unsigned int expected;  // value it waited for
    unsigned int reserved[3];
};

// ---------------------------------------------------------------------------
// kernels in a row
// ---------------------------------------------------------------------------
// A kernel launched with launch_chained may start before the kernel ahead of it in the stream has ended, if that one is such a
// kernel too (or another that issues launch_dependents): then it starts when all blocks of the first are past their own
// chain_wait(), and waits in its chain_wait() until the first is through and its stores are visible.  Its launch and the
// start of its blocks are off the path.  Behind any other kernel, a copy or an event it starts when that has ended.
// Calls one by one, as Python issues them: 13.1 M bf16 elements through the one-rank pass 10.3 -> 7.9 us, encode of 16 MiB
// 8.2 -> 6.6, decode 8.2 -> 5.6.  In a CUDA graph, whose plain launches follow one another more closely, 7.80 -> 7.65,
// 6.90 -> 6.31 and 5.96 -> 5.37, and each behind a kernel of torch 8.67 -> 9.08, 8.14 -> 7.73 and 7.17 -> 6.80.
// First the wait, then the permission for the next kernel: so all that is ahead of a kernel in the stream has ended before the one
// behind it starts.  The other way round, three and more were on the GPU at once.  A kernel of another library that reads, ahead of
// its own wait, what an earlier kernel than the one before it has written would have read too soon; and the blocks
// of grids below one wave, of which some SMs then held more than others, took longer (1 Mi bf16 elements encoded and
// decoded in a graph 4.38 -> 3.41 us, a one-rank pass of 1 Mi fp32 elements with a stochastic code-book and one kept value 17.7 ->
// 11.2).  Grids of several waves pay a little for it: the one-rank pass above 7.81 -> 7.93 us, encode of 16 MiB 6.51 -> 6.56, decode 5.72
// -> 5.62.  Their last blocks could give the permission at once, since others must have ended for them to start; with a
// test for that on the grid's size the same three took 8.03, 6.51 and 5.72.
// Only for kernels that wait for nobody else.  chain_wait comes before the first access to memory (constants and parameters
// aside), in every thread; without the attribute it returns at once.
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename P>
static cudaError_t launch_chained(void (*kernel)(const P), unsigned grid, cudaStream_t stream, const P& p) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(kThreads);
    config.stream = stream;
    config.attrs = &attr;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, p);
}

// ---------------------------------------------------------------------------
// dtype traits
// ---------------------------------------------------------------------------
template <typename T> struct Src;

template <> struct Src<__nv_bfloat16> {
    static constexpr int kBytes = 2;
    __device__ __forceinline__ static float up(uint16_t bits) { return __uint_as_float(uint32_t(bits) << 16); }
    __device__ __forceinline__ static uint16_t down(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }
    // two elements per 32-bit word: one conversion instruction per pair
    __device__ __forceinline__ static void up2(uint32_t w, float& lo, float& hi) {
        lo = __uint_as_float(w << 16);
        hi = __uint_as_float(w & 0xffff0000u);
    }
    __device__ __forceinline__ static uint32_t down2(float lo, float hi) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&v);
    }
};
template <> struct Src<__half> {
    static constexpr int kBytes = 2;
    __device__ __forceinline__ static float up(uint16_t bits) { return __half2float(__ushort_as_half(bits)); }
    __device__ __forceinline__ static uint16_t down(float v) { return __half_as_ushort(__float2half_rn(v)); }
    __device__ __forceinline__ static void up2(uint32_t w, float& lo, float& hi) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
        lo = f.x;
        hi = f.y;
    }
    __device__ __forceinline__ static uint32_t down2(float lo, float hi) {
        const __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&v);
    }
};
template <> struct Src<float> {
    static constexpr int kBytes = 4;
    __device__ __forceinline__ static float up(uint32_t bits) { return __uint_as_float(bits); }
    __device__ __forceinline__ static uint32_t down(float v) { return __float_as_uint(v); }
};

// ---------------------------------------------------------------------------
// global memory accesses
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint4 ld16_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld16(const void* p) {
    uint4 v;
    asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void st16(void* p, uint4 v) {
    asm volatile("st.global.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
struct alignas(32) U8x32 { uint32_t w[8]; };
// 256-bit accesses (sm_100+): one instruction per 32-byte sector.
__device__ __forceinline__ U8x32 ld32_stream(const void* p) {
    U8x32 v;
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]),
                   "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p));
    return v;
}
__device__ __forceinline__ U8x32 ld32(const void* p) {
    U8x32 v;
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]),
                   "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p));
    return v;
}
__device__ __forceinline__ void st32(void* p, const U8x32& v) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]),
                 "r"(v.w[2]), "r"(v.w[3]), "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]), "r"(v.w[7]) : "memory");
}

// ---------------------------------------------------------------------------
// 16 source elements <-> 16 floats
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void load16(const T* base, int64_t first, int64_t numel, bool vec_ok, float (&out)[16],
                                       bool streaming) {
    if (vec_ok && first + 16 <= numel) {
        if constexpr (sizeof(T) == 2) {
            U8x32 v = streaming ? ld32_stream(base + first) : ld32(base + first);
#pragma unroll
            for (int i = 0; i < 8; ++i) Src<T>::up2(v.w[i], out[2 * i], out[2 * i + 1]);
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                U8x32 v = streaming ? ld32_stream(base + first + 8 * h) : ld32(base + first + 8 * h);
#pragma unroll
                for (int i = 0; i < 8; ++i) out[8 * h + i] = __uint_as_float(v.w[i]);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int64_t at = first + i;
            if (at < numel) {
                if constexpr (sizeof(T) == 2)
                    out[i] = Src<T>::up(reinterpret_cast<const uint16_t*>(base)[at]);
                else
                    out[i] = reinterpret_cast<const float*>(base)[at];
            } else {
                out[i] = 0.0f;
            }
        }
    }
}

// Rounds to T and stores; `vals` is replaced by the rounded values (as float).
template <typename T>
__device__ __forceinline__ void round16(float (&vals)[16]) {
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int i = 0; i < 8; ++i) Src<T>::up2(Src<T>::down2(vals[2 * i], vals[2 * i + 1]), vals[2 * i], vals[2 * i + 1]);
    }
}

template <typename T>
__device__ __forceinline__ void store16(T* base, int64_t first, int64_t numel, bool vec_ok, const float (&vals)[16]) {
    if (vec_ok && first + 16 <= numel) {
        if constexpr (sizeof(T) == 2) {
            U8x32 v;
#pragma unroll
            for (int i = 0; i < 8; ++i) v.w[i] = Src<T>::down2(vals[2 * i], vals[2 * i + 1]);
            st32(base + first, v);
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                U8x32 v;
#pragma unroll
                for (int i = 0; i < 8; ++i) v.w[i] = __float_as_uint(vals[8 * h + i]);
                st32(base + first + 8 * h, v);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int64_t at = first + i;
            if (at < numel) {
                if constexpr (sizeof(T) == 2)
                    reinterpret_cast<uint16_t*>(base)[at] = Src<T>::down(vals[i]);
                else
                    reinterpret_cast<float*>(base)[at] = vals[i];
            }
        }
    }
}

// 16 elements as loaded, for kernels that hold several loads in flight.  Plain (not read-only) loads: an output may be
// the buffer that was read, a thread only ever writes the elements that it has read itself.
template <typename T> struct Raw16 {
    U8x32 part[sizeof(T) / 2];
};
__device__ __forceinline__ U8x32 ld32_once(const void* p) {
    U8x32 v;
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]),
                   "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld16_once(const void* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
template <typename T>
__device__ __forceinline__ Raw16<T> raw16(const T* p) {
    Raw16<T> r;
#pragma unroll
    for (int h = 0; h < int(sizeof(T)) / 2; ++h) r.part[h] = ld32_once(p + 16 / (sizeof(T) / 2) * h);
    return r;
}
template <typename T>
__device__ __forceinline__ Raw16<T> down16(const float (&v)[16]) {
    Raw16<T> r;
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int i = 0; i < 8; ++i) r.part[0].w[i] = Src<T>::down2(v[2 * i], v[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) r.part[i / 8].w[i % 8] = __float_as_uint(v[i]);
    }
    return r;
}
template <typename T>
__device__ __forceinline__ void up16(const Raw16<T>& r, float (&v)[16]) {
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int i = 0; i < 8; ++i) Src<T>::up2(r.part[0].w[i], v[2 * i], v[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r.part[i / 8].w[i % 8]);
    }
}

// Tensor ends, element by element.  Out of line on purpose: inlined, their sixteen addresses and predicates cost the
// whole-tile path registers (spills at four blocks per SM).
template <typename T>
__device__ __noinline__ void load16_edge(const T* base, int64_t first, int64_t numel, float* out) {
    float v[16];
    load16<T>(base, first, numel, false, v, false);
#pragma unroll
    for (int i = 0; i < 16; ++i) out[i] = v[i];
}
template <typename T>
__device__ __noinline__ void store16_edge(T* base, int64_t first, int64_t numel, const float* vals) {
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = vals[i];
    store16<T>(base, first, numel, false, v);
}
// 16 elements at `first`, zeros past the end; `vec`: the tensor starts on 32 bytes.
template <typename T>
__device__ __forceinline__ void load16_any(const T* base, int64_t first, int64_t numel, bool vec, float (&out)[16]) {
    if (vec && first + 16 <= numel) {
        up16<T>(raw16(base + first), out);
    } else {
        float v[16];
        load16_edge<T>(base, first, numel, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) out[i] = v[i];
    }
}
template <typename T>
__device__ __forceinline__ void store16_any(T* base, int64_t first, int64_t numel, bool vec, const float (&vals)[16]) {
    if (vec && first + 16 <= numel) {
        store16<T>(base + first, 0, 16, true, vals);
    } else {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = vals[i];
        store16_edge<T>(base, first, numel, v);
    }
}

// The same for tensors of any element alignment, inline: kernels of unaligned calls are instantiated apart from those of
// aligned ones, so what this takes in registers costs the others nothing.  The widest accesses that the address allows
// (it is a tensor's, alike for every chunk); only the chunk with the tensor's end goes element by element.
template <typename T>
__device__ __forceinline__ void load16_ragged(const T* base, int64_t first, int64_t numel, float (&out)[16]) {
    if (first + 16 > numel) {
        float v[16];
        load16_edge<T>(base, first, numel, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) out[i] = v[i];
        return;
    }
    const T* p = base + first;
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    Raw16<T> r;
    constexpr int kWords = 4 * int(sizeof(T));
    uint32_t w[kWords];
    if ((a & 31) == 0) {
        r = raw16(p);
        up16<T>(r, out);
        return;
    }
    if ((a & 15) == 0) {
#pragma unroll
        for (int i = 0; i < kWords / 4; ++i) {
            const uint4 v = ld16(reinterpret_cast<const uint4*>(p) + i);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    } else if (sizeof(T) == 4 || (a & 3) == 0) {
#pragma unroll
        for (int i = 0; i < kWords; ++i) w[i] = reinterpret_cast<const uint32_t*>(p)[i];
    } else {                                            // 16-bit elements from an odd one on: the words between lie on 4 bytes
        const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
        uint32_t before = uint32_t(h[0]) << 16;
#pragma unroll
        for (int i = 0; i < kWords; ++i) {
            const uint32_t next = i + 1 < kWords ? *reinterpret_cast<const uint32_t*>(h + 1 + 2 * i) : uint32_t(h[15]);
            w[i] = __funnelshift_r(before, next, 16);
            before = next;
        }
    }
#pragma unroll
    for (int i = 0; i < kWords; ++i) r.part[i / 8].w[i % 8] = w[i];
    up16<T>(r, out);
}
template <typename T>
__device__ __forceinline__ void store16_ragged(T* base, int64_t first, int64_t numel, const float (&vals)[16]) {
    if (first + 16 > numel) {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = vals[i];
        store16_edge<T>(base, first, numel, v);
        return;
    }
    T* p = base + first;
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    constexpr int kWords = 4 * int(sizeof(T));
    if ((a & 31) == 0) {
        store16<T>(p, 0, 16, true, vals);
        return;
    }
    uint32_t w[kWords];
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int i = 0; i < kWords; ++i) w[i] = Src<T>::down2(vals[2 * i], vals[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < kWords; ++i) w[i] = __float_as_uint(vals[i]);
    }
    if ((a & 15) == 0) {
#pragma unroll
        for (int i = 0; i < kWords / 4; ++i)
            st16(reinterpret_cast<uint4*>(p) + i, make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]));
    } else if (sizeof(T) == 4 || (a & 3) == 0) {
#pragma unroll
        for (int i = 0; i < kWords; ++i) reinterpret_cast<uint32_t*>(p)[i] = w[i];
    } else {
        uint16_t* h = reinterpret_cast<uint16_t*>(p);
        h[0] = uint16_t(w[0]);
#pragma unroll
        for (int i = 0; i + 1 < kWords; ++i)
            *reinterpret_cast<uint32_t*>(h + 1 + 2 * i) = __funnelshift_r(w[i], w[i + 1], 16);
        h[15] = uint16_t(w[kWords - 1] >> 16);
    }
}

// How a chunk lies in its tensors: inside, all of them on 32 bytes; perhaps with their end in it; on any element.
enum : int { kFitWhole = 0, kFitTail = 1, kFitRagged = 2 };
template <typename T, int kFit>
__device__ __forceinline__ void load16_fit(const T* base, int64_t first, int64_t numel, float (&out)[16]) {
    if constexpr (kFit == kFitWhole)
        up16<T>(raw16(base + first), out);
    else if constexpr (kFit == kFitTail)
        load16_any<T>(base, first, numel, true, out);
    else
        load16_ragged<T>(base, first, numel, out);
}
template <typename T, int kFit>
__device__ __forceinline__ void store16_fit(T* base, int64_t first, int64_t numel, const float (&vals)[16]) {
    if constexpr (kFit == kFitWhole)
        store16<T>(base + first, 0, 16, true, vals);
    else if constexpr (kFit == kFitTail)
        store16_any<T>(base, first, numel, true, vals);
    else
        store16_ragged<T>(base, first, numel, vals);
}
// Host: do all of these (null included) start on `bytes`?
inline bool on_boundary(uintptr_t bytes, const void* a, const void* b = nullptr, const void* c = nullptr,
                        const void* d = nullptr) {
    return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
             reinterpret_cast<uintptr_t>(d)) & (bytes - 1)) == 0;
}

// 16 floats, two to an instruction (sm_100+), with the roundings of the scalar forms.  Never a packed product before a packed sum: the
// assembler contracts the two, although both ask for a rounding of their own.
__device__ __forceinline__ void mul16(float (&v)[16], float s) {
#pragma unroll
    for (int i = 0; i < 16; i += 2)
        asm("{.reg .b64 a, b; mov.b64 a, {%0, %1}; mov.b64 b, {%2, %2}; mul.rn.f32x2 a, a, b; mov.b64 {%0, %1}, a;}"
            : "+f"(v[i]), "+f"(v[i + 1]) : "f"(s));
}
__device__ __forceinline__ void add16(float (&v)[16], float s) {
#pragma unroll
    for (int i = 0; i < 16; i += 2)
        asm("{.reg .b64 a, b; mov.b64 a, {%0, %1}; mov.b64 b, {%2, %2}; add.rn.f32x2 a, a, b; mov.b64 {%0, %1}, a;}"
            : "+f"(v[i]), "+f"(v[i + 1]) : "f"(s));
}

// v = v * s + add, each with one rounding.
__device__ __forceinline__ void fma16(float (&v)[16], float s, float add) {
#pragma unroll
    for (int i = 0; i < 16; i += 2)
        asm("{.reg .b64 a, b, c; mov.b64 a, {%0, %1}; mov.b64 b, {%2, %2}; mov.b64 c, {%3, %3}; fma.rn.f32x2 a, a, b, c; mov.b64 {%0, %1}, a;}"
            : "+f"(v[i]), "+f"(v[i + 1]) : "f"(s), "f"(add));
}

// prepared = T(x + residual), which is also returned in T
template <typename T>
__device__ __forceinline__ Raw16<T> compensate16(float (&v)[16], const float (&r)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += r[i];
    const Raw16<T> held = down16<T>(v);
    if constexpr (sizeof(T) == 2) up16<T>(held, v);
    return held;
}

// ---------------------------------------------------------------------------
// wire-order packing of 16 codes
// ---------------------------------------------------------------------------
// Round-to-nearest-even quantization without a float->int conversion: adding
// 1.5 * 2^23 to t = v * mul leaves rint(t) in the low mantissa bits, so the low
// byte (nibble) of the result's bit pattern is the two's-complement code.  The
// product is rounded to fp32 first, exactly as rint(v * mul) would see it.
constexpr float kRoundMagic = 12582912.0f;  // bits 0x4B400000

template <int LIM>
__device__ __forceinline__ uint32_t quant_bits(float v, float mul) {
    float r = __fadd_rn(__fmul_rn(v, mul), kRoundMagic);
    r = fminf(fmaxf(r, kRoundMagic - float(LIM)), kRoundMagic + float(LIM));
    return __float_as_uint(r);
}
// s / LIM, correctly rounded for every finite s (all were tried) but -0, which gives +0 and is no scale: the product with 1 / LIM
// and one Newton correction by its exact remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000", 1990), five instructions and no branch.
template <int LIM>
__device__ __forceinline__ float over_limit(float s) {
    constexpr float inverse = 1.0f / float(LIM);
    const float q = __fmul_rn(s, inverse);
    const float t = __fmaf_rn(__fmaf_rn(-q, float(LIM), s), inverse, q);
    return fabsf(s) < INFINITY ? t : q;
}
__device__ __forceinline__ int code_of_bits(uint32_t bits) { return int(bits) - 0x4B400000; }

// Low bytes of 16 bit patterns -> 16 wire-ordered bytes, three byte permutes per word.
template <int WordBytes>
__device__ __forceinline__ uint4 pack16_low_bytes(const uint32_t (&b)[16]) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t e0 = b[4 * j], e1 = b[4 * j + 1], e2 = b[4 * j + 2], e3 = b[4 * j + 3];
        if constexpr (WordBytes == 2) {   // memory bytes: e1 e0 e3 e2
            w[j] = __byte_perm(__byte_perm(e1, e0, 0x0040), __byte_perm(e3, e2, 0x0040), 0x5410);
        } else {                          // memory bytes: e3 e2 e1 e0
            w[j] = __byte_perm(__byte_perm(e3, e2, 0x0040), __byte_perm(e1, e0, 0x0040), 0x5410);
        }
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// 16 wire-ordered int8 codes -> their values as floats: flip the sign bit of every
// byte, drop the byte into the mantissa of 2^23 and subtract 2^23 + 128 (exact).
template <int WordBytes>
__device__ __forceinline__ void unpack16_i8_fast(uint4 v, float (&out)[16]) {
    const uint32_t w[4] = {v.x ^ 0x80808080u, v.y ^ 0x80808080u, v.z ^ 0x80808080u, v.w ^ 0x80808080u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int pos = WordBytes == 2 ? (e ^ 1) : (3 - e);
            out[4 * j + e] = __uint_as_float(__byte_perm(w[j], 0x4B000000u, 0x7540 | pos)) - 8388736.0f;
        }
    }
}

// Low nibbles of 16 bit patterns -> 8 wire-ordered bytes: even and odd elements are gathered as bytes, then interleaved.
template <int WordBytes>
__device__ __forceinline__ uint2 pack16_low_nibbles(const uint32_t (&b)[16]) {
    uint32_t w[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const uint32_t* e = b + 8 * j;
        uint32_t hi, lo;
        if constexpr (WordBytes == 2) {
            hi = __byte_perm(__byte_perm(e[2], e[0], 0x0040), __byte_perm(e[6], e[4], 0x0040), 0x5410);
            lo = __byte_perm(__byte_perm(e[3], e[1], 0x0040), __byte_perm(e[7], e[5], 0x0040), 0x5410);
        } else {
            hi = __byte_perm(__byte_perm(e[6], e[4], 0x0040), __byte_perm(e[2], e[0], 0x0040), 0x5410);
            lo = __byte_perm(__byte_perm(e[7], e[5], 0x0040), __byte_perm(e[3], e[1], 0x0040), 0x5410);
        }
        w[j] = ((hi << 4) & 0xf0f0f0f0u) | (lo & 0x0f0f0f0fu);
    }
    return make_uint2(w[0], w[1]);
}

// 8 wire-ordered int4 bytes -> their values as floats: (c ^ 8) dropped into the mantissa of 2^23, minus 2^23 + 8 (exact).
template <int WordBytes>
__device__ __forceinline__ void unpack16_i4_fast(uint2 v, float (&out)[16]) {
    const uint32_t w[2] = {v.x ^ 0x88888888u, v.y ^ 0x88888888u};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const uint32_t hi = (w[j] >> 4) & 0x0f0f0f0fu, lo = w[j] & 0x0f0f0f0fu;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int pos = WordBytes == 2 ? ((e >> 1) ^ 1) : (3 - (e >> 1));
            out[8 * j + e] = __uint_as_float(__byte_perm((e & 1) ? lo : hi, 0x4B000000u, 0x7540 | pos)) - 8388616.0f;
        }
    }
}

// ---------------------------------------------------------------------------
// cross-GPU signalling: release stores, acquire loads, bounded waits
// ---------------------------------------------------------------------------
__device__ __forceinline__ void st_release_sys(unsigned int* p, unsigned int v) {
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

using SignalSpec = LbcSignal;  // producer side, see lbc_api.h
using WaitSpec = LbcWait;      // consumer side, see lbc_api.h

// Returns false when the wait ran out; every thread of the block gets the same answer.
__device__ __forceinline__ bool block_wait(const WaitSpec& w) {
    if (w.flags == nullptr || w.count == 0) return true;
    __shared__ int ok;
    if (threadIdx.x == 0) ok = 1;
    __syncthreads();
    if (threadIdx.x < w.count) {
        const unsigned int* f = w.flags + threadIdx.x;
        unsigned int seen = ld_acquire_sys(f);
        if (int(seen - w.epoch) < 0) {
            const unsigned long long t0 = global_ns();
            unsigned int spins = 0;
            for (;;) {
                seen = ld_acquire_sys(f);
                if (int(seen - w.epoch) >= 0) break;
                if ((++spins & 63u) == 0) {
                    volatile DeviceStatus* st = static_cast<volatile DeviceStatus*>(w.status);
                    // an earlier wait of this group already ran out: give up at once, so that the
                    // kernels queued behind a failed collective drain quickly
                    const bool failed_before = st != nullptr && st->code != 0u;
                    if (failed_before) {
                        ok = 0;
                        break;
                    }
                    if (global_ns() - t0 > w.timeout_ns) {
                        ok = 0;
                        // plain stores: the status word may live in mapped host memory, where
                        // device atomics are not guaranteed; any timed-out thread's report will do
                        if (st != nullptr) {
                            st->phase = w.phase;
                            st->peer = threadIdx.x;
                            st->seen = seen;
                            st->expected = w.epoch;
                            __threadfence_system();
                            st->code = 1u;
                            __threadfence_system();
                        }
                        break;
                    }
                }
                __nanosleep(64);
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

// ---------------------------------------------------------------------------
// bulk asynchronous stores (TMA engine): shared memory -> global memory, own or a peer's.
// The copy engine moves the tile, so a back-pressured NVLink write does not stall the SM's
// load/store pipeline the way per-thread peer stores do.  No multicast, no tensor map: plain
// `cp.async.bulk` with 16-byte aligned addresses and sizes.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void fence_smem_to_async_proxy() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bulk_store(void* gmem_dst, const void* smem_src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gmem_dst),
                 "r"(smem_addr(smem_src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// At most one committed group may still be reading shared memory afterwards.
__device__ __forceinline__ void bulk_wait_read_1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
// Every committed group has completed its writes.
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Called by every thread after its last remote store.
// Stores through an NVLink multicast address: the switch writes the same bytes into the mapped
// region of every GPU of the multicast group (this GPU included), so one store leaves the SM
// instead of one per destination.  The data moves through .f32 registers bit for bit.
__device__ __forceinline__ void multimem_st16(void* mc_addr, uint4 v) {
    asm volatile("multimem.st.weak.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(mc_addr), "f"(__uint_as_float(v.x)),
                 "f"(__uint_as_float(v.y)), "f"(__uint_as_float(v.z)), "f"(__uint_as_float(v.w))
                 : "memory");
}
__device__ __forceinline__ void multimem_st8(void* mc_addr, uint2 v) {
    asm volatile("multimem.st.weak.global.v2.f32 [%0], {%1, %2};" ::"l"(mc_addr), "f"(__uint_as_float(v.x)),
                 "f"(__uint_as_float(v.y))
                 : "memory");
}

__device__ __forceinline__ void grid_signal(const SignalSpec& s) {
    if (s.num_remote <= 0) return;
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence_system();
        const unsigned int done = atomicAdd(s.block_counter, 1u);
        if (done == gridDim.x * gridDim.y - 1) {
            *s.block_counter = 0u;
            __threadfence_system();
            for (int r = 0; r < s.num_remote; ++r) st_release_sys(s.remote_flags[r] + s.my_slot, s.epoch);
        }
    }
}

}  // namespace lbc
