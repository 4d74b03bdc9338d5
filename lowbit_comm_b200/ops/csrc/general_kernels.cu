// General codec kernels: every combination the policy object allows that the
// production-profile kernels do not cover — top-k (1 or 2 values kept verbatim
// per group), 4-bit code-books (normal, uniform, e3m0, e2m1), stochastic
// rounding — for fp16/bf16/fp32 sources, group sizes 16/32/64, both payload
// layouts.  One kernel per (dtype, k, kind of code); group size, layout, code-book
// and the rounding of linear codes are runtime parameters.
//
// Parity: quantization/quant_kernel.cuh:25-153 (top-k selection, scale = the
// (k+1)-th largest magnitude, selected elements zeroed), inner.cuh:9-96
// (code-book search, rounding rule, stochastic offsets), dequant_kernel.cuh
// :15-44,130-148 (decode and top-k write-back), and the fp32 twins.
// Tie-breaking between equal magnitudes: lowest index first for 16-bit
// sources, highest index first for fp32 sources.
//
// What bounds these kernels is the instruction issue, not memory: selecting, searching a code-book and packing cost
// more cycles per element than its bytes cost DRAM.  Hence: k and the kind of code are template parameters (nothing is
// selected that the profile does not keep); kept elements are patched into the packed words (8 predicated permutes
// instead of 32 selects on the values); a code of a code-book is one look-up and one addition; payload
// words move as vectors; records of the compact layout, which break the alignment, are built in shared memory.
// Measured on a B200, first form / now: encode + decode of 5 M fp32 elements, e2m1 code-book, 81 -> 11.9 us (the search in a
// table in constant memory took one pass per distinct entry in a warp; now kernels and host calls are level); all-reduce
// of one rank, 32 Mi bf16 elements, one kept value per group, 107 -> 22.9 us, two 24.5, fp16 in 4 bits 22.9; 16 Mi 12.1,
// fp32 with two kept values 21.2.  What gave most: no clamp and no NaN test where the selection has shown that no value
// needs them, no trip through packed bytes and a block per tile (72 -> 36 us), no places of the kept elements where
// magnitudes decide (35.9 -> 30.8), the next tile under way without a residual (26.2 -> 22.9).

#include <cmath>
#include <cstring>
#include <type_traits>

#include "codec_device.cuh"
#include "common.cuh"
#include "lbc_api.h"

namespace lbc {

// The four 15-entry tables (normal, uniform, e3m0, e2m1); the device copy ends every row with an infinity.
#define LBC_BOOK_NORMAL                                                                                              \
    -1.0f, -0.815410147f, -0.655160150f, -0.510228027f, -0.375324982f, -0.246951370f, -0.122538030f, 0.0f,           \
        0.122538030f, 0.246951370f, 0.375324982f, 0.510228027f, 0.655160150f, 0.815410147f, 1.0f
#define LBC_BOOK_UNIFORM                                                                                             \
    -1.0f, -0.85714286f, -0.71428571f, -0.57142857f, -0.42857143f, -0.28571429f, -0.14285714f, 0.0f, 0.14285714f,    \
        0.28571429f, 0.42857143f, 0.57142857f, 0.71428571f, 0.85714286f, 1.0f
#define LBC_BOOK_E3M0                                                                                                \
    -1.0f, -0.5f, -0.25f, -0.125f, -0.0625f, -0.03125f, -0.015625f, 0.0f, 0.015625f, 0.03125f, 0.0625f, 0.125f,      \
        0.25f, 0.5f, 1.0f
#define LBC_BOOK_E2M1                                                                                                \
    -1.0f, -0.6666666666666666f, -0.5f, -0.3333333333333333f, -0.25f, -0.16666666666666666f, -0.125f, 0.0f, 0.125f,  \
        0.16666666666666666f, 0.25f, 0.3333333333333333f, 0.5f, 0.6666666666666666f, 1.0f
#define LBC_CODEBOOKS {{LBC_BOOK_NORMAL}, {LBC_BOOK_UNIFORM}, {LBC_BOOK_E3M0}, {LBC_BOOK_E2M1}}

__constant__ float kCodebooks[4][16] = {{LBC_BOOK_NORMAL, INFINITY},
                                        {LBC_BOOK_UNIFORM, INFINITY},
                                        {LBC_BOOK_E3M0, INFINITY},
                                        {LBC_BOOK_E2M1, INFINITY}};

// Counter-based uniform in (0, 1]: a 64-bit mix of (seed, element index).
__device__ __forceinline__ float uniform01(unsigned long long seed, unsigned long long index) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (index + 1ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (float(unsigned(z >> 40)) + 1.0f) * (1.0f / 16777216.0f);
}

template <typename T>
__device__ __forceinline__ void store_word(uint8_t* p, uint32_t bits) {
    if constexpr (sizeof(T) == 2)
        *reinterpret_cast<uint16_t*>(p) = uint16_t(bits);
    else
        *reinterpret_cast<uint32_t*>(p) = bits;
}

template <typename T>
__device__ __forceinline__ uint32_t load_word(const uint8_t* p) {
    if constexpr (sizeof(T) == 2)
        return *reinterpret_cast<const uint16_t*>(p);
    else
        return *reinterpret_cast<const uint32_t*>(p);
}

template <typename T>
__device__ __forceinline__ uint32_t bits_of(float v) {
    return uint32_t(Src<T>::down(v));
}
template <typename T>
__device__ __forceinline__ float value_of(uint32_t bits) {
    if constexpr (sizeof(T) == 2)
        return Src<T>::up(uint16_t(bits));
    else
        return __uint_as_float(bits);
}

// The bits a conversion to T gives (16-bit types: one pattern for every NaN).
template <typename T>
__device__ __forceinline__ uint32_t canonical(uint32_t bits) {
    return bits_of<T>(value_of<T>(bits));
}

// N bytes at an address that is even, in the widest accesses its alignment allows.
template <int N>
__device__ __forceinline__ void store_bytes(uint8_t* p, const uint32_t (&w)[4]) {
    if ((reinterpret_cast<uintptr_t>(p) & 3) == 0) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) reinterpret_cast<uint32_t*>(p)[i] = w[i];
    } else {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) reinterpret_cast<uint16_t*>(p)[i] = uint16_t(w[i / 2] >> (16 * (i & 1)));
    }
}
template <int N>
__device__ __forceinline__ void load_bytes(const uint8_t* p, uint32_t (&w)[4]) {
    w[0] = w[1] = w[2] = w[3] = 0;
    if ((reinterpret_cast<uintptr_t>(p) & 3) == 0) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) w[i] = reinterpret_cast<const uint32_t*>(p)[i];
    } else {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) w[i / 2] |= uint32_t(reinterpret_cast<const uint16_t*>(p)[i]) << (16 * (i & 1));
    }
}

// How the 16 elements of a thread become code bytes.
// kBookNoise is the code-book with stochastic rounding, which has kernels of its own: two divisions per element, and what they
// hold in registers would spill in the kernels of the deterministic one.
enum : int { kLinear8 = 0, kLinear4 = 1, kBook = 2, kBookNoise = 3 };

template <int KIND> struct Kind {
    static constexpr bool book = KIND == kBook || KIND == kBookNoise;
    static constexpr int bit = KIND == kLinear8 ? 8 : 4;
    static constexpr int lim = KIND == kLinear8 ? 127 : 7;          // linear only
    static constexpr int CB = kElemsPerThread * bit / 8;            // code bytes per thread
    static constexpr uint32_t zero_code = book ? 7u : 0u;           // the code of 0.0
};

// Word count of a group's metadata: the scale, and for top-k an index word and the kept values.
__host__ __device__ constexpr int meta_words(int topk) { return topk == 0 ? 1 : topk + 2; }

// The 16 elements of a thread as they lie in memory (16-bit sources: two per word).
template <typename T> struct Packed16 {
    static constexpr int kWords = 16 * int(sizeof(T)) / 4;
    uint32_t w[kWords];
};

template <typename T>
__device__ __forceinline__ Packed16<T> pack_elems(const float (&v)[16]) {
    Packed16<T> p;
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int i = 0; i < 8; ++i) p.w[i] = Src<T>::down2(v[2 * i], v[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) p.w[i] = __float_as_uint(v[i]);
    }
    return p;
}
template <typename T>
__device__ __forceinline__ void unpack_elems(const Packed16<T>& p, float (&v)[16]) {
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int i = 0; i < 8; ++i) Src<T>::up2(p.w[i], v[2 * i], v[2 * i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(p.w[i]);
    }
}

// Tensor ends and unaligned tensors; out of line so that the common path keeps its registers (see load16_edge).
template <typename T>
__device__ __noinline__ void load_elems_edge(const T* base, int64_t first, int64_t n, uint32_t* w) {
    if constexpr (sizeof(T) == 2) {
        const uint16_t* b = reinterpret_cast<const uint16_t*>(base);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int64_t at = first + 2 * i;
            w[i] = (at < n ? uint32_t(b[at]) : 0u) | (at + 1 < n ? uint32_t(b[at + 1]) << 16 : 0u);
        }
    } else {
        const uint32_t* b = reinterpret_cast<const uint32_t*>(base);
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = first + i < n ? b[first + i] : 0u;
    }
}
template <typename T>
__device__ __noinline__ void store_elems_edge(T* base, int64_t first, int64_t n, const uint32_t* w) {
    if constexpr (sizeof(T) == 2) {
        uint16_t* b = reinterpret_cast<uint16_t*>(base);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (first + i < n) b[first + i] = uint16_t(w[i / 2] >> (16 * (i & 1)));
    } else {
        uint32_t* b = reinterpret_cast<uint32_t*>(base);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (first + i < n) b[first + i] = w[i];
    }
}

// 16 elements at `first`, zeros past the end; `vec`: the tensor starts on 32 bytes.
template <typename T>
__device__ __forceinline__ Packed16<T> load_elems(const T* base, int64_t first, int64_t n, bool vec) {
    constexpr int kWords = Packed16<T>::kWords;
    Packed16<T> p;
    if (vec && first + 16 <= n) {
        const Raw16<T> r = raw16(base + first);
#pragma unroll
        for (int i = 0; i < kWords; ++i) p.w[i] = r.part[i / 8].w[i % 8];
    } else {
        uint32_t w[kWords];
        load_elems_edge<T>(base, first, n, w);
#pragma unroll
        for (int i = 0; i < kWords; ++i) p.w[i] = w[i];
    }
    return p;
}

template <typename T>
__device__ __forceinline__ void store_elems(T* base, int64_t first, int64_t n, bool vec, const Packed16<T>& p) {
    constexpr int kWords = Packed16<T>::kWords;
    if (vec && first + 16 <= n) {
#pragma unroll
        for (int h = 0; h < kWords / 8; ++h) {
            U8x32 v;
#pragma unroll
            for (int i = 0; i < 8; ++i) v.w[i] = p.w[8 * h + i];
            st32(reinterpret_cast<uint8_t*>(base + first) + 32 * h, v);
        }
    } else {
        uint32_t w[kWords];
#pragma unroll
        for (int i = 0; i < kWords; ++i) w[i] = p.w[i];
        store_elems_edge<T>(base, first, n, w);
    }
}

// Puts the element with bit pattern `bits` at position `at` (nothing when it is not one of this thread's 16).
template <typename T>
__device__ __forceinline__ void patch_elem(Packed16<T>& p, int at, uint32_t bits) {
    if constexpr (sizeof(T) == 2) {
        const uint32_t how = (at & 1) ? 0x5410u : 0x3254u;
#pragma unroll
        for (int j = 0; j < 8; ++j) p.w[j] = __byte_perm(p.w[j], bits, j == (at >> 1) ? how : 0x3210u);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) p.w[j] = __byte_perm(p.w[j], bits, j == at ? 0x7654u : 0x3210u);
    }
}

// Puts the element at position `at` of `from` in the same place.
template <typename T>
__device__ __forceinline__ void copy_elem(Packed16<T>& p, const Packed16<T>& from, int at) {
    if constexpr (sizeof(T) == 2) {
        const uint32_t how = (at & 1) ? 0x7610u : 0x3254u;
#pragma unroll
        for (int j = 0; j < 8; ++j) p.w[j] = __byte_perm(p.w[j], from.w[j], j == (at >> 1) ? how : 0x3210u);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) p.w[j] = __byte_perm(p.w[j], from.w[j], j == at ? 0x7654u : 0x3210u);
    }
}

// Gives the element at position `at` the code of 0.0 (the value itself travels in the metadata).
template <typename T, int KIND>
__device__ __forceinline__ void patch_code(uint32_t (&w)[4], int at) {
    constexpr int per_word = 32 / Kind<KIND>::bit;
    const int e = at & (per_word - 1);
    const int byte = KIND == kLinear8 ? e : e >> 1;
    const int pos = sizeof(T) == 2 ? byte ^ 1 : 3 - byte;                 // wire order inside the word
    const uint32_t field = KIND == kLinear8 ? 0xffu << (8 * pos) : 0xfu << (8 * pos + ((e & 1) ? 0 : 4));
    const int word = at >= 0 ? at / per_word : -1;
#pragma unroll
    for (int j = 0; j < 16 / per_word; ++j) {
        const uint32_t f = j == word ? field : 0u;
        w[j] = (w[j] & ~f) | (f & (Kind<KIND>::zero_code * 0x11111111u));
    }
}

// What a group's metadata says.
struct GroupMeta {
    float stored;             // the scale, exact in T
    int idx[2];               // positions of the kept elements inside the group
    uint32_t kept[2];         // their bits
    bool tame;                // no infinity and no NaN in the group (fp32: false where it is not asked for)
};

// May the warp's linear codes go without a clamp?  Code-books have a test of their own (book_near) and are not asked: a vote that
// nobody reads stays in the code, and this one waits for the group's scale (fp32 e2m1, two passes, 4 Mi elements: 11.5 -> 10.8 us).
template <int KIND>
__device__ __forceinline__ bool all_near(const GroupMeta& m) {
    return !Kind<KIND>::book && __all_sync(0xffffffffu, m.tame && m.stored < kNearScale);
}

// Magnitude bits of infinity.
template <typename T>
__device__ __forceinline__ constexpr uint32_t inf_bits() {
    return std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u;
}

// The k largest magnitudes of a group and the next one, the scale.  `v` are the thread's 16 values, `p` the same in T;
// the `lanes` threads of a group call this together and all get the answer.  fp32: v of a kept element turns into NaN.
template <typename T, int TOPK, int KIND>
__device__ __forceinline__ GroupMeta select_group(float (&v)[16], const Packed16<T>& p, int lane, int lanes) {
    GroupMeta m;
    m.idx[0] = m.idx[1] = 0;
    m.kept[0] = m.kept[1] = 0u;
    m.tame = false;
    if constexpr (sizeof(T) == 2 && TOPK == 0) {
        uint32_t best = 0u;                                              // magnitudes as integers, two at a time
#pragma unroll
        for (int i = 0; i < 8; ++i) best = __vmaxu2(best, p.w[i] & 0x7fff7fffu);
        uint32_t top = max(best >> 16, best & 0xffffu);
        over_group(lanes, [&](int off) { top = max(top, __shfl_xor_sync(0xffffffffu, top, off)); });
        m.stored = Src<T>::up(uint16_t(top));
        m.tame = top < inf_bits<T>();
    } else if constexpr (sizeof(T) == 2) {
        // key = magnitude bits << 17 | (63 - index) << 1 | sign: integer order is the order of the format (larger
        // magnitude first, lower index on ties), and a key holds everything that is stored of a kept element
        uint32_t k0 = 0u, k1 = 0u, k2 = 0u;                              // k0 >= k1 >= k2
        auto put = [&](uint32_t c) {
            const uint32_t a = min(k0, c);
            k0 = max(k0, c);
            if constexpr (TOPK == 1) {
                k1 = max(k1, a);
            } else {
                const uint32_t b = min(k1, a);
                k1 = max(k1, a);
                k2 = max(k2, b);
            }
        };
        const uint32_t low = uint32_t(63 - lane * 16) << 1;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            put((__funnelshift_l(p.w[i], p.w[i], 17) & 0xfffe0001u) | (low - 4 * i));
            put((__funnelshift_l(p.w[i], p.w[i], 1) & 0xfffe0001u) | (low - 4 * i - 2));
        }
        if constexpr (TOPK == 2) {
            over_group(lanes, [&](int off) {
                const uint32_t o0 = __shfl_xor_sync(0xffffffffu, k0, off);
                const uint32_t o1 = __shfl_xor_sync(0xffffffffu, k1, off);
                const uint32_t o2 = __shfl_xor_sync(0xffffffffu, k2, off);
                put(o0);
                put(o1);
                put(o2);
            });
        } else {                                                         // (straight-line steps spill at five blocks per SM)
            for (int off = lanes / 2; off > 0; off >>= 1) {
                const uint32_t o0 = __shfl_xor_sync(0xffffffffu, k0, off, lanes);
                const uint32_t o1 = __shfl_xor_sync(0xffffffffu, k1, off, lanes);
                put(o0);
                put(o1);
            }
        }
        m.idx[0] = 63 - int((k0 >> 1) & 0xffu);
        m.kept[0] = canonical<T>((k0 >> 17) | ((k0 & 1u) << 15));
        if constexpr (TOPK == 2) {
            m.idx[1] = 63 - int((k1 >> 1) & 0xffu);
            m.kept[1] = canonical<T>((k1 >> 17) | ((k1 & 1u) << 15));
        }
        m.stored = Src<T>::up(uint16_t((TOPK == 1 ? k1 : k2) >> 17));
        m.tame = (k0 >> 17) < inf_bits<T>();
    } else {
        auto largest = [&]() {                                           // -1: nothing but NaN left
            float a = -1.0f;
#pragma unroll
            for (int i = 0; i < 16; ++i) a = fmaxf(a, fabsf(v[i]));
            for (int off = lanes / 2; off > 0; off >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, off, lanes));
            return a;
        };
        if constexpr (!Kind<KIND>::book) {      // (linear codes without a clamp: the first maximum looks for a NaN)
            float top = fabsf(v[0]);
#pragma unroll
            for (int i = 1; i + 1 < 16; i += 2) top = max_nan(top, fabsf(v[i]), fabsf(v[i + 1]));
            top = max_nan(top, fabsf(v[15]));
            over_group(lanes, [&](int off) { top = max_nan(top, __shfl_xor_sync(0xffffffffu, top, off)); });
            m.tame = top < INFINITY;
            m.stored = top;
            if (!__all_sync(0xffffffffu, m.tame)) m.stored = largest();
        } else {
            m.stored = largest();
        }
#pragma unroll
        for (int j = 0; j < TOPK; ++j) {
            int at = -1;
            float value = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (fabsf(v[i]) == m.stored) {
                    at = lane * 16 + i;
                    value = v[i];
                }
            int best = at;
            for (int off = lanes / 2; off > 0; off >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, off, lanes));
            m.idx[j] = best;
            m.kept[j] = __shfl_sync(0xffffffffu, __float_as_uint(value), best < 0 ? 0 : best >> 4, lanes);
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (best == lane * 16 + i) v[i] = __uint_as_float(0x7fffffffu);   // out of the next rounds
            m.stored = largest();
        }
    }
    return m;
}

// ---- the scale of a group without the places of what it keeps ------------------------------------------------------
template <typename T>
__device__ __forceinline__ uint32_t abs_min2(uint32_t a, uint32_t b) {
    uint32_t r;
    if constexpr (std::is_same<T, __half>::value)
        asm("min.NaN.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else
        asm("min.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// All ones in the halves of `a` whose magnitude is above that of `b`, which has no signs.
template <typename T>
__device__ __forceinline__ uint32_t abs_above2(uint32_t a, uint32_t b) {
    uint32_t r;
    if constexpr (std::is_same<T, __half>::value)
        asm("{.reg .b32 m; abs.f16x2 m, %1; set.gt.u32.f16x2 %0, m, %2;}" : "=r"(r) : "r"(a), "r"(b));
    else
        asm("{.reg .b32 m; abs.bf16x2 m, %1; set.gt.u32.bf16x2 %0, m, %2;}" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The (TOPK + 1)-th largest magnitude of a group and the one before it; all `lanes` threads of the group get the answer.
struct GroupTop {
    float stored, last_kept;
    bool finite;               // no infinity and no NaN in the group
};
template <typename T, int TOPK>
__device__ __forceinline__ GroupTop top_of_group(const Packed16<T>& p, int lanes) {
    static_assert(TOPK == 1 || TOPK == 2, "two or three magnitudes");
    GroupTop g;
    if constexpr (sizeof(T) == 2) {
        uint32_t k0 = p.w[0], k1 = 0u, k2 = 0u;                  // per half word, |k0| >= |k1| >= |k2|
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            const uint32_t a = abs_min2<T>(k0, p.w[i]);
            k0 = abs_max2<T>(k0, p.w[i]);
            if (TOPK == 2) k2 = abs_max2<T>(k2, abs_min2<T>(k1, a));
            k1 = abs_max2<T>(k1, a);
        }
        uint32_t t0 = k0 & 0x7fffu, t1 = k1 & 0x7fffu, t2 = k2 & 0x7fffu;
        auto merge = [&](uint32_t o0, uint32_t o1, uint32_t o2) {
            if (TOPK == 2) t2 = max(max(t2, o2), max(min(t0, o1), min(t1, o0)));
            t1 = max(max(t1, o1), min(t0, o0));
            t0 = max(t0, o0);
        };
        merge(k0 >> 16 & 0x7fffu, k1 >> 16 & 0x7fffu, k2 >> 16 & 0x7fffu);
        over_group(lanes, [&](int off) {
            const uint32_t o = __shfl_xor_sync(0xffffffffu, t0 << 16 | t1, off);
            merge(o >> 16, o & 0xffffu, TOPK == 2 ? __shfl_xor_sync(0xffffffffu, t2, off) : 0u);
        });
        g.stored = Src<T>::up(uint16_t(TOPK == 1 ? t1 : t2));
        g.last_kept = Src<T>::up(uint16_t(TOPK == 1 ? t0 : t1));
        g.finite = t0 < inf_bits<T>();
    } else {
        float t0 = 0.0f, t1 = 0.0f, t2 = 0.0f;
        auto merge = [&](float o0, float o1, float o2) {
            if (TOPK == 2) t2 = max3(t2, o2, fmaxf(fminf(t0, o1), fminf(t1, o0)));
            t1 = max3(t1, o1, fminf(t0, o0));
            t0 = max_nan(t0, o0);
        };
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const float a = fabsf(__uint_as_float(p.w[i])), b = fabsf(__uint_as_float(p.w[i + 1]));
            merge(max_nan(a, b), fminf(a, b), 0.0f);
        }
        over_group(lanes, [&](int off) {
            merge(__shfl_xor_sync(0xffffffffu, t0, off), __shfl_xor_sync(0xffffffffu, t1, off),
                  TOPK == 2 ? __shfl_xor_sync(0xffffffffu, t2, off) : 0.0f);
        });
        g.stored = TOPK == 1 ? t1 : t2;
        g.last_kept = TOPK == 1 ? t0 : t1;
        g.finite = t0 < INFINITY;                                // false for NaN
    }
    return g;
}

// Is what a receiver has, the k kept elements verbatim and the others decoded, the same whichever of several equal magnitudes
// are kept?  Everything above the scale is kept in any case, and
//  - nothing else is, if the last kept magnitude is above the scale; or
//  - what else is kept equals the scale, and its own code gives it back (16-bit types: T(L * (scale / L)) = scale for every
//    scale that is not clamped); or
//  - the scale is zero, and what else is kept is +0, like its decoded value.
// Then the places need not be found, which took a key with index and sign through every comparison.
template <typename T, int TOPK>
__device__ __forceinline__ bool kept_by_magnitude(const GroupTop& g, const Packed16<T>& p, bool noise) {
    bool ok = g.finite && g.stored < kNearScale && (g.last_kept > g.stored || (sizeof(T) == 2 && !noise && g.stored >= 1.0e-6f));
    if (__all_sync(0xffffffffu, ok)) return true;
    if (!ok && g.finite && !noise && g.stored == 0.0f) {
        bool minus = false;
#pragma unroll
        for (int i = 0; i < Packed16<T>::kWords; ++i) {
            if (sizeof(T) == 2) minus = minus || (p.w[i] & 0xffffu) == 0x8000u || p.w[i] >> 16 == 0x8000u;
            else minus = minus || p.w[i] == 0x80000000u;
        }
        ok = !minus;
    }
    return __all_sync(0xffffffffu, ok);
}
template <typename T>
__device__ __forceinline__ void keep_above(Packed16<T>& y, const Packed16<T>& from, float stored) {
    if constexpr (sizeof(T) == 2) {
        const uint32_t scale = Src<T>::down2(stored, stored);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t m = abs_above2<T>(from.w[i], scale);
            y.w[i] = (from.w[i] & m) | (y.w[i] & ~m);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (fabsf(__uint_as_float(from.w[i])) > stored) y.w[i] = from.w[i];
    }
}

// Rounding parameters of one call.
constexpr float kThresholdScale = 1152921504606846976.0f;      // 2^60
__device__ __forceinline__ float fma_saturated(float a, float b, float c) {
    float r;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t how) {      // with the sign mode, which __byte_perm lacks
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(how));
    return r;
}
struct CodeRule {
    uint32_t step;             // kBook: the entry of LbcBook::steps that this lane of the warp holds
    float nudge;
    // kBook: thresholds[c] = -2^60 * the largest float below the least t = value / scale whose code is above c
    const float* thresholds;
    const float* table;        // kBookNoise: the code-book
    int stochastic;            // linear
    unsigned long long seed;
    template <int KIND>
    __device__ __forceinline__ static CodeRule of(const LbcBook& book, int quant_type, int stochastic, unsigned long long seed) {
        CodeRule r{0u, 0.0f, book.thresholds, KIND == kBookNoise ? kCodebooks[quant_type - 1] : nullptr, stochastic, seed};
        if (KIND == kBook) {
            r.step = book.steps[threadIdx.x & 31];
            r.nudge = book.nudge;
        }
        return r;
    }
};

// ---- deterministic code-books -----------------------------------------------------------------------------------
// A code is 7 plus or minus the number of thresholds that |t|, t = value / scale, has reached.  The bits of |t| down to its
// second mantissa bit name one of 32 buckets (2^-7 to 2, four to an octave), none of which holds two thresholds in any of the
// four tables; the entry of a bucket, added to the bits below, carries into the count when they reach its threshold.  Each lane
// of the warp holds one entry, and a shuffle, whose index is its five low bits, looks it up.  Counting the fourteen
// thresholds one by one took 28 issue slots per element, this takes six.
// A tie goes to the lower entry, so the two signs differ by the last bit of |t|: the sign is appended to it.  Two thresholds
// at powers of two (the lowest of e3m0 and of e2m1) differ by more, because the rule's t - entry rounds there; `nudge`, half
// a bit of the octave below them, takes both signs to the same side.
// t, correctly rounded where that decides: value * (1 / scale) with one Newton correction by its exact remainder (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000", 1990).  Before its rounding the corrected quotient is off
// by 3 * 2^-24 ulp at most; quotients of two floats that lie nearer than ten times that to a rounding boundary beside a threshold
// solve v * 2^k = m * s + d for a small d, and none of them rounds wrongly; quotients of 16-bit operands lie 2^-11 ulp away.
// It holds for scales up to 1e30 (nothing that decides overflows or underflows) with no value above the scale but kept ones.
struct BookCode {
    uint32_t bits;             // the count in the top byte
    uint32_t t;                // the sign on top
};
__device__ __forceinline__ BookCode book_code(float v, float safe, float inverse, const CodeRule& rule) {
    float t = __fmul_rn(v, inverse);
    t = __fmaf_rn(__fmaf_rn(-t, safe, v), inverse, t);
    BookCode c;
    c.t = __float_as_uint(__fsub_rn(t, rule.nudge));
    const uint32_t key = max(__funnelshift_l(c.t, c.t, 1), 0x78000000u);      // no threshold below 2^-7.  NaN: the last bucket, 7
    c.bits = key * 4u + __shfl_sync(0xffffffffu, rule.step, int(key >> 22));
    return c;
}
// Eight of them -> one word of wire-ordered codes (see pack16_low_nibbles): 7 + count, or 7 - count = 7 ^ count.
template <int WordBytes>
__device__ __forceinline__ uint32_t pack_book(const BookCode (&c)[8]) {
    uint32_t k[2], s[2];
#pragma unroll
    for (int odd = 0; odd < 2; ++odd) {
        const BookCode &a = c[odd], &b = c[2 + odd], &d = c[4 + odd], &e = c[6 + odd];
        const uint32_t k0 = prmt(b.bits, a.bits, 0x0073), k1 = prmt(e.bits, d.bits, 0x0073);
        const uint32_t s0 = prmt(b.t, a.t, 0x00fb), s1 = prmt(e.t, d.t, 0x00fb);      // 0xff where the sign is set
        k[odd] = WordBytes == 2 ? prmt(k0, k1, 0x5410) : prmt(k1, k0, 0x5410);
        s[odd] = WordBytes == 2 ? prmt(s0, s1, 0x5410) : prmt(s1, s0, 0x5410);
    }
    const uint32_t counts = ((k[0] << 4) & 0xf0f0f0f0u) | (k[1] & 0x0f0f0f0fu);
    const uint32_t signs = (s[0] & 0xf0f0f0f0u) | (s[1] & 0x0f0f0f0fu);
    return ((counts ^ signs) & 0x77777777u) + (~signs & 0x77777777u);
}
// A scale that is infinite, NaN or above 1e30: the machine's division and one saturated multiply-add per threshold (1 when
// t has reached it, else 0: the exact difference times 2^60 is above 1 or not above 0).  NaN: 14, as the search has it.
__device__ __noinline__ void book_codes_far(const float* v, float safe, const float* thresholds, uint32_t* b) {
    for (int i = 0; i < 16; ++i) {
        const float t = v[i] / safe;
        float q = kRoundMagic;
        for (int c = 0; c < 14; ++c) q += fma_saturated(t, kThresholdScale, thresholds[c]);
        b[i] = __float_as_uint(t == t ? q : kRoundMagic + 14.0f);
    }
}
// Is the scale of every group of the warp one that book_code takes?  (A 16-bit group with more NaN than it keeps has NaN for
// its scale, which bounds no value: the test is on the scale as stored, false for NaN.)
__device__ __forceinline__ bool book_near(float stored) { return __all_sync(0xffffffffu, stored < kNearScale); }

// Codes of 16 values against the group's scale, as bit patterns whose low byte (nibble) is the code.  With `near` (no infinity, no
// NaN and no scale above kNearScale in any group of the warp) no value that is not kept verbatim is larger than the scale, so
// |value * mul| rounds to at most the limit, neither the clamp nor the test for NaN has anything to do, and the quotient
// needs no branch.  kPacked: products two to an instruction and that quotient; without, the 16-bit encoders are a little faster (4 Mi bf16
// elements in records, one kept value, 5.11 / 5.04 us; fp32 ones 5.43 / 6.46).
template <int KIND, bool kPacked>
__device__ __forceinline__ void encode_general(const float (&v)[16], float stored, bool near, const CodeRule& rule,
                                               int64_t first, uint32_t (&b)[16]) {
    static_assert(KIND != kBook, "book_code");
    constexpr int lim = Kind<KIND>::lim;
#pragma unroll
    for (int i = 0; i < 16; ++i) b[i] = 0u;
    const float safe = fmaxf(stored, 1.0e-6f);
    if constexpr (!Kind<KIND>::book) {
        float t[16];
        if (kPacked && near && !rule.stochastic) {
#pragma unroll
            for (int i = 0; i < 16; ++i) t[i] = v[i];
            fma16(t, limit_over<lim>(safe), 0.0f);             // (see encode16_near)
            add16(t, kRoundMagic);
#pragma unroll
            for (int i = 0; i < 16; ++i) b[i] = __float_as_uint(t[i]);
            return;
        }
        const float mul = float(lim) / safe;
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = __fmul_rn(v[i], mul);
        if (!kPacked && near && !rule.stochastic) {
            add16(t, kRoundMagic);
#pragma unroll
            for (int i = 0; i < 16; ++i) b[i] = __float_as_uint(t[i]);
            return;
        }
        if (rule.stochastic) {      // two roundings, the product's and the sum's, as the oracle has it
#pragma unroll
            for (int i = 0; i < 16; ++i)
                t[i] = __fadd_rn(t[i], uniform01(rule.seed, (unsigned long long)(first + i)) - 0.5f);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float r = __fadd_rn(t[i] == t[i] ? t[i] : 0.0f, kRoundMagic);   // rint(t) in the low bits; NaN: code 0
            b[i] = __float_as_uint(fminf(fmaxf(r, kRoundMagic - float(lim)), kRoundMagic + float(lim)));
        }
    } else {
        // The last entry that is not above t, by looking at all of them in order: their addresses are the same for every
        // thread, where a search's are not (constant memory serves one address at a time).  NaN: the last, 14.
        // Encode of 16 Mi elements, an unrolled search / a search in a loop over the elements / here: bf16 158 / 187 / 94 us,
        // fp32 179 / 187 / 95.
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float t = v[i] / safe;
            float below = rule.table[0], gap = rule.table[1] - rule.table[0];
            uint32_t lo = 0u;
#pragma unroll
            for (int c = 1; c < 15; ++c) {
                const bool reached = !(t < rule.table[c]);
                lo += reached ? 1u : 0u;
                below = reached ? rule.table[c] : below;
                gap = reached ? rule.table[c + 1] - rule.table[c] : gap;
            }
            const bool up = uniform01(rule.seed, (unsigned long long)(first + i)) < (t - below) / gap;
            b[i] = lo + (up ? 1u : 0u);
        }
    }
}

template <typename T, int KIND>
__device__ __forceinline__ void pack_codes(const uint32_t (&b)[16], uint32_t (&w)[4]) {
    if constexpr (KIND == kLinear8) {
        const uint4 c = pack16_low_bytes<sizeof(T)>(b);
        w[0] = c.x; w[1] = c.y; w[2] = c.z; w[3] = c.w;
    } else {
        const uint2 c = pack16_low_nibbles<sizeof(T)>(b);
        w[0] = c.x; w[1] = c.y; w[2] = w[3] = 0u;
    }
}

// Values to packed codes.  Convergent.
template <typename T, int KIND>
__device__ __forceinline__ void encode_words(const float (&v)[16], float stored, bool near, const CodeRule& rule,
                                             int64_t first, uint32_t (&w)[4]) {
    uint32_t b[16];
    if constexpr (KIND == kBook) {
        const float safe = fmaxf(stored, 1.0e-6f);
        if (book_near(stored)) {
            const float inverse = __frcp_rn(safe);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                BookCode c[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) c[e] = book_code(v[8 * j + e], safe, inverse, rule);
                w[j] = pack_book<sizeof(T)>(c);
            }
            w[2] = w[3] = 0u;
            return;
        }
        float far[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) far[i] = v[i];
        book_codes_far(far, safe, rule.thresholds, b);
    } else {
        encode_general<KIND, sizeof(T) == 4>(v, stored, near, rule, first, b);
    }
    pack_codes<T, KIND>(b, w);
}

// 16 codes -> T(value), scale applied; `lut` is the code-book in shared memory.
template <typename T, int KIND>
__device__ __forceinline__ Packed16<T> decode_codes(const uint32_t (&w)[4], float stored, const float* lut) {
    float d[16];
    if constexpr (KIND == kLinear8) {
        unpack16_i8_fast<sizeof(T)>(make_uint4(w[0], w[1], w[2], w[3]), d);
        const float step = stored / 127.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) d[i] = __fmul_rn(d[i], step);
    } else {
        const float step = KIND == kLinear4 ? stored / 7.0f : stored;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t hi = (w[j] >> 4) & 0x0f0f0f0fu, lo = w[j] & 0x0f0f0f0fu;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int byte = e >> 1, pos = sizeof(T) == 2 ? byte ^ 1 : 3 - byte;
                const uint32_t four = (e & 1) ? lo : hi;
                float value;
                if constexpr (KIND == kLinear4)     // (c ^ 8) in the mantissa of 2^23, minus 2^23 + 8: exact
                    value = __uint_as_float(__byte_perm(four ^ 0x08080808u, 0x4B000000u, 0x7540 | pos)) - 8388616.0f;
                else
                    value = lut[(four >> (8 * pos)) & 0xfu];
                d[8 * j + e] = __fmul_rn(value, step);
            }
        }
    }
    return pack_elems<T>(d);
}

// The same from the patterns of encode_general, without a trip through packed bytes.
template <typename T, int KIND>
__device__ __forceinline__ Packed16<T> decode_bits(const uint32_t (&b)[16], float stored, const float* lut) {
    float d[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) d[i] = Kind<KIND>::book ? lut[b[i] & 0xfu] : __uint_as_float(b[i]);
    if constexpr (Kind<KIND>::book) {
        mul16(d, stored);
    } else {
        add16(d, -kRoundMagic);
        mul16(d, over_limit<Kind<KIND>::lim>(stored));
    }
    return pack_elems<T>(d);
}

// Values -> T(decode(encode(value))).  Convergent.
template <typename T, int KIND>
__device__ __forceinline__ Packed16<T> requantize(const float (&v)[16], float stored, bool near, const CodeRule& rule,
                                                  int64_t first, const float* lut) {
    uint32_t b[16];
    if constexpr (KIND == kBook) {
        const float safe = fmaxf(stored, 1.0e-6f);
        if (book_near(stored)) {
            const float inverse = __frcp_rn(safe);
            const float entry = lut[7 + (threadIdx.x & 7)];             // the entries from zero on, one per lane
            float d[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const BookCode c = book_code(v[i], safe, inverse, rule);
                const float size = __shfl_sync(0xffffffffu, entry, int(c.bits >> 24), 8);
                // (adding zero makes the zero of code 7 positive, as the decoder's product is)
                d[i] = __fmaf_rn(size, __uint_as_float(__float_as_uint(stored) ^ (c.t & 0x80000000u)), 0.0f);
            }
            return pack_elems<T>(d);
        }
        float far[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) far[i] = v[i];
        book_codes_far(far, safe, rule.thresholds, b);
    } else {
        encode_general<KIND, true>(v, stored, near, rule, first, b);
    }
    return decode_bits<T, KIND>(b, stored, lut);
}

template <int KIND>
__device__ __forceinline__ void load_code_words(const uint8_t* p, uint32_t (&w)[4], bool vec) {
    if (vec) {
        if constexpr (KIND == kLinear8) {
            const uint4 c = ld16(p);
            w[0] = c.x; w[1] = c.y; w[2] = c.z; w[3] = c.w;
        } else {
            const uint2 c = *reinterpret_cast<const uint2*>(p);
            w[0] = c.x; w[1] = c.y; w[2] = w[3] = 0u;
        }
    } else {
        load_bytes<Kind<KIND>::CB>(p, w);
    }
}

// Reads the metadata of a group; decode_group turns one thread's codes into elements with the kept ones written back.
template <typename T, int TOPK, int KIND>
__device__ __forceinline__ Packed16<T> decode_group(const uint32_t (&w)[4], const uint8_t* meta, int lane, const float* lut) {
    Packed16<T> p = decode_codes<T, KIND>(w, value_of<T>(load_word<T>(meta)), lut);
    if constexpr (TOPK >= 1) {
        const uint32_t index_word = load_word<T>(meta + sizeof(T));
#pragma unroll
        for (int j = 0; j < TOPK; ++j) {
            const int at = int((index_word >> (8 * j)) & 0xffu) - lane * 16;
            patch_elem<T>(p, at, canonical<T>(load_word<T>(meta + (2 + j) * sizeof(T))));
        }
    }
    return p;
}

// Geometry shared by the kernels: thread `chunk` owns 16 elements, `lanes` threads a group.
struct GroupShape {
    int shift, lanes, VB, MB;
    template <typename T, int TOPK, int KIND>
    __device__ __forceinline__ static GroupShape of(int group_size) {
        GroupShape s;
        s.shift = group_size == 64 ? 2 : (group_size == 32 ? 1 : 0);
        s.lanes = 1 << s.shift;
        s.VB = group_size * Kind<KIND>::bit / 8;
        s.MB = meta_words(TOPK) * int(sizeof(T));
        return s;
    }
};

// The words of a group's metadata, dealt to the threads of the group.
template <typename T, int TOPK>
__device__ __forceinline__ void put_meta(uint8_t* meta, const GroupMeta& m, int lane, int lanes) {
    const uint32_t scale = bits_of<T>(m.stored);
    uint32_t index_word = uint32_t(m.idx[0]);
    if (TOPK == 2) index_word |= uint32_t(m.idx[1]) << 8;
#pragma unroll
    for (int i = 0; i < meta_words(TOPK); ++i) {
        const uint32_t word = i == 0 ? scale : (i == 1 ? index_word : m.kept[i == 2 ? 0 : 1]);
        if ((i & (lanes - 1)) == lane) store_word<T>(meta + i * sizeof(T), word);
    }
}

template <typename T, int TOPK, int KIND>
__global__ void __launch_bounds__(kThreads, 4) quant_general_kernel(const __grid_constant__ LbcQuantGeneral p) {
    chain_wait();
    const GroupShape shape = GroupShape::of<T, TOPK, KIND>(p.group_size);
    const int lanes = shape.lanes, VB = shape.VB, MB = shape.MB;
    constexpr int CB = Kind<KIND>::CB;
    const T* x = static_cast<const T*>(p.x);
    const T* res = static_cast<const T*>(p.residual);
    T* prep = static_cast<T*>(p.prepared_out);
    const int64_t n = p.numel;
    const int64_t num_groups = (n + p.group_size - 1) / p.group_size;
    const int64_t num_chunks = num_groups << shape.shift;
    const int64_t chunk_span = (num_chunks + 31) / 32 * 32;
    const bool x_vec = (reinterpret_cast<uintptr_t>(x) & 31) == 0;
    const bool r_vec = (reinterpret_cast<uintptr_t>(res) & 31) == 0;
    const bool p_vec = (reinterpret_cast<uintptr_t>(prep) & 31) == 0;
    const bool scatter = p.num_dst > 0 && p.shard_groups > 0;
    const int copies = (p.num_dst > 0 && !scatter) ? p.num_dst : 1;
    const CodeRule rule = CodeRule::of<KIND>(p.book, p.quant_type, p.stochastic, p.seed);
    for (int64_t chunk = int64_t(blockIdx.x) * kThreads + threadIdx.x; chunk < chunk_span;
         chunk += int64_t(gridDim.x) * kThreads) {
        const bool live = chunk < num_chunks;
        const int64_t first = chunk * kElemsPerThread;
        const int64_t g = chunk >> shape.shift;
        const int lane = int(chunk) & (lanes - 1);
        Packed16<T> elems = load_elems<T>(x, first, n, x_vec);          // zeros past the end
        float v[16];
        unpack_elems<T>(elems, v);
        if (res != nullptr) {
            float r[16];
            unpack_elems<T>(load_elems<T>(res, first, n, r_vec), r);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += r[i];
            elems = pack_elems<T>(v);
            if constexpr (sizeof(T) == 2) unpack_elems<T>(elems, v);
        }
        if (prep != nullptr && live) store_elems<T>(prep, first, n, p_vec, res != nullptr ? elems : pack_elems<T>(v));
        const GroupMeta m = select_group<T, TOPK, KIND>(v, elems, lane, lanes);
        uint32_t w[4];
        encode_words<T, KIND>(v, m.stored, all_near<KIND>(m), rule, first, w);
#pragma unroll
        for (int j = 0; j < TOPK; ++j) patch_code<T, KIND>(w, m.idx[j] - lane * 16);
        if (!live) continue;
        for (int d = 0; d < copies; ++d) {      // one payload, the same payload in every rank's slot, or one shard
            uint8_t* base = p.num_dst > 0 ? p.dst[d] : p.out;
            int64_t gl = g, layout = num_groups;
            if (scatter) {
                const int64_t owner = g / p.shard_groups;
                base = p.dst[owner];
                gl = g - owner * p.shard_groups;
                layout = p.shard_groups;
            }
            uint8_t* vptr = p.compact ? base + gl * (VB + MB) : base + gl * VB;
            uint8_t* mptr = p.compact ? vptr + VB : base + layout * VB + gl * MB;
            vptr += lane * CB;
            if ((reinterpret_cast<uintptr_t>(vptr) & (CB - 1)) == 0) {
                if constexpr (CB == 16)
                    st16(vptr, make_uint4(w[0], w[1], w[2], w[3]));
                else
                    *reinterpret_cast<uint2*>(vptr) = make_uint2(w[0], w[1]);
            } else {
                store_bytes<CB>(vptr, w);
            }
            put_meta<T, TOPK>(mptr, m, lane, lanes);
        }
    }
    grid_signal(p.signal);      // no-op without destinations to notify
}

// Encode of a payload of this GPU alone, on its vectors: no destinations, shards or signal, whole tiles without a test per
// chunk.  kCompact: records, built in shared memory.
// What bounds it: instruction issue.  quant_general_kernel, which asks every chunk where it goes, and here, 64 MiB beyond L2:
// bf16, one kept value 34.8 -> 30.6 us, e2m1 36.8 -> 31.1, fp32 25.6 -> 20.7 and 22.0 -> 17.4.
// Blocks per SM with a residual, 4 / 5 (no spills at either in these), 64 MiB: bf16, one kept value 32.1 / 30.6, two 39.8 /
// 40.3, e2m1 31.9 / 33.8; fp32 23.0 / 21.7, 29.3 / 27.5, 19.0 / 18.9, e2m1 with one kept value 23.8 / 25.1.
template <typename T, int TOPK, int KIND>
constexpr int encode_blocks() {
    if (KIND == kBook) return sizeof(T) == 4 && TOPK == 0 ? 5 : 4;
    return KIND != kBookNoise && (TOPK == 1 || (TOPK == 2 && sizeof(T) == 4)) ? 5 : 4;
}
// kPrepare: with a residual or prepared_out.  Without, in kernels that know it, four blocks per SM, 16-bit code-books five:
// 4 / 5, bf16, one kept value 2 Mi elements 2.74 / 3.37, 8 Mi 8.10 / 8.28, two 9.97 / 10.5, e2m1 8.67 / 8.16; fp32, one kept
// value 4 Mi 4.60 / 5.20, e2m1 5.09 / 5.40.
template <typename T, int KIND>
constexpr int encode_plain_blocks() { return KIND == kBook && sizeof(T) == 2 ? 5 : 4; }
template <typename T, int TOPK, int KIND, bool kCompact, bool kPrepare>
__global__ void __launch_bounds__(kThreads, kPrepare ? encode_blocks<T, TOPK, KIND>() : encode_plain_blocks<T, KIND>())
encode_general_kernel(const __grid_constant__ LbcQuantGeneral p) {
    chain_wait();
    const GroupShape shape = GroupShape::of<T, TOPK, KIND>(p.group_size);
    const int lanes = shape.lanes, VB = shape.VB, MB = shape.MB;
    constexpr int CB = Kind<KIND>::CB;
    const T* x = static_cast<const T*>(p.x);
    const T* res = kPrepare ? static_cast<const T*>(p.residual) : nullptr;
    T* prep = kPrepare ? static_cast<T*>(p.prepared_out) : nullptr;
    const int64_t n = p.numel;
    const int64_t num_groups = (n + p.group_size - 1) >> (shape.shift + 4);
    const int64_t num_chunks = num_groups << shape.shift;
    const bool x_vec = (reinterpret_cast<uintptr_t>(x) & 31) == 0, r_vec = (reinterpret_cast<uintptr_t>(res) & 31) == 0;
    const bool p_vec = (reinterpret_cast<uintptr_t>(prep) & 31) == 0, vec = x_vec && r_vec && p_vec;
    __shared__ __align__(16) uint8_t spans[kThreads / 32][kCompact ? kWarpSpan : 16];
    const CodeRule rule = CodeRule::of<KIND>(p.book, p.quant_type, p.stochastic, p.seed);
    const int lane = threadIdx.x & (lanes - 1), wlane = threadIdx.x & 31;      // (a tile is whole groups)

    for (int64_t c0 = int64_t(blockIdx.x) * kThreads; c0 < num_chunks; c0 += int64_t(gridDim.x) * kThreads) {
        const int64_t chunk = c0 + threadIdx.x, first = chunk * kElemsPerThread;
        // (fp32 with fewer than two kept values is faster with the tests: 64 MiB, e2m1 18.9 -> 17.4 us, one kept value 21.6 -> 20.7, two
        // 27.6 -> 29.2)
        const bool whole = (sizeof(T) == 2 || TOPK == 2) && vec && (c0 + kThreads) * kElemsPerThread <= n;
        const bool live = whole || chunk < num_chunks;
        const int64_t end = whole ? first + 16 : n;                            // (folds the tests of a whole tile)
        Packed16<T> elems = load_elems<T>(x, first, end, whole || x_vec);                 // zeros past the end
        float v[16];
        unpack_elems<T>(elems, v);
        if (res != nullptr) {
            float r[16];
            unpack_elems<T>(load_elems<T>(res, first, end, whole || r_vec), r);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += r[i];
            elems = pack_elems<T>(v);
            if constexpr (sizeof(T) == 2) unpack_elems<T>(elems, v);
        }
        if (prep != nullptr && live) store_elems<T>(prep, first, end, whole || p_vec, res != nullptr ? elems : pack_elems<T>(v));
        const GroupMeta m = select_group<T, TOPK, KIND>(v, elems, lane, lanes);
        uint32_t w[4];
        encode_words<T, KIND>(v, m.stored, all_near<KIND>(m), rule, first, w);
#pragma unroll
        for (int j = 0; j < TOPK; ++j) patch_code<T, KIND>(w, m.idx[j] - lane * 16);
        if constexpr (kCompact) {
            uint8_t* span = spans[threadIdx.x >> 5];
            uint8_t* rec = span + (wlane >> shape.shift) * (VB + MB);
            span_put_codes<CB>(rec + lane * CB, w);
            put_meta<T, TOPK>(rec + VB, m, lane, lanes);
            __syncwarp();
            const int64_t g0 = (chunk - wlane) >> shape.shift;
            const int groups = whole ? 32 >> shape.shift : int(max(int64_t(0), min(int64_t(32 >> shape.shift), num_groups - g0)));
            span_to_global(p.out + g0 * (VB + MB), span, groups * (VB + MB), wlane);
            __syncwarp();
        } else if (live) {
            uint8_t* codes = p.out + chunk * CB;
            if constexpr (CB == 16)
                st16(codes, make_uint4(w[0], w[1], w[2], w[3]));
            else
                *reinterpret_cast<uint2*>(codes) = make_uint2(w[0], w[1]);
            put_meta<T, TOPK>(p.out + num_groups * VB + (chunk >> shape.shift) * MB, m, lane, lanes);
        }
    }
}

// The code-book in shared memory: 15 words in 15 banks, so a warp's look-ups never conflict (the constant cache
// serialises them).  Block-wide.
template <int KIND>
__device__ __forceinline__ void load_lut(float (&lut)[16], int quant_type) {
    if constexpr (Kind<KIND>::book) {
        if (threadIdx.x < 16) lut[threadIdx.x] = kCodebooks[quant_type - 1][threadIdx.x];
        __syncthreads();
    }
}

// kMayAdd: with p.accumulate, out = T(out + decode).
template <typename T, int TOPK, int KIND, bool kMayAdd, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) dequant_general_kernel(const __grid_constant__ LbcDequantGeneral p) {
    chain_wait();
    const GroupShape shape = GroupShape::of<T, TOPK, KIND>(p.group_size);
    const int lanes = shape.lanes, VB = shape.VB, MB = shape.MB;
    constexpr int CB = Kind<KIND>::CB;
    __shared__ float lut[16];
    load_lut<KIND>(lut, p.quant_type);
    T* out = static_cast<T*>(p.out);
    const int64_t n = p.numel;
    const int64_t num_groups = (n + p.group_size - 1) / p.group_size;
    const int64_t num_chunks = num_groups << shape.shift;
    const bool o_vec = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
    const bool c_vec = !p.compact && (reinterpret_cast<uintptr_t>(p.src) & (CB - 1)) == 0;
    for (int64_t chunk = int64_t(blockIdx.x) * kThreads + threadIdx.x; chunk < num_chunks;
         chunk += int64_t(gridDim.x) * kThreads) {
        const int64_t first = chunk * kElemsPerThread;
        const int64_t g = chunk >> shape.shift;
        const int lane = int(chunk) & (lanes - 1);
        // Records are read where they lie.  Turning a warp's span of them through shared memory, as the encoder does, was as
        // fast or slower in every profile (16 Mi elements, records of 64 / k = 1, 16 / k = 2, int8: bf16 18.9 against 17.2 us,
        // 22.9 against 18.8; fp32 20.9 against 20.1, 26.9 against 23.0).
        const uint8_t* vptr = p.compact ? p.src + g * (VB + MB) : p.src + g * VB;
        const uint8_t* meta = p.compact ? vptr + VB : p.src + num_groups * VB + g * MB;
        uint32_t w[4];
        load_code_words<KIND>(vptr + lane * CB, w, c_vec);
        Packed16<T> d = decode_group<T, TOPK, KIND>(w, meta, lane, lut);
        if (kMayAdd && p.accumulate) {
            float a[16], b[16];
            unpack_elems<T>(d, a);
            unpack_elems<T>(load_elems<T>(out, first, n, o_vec), b);
#pragma unroll
            for (int i = 0; i < 16; ++i) a[i] += b[i];
            d = pack_elems<T>(a);
        }
        store_elems<T>(out, first, n, o_vec, d);
    }
}

template <typename T, int TOPK, int KIND>
__global__ void __launch_bounds__(kThreads) reduce_general_kernel(const __grid_constant__ LbcReduceGeneral p) {
    if (!block_wait(p.wait)) return;      // bounded; the status word says which flag never came
    const GroupShape shape = GroupShape::of<T, TOPK, KIND>(p.group_size);
    const int lanes = shape.lanes, VB = shape.VB, MB = shape.MB;
    constexpr int CB = Kind<KIND>::CB;
    __shared__ float lut[16];
    load_lut<KIND>(lut, p.quant_type);
    T* out = static_cast<T*>(p.out);
    const T* prep = static_cast<const T*>(p.prepared);
    T* res = static_cast<T*>(p.residual_out);
    const int64_t n = p.numel;
    const int64_t num_groups = (n + p.group_size - 1) / p.group_size;
    const int64_t num_chunks = num_groups << shape.shift;
    const bool o_vec = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
    const bool p_vec = (reinterpret_cast<uintptr_t>(prep) & 31) == 0;
    const bool r_vec = (reinterpret_cast<uintptr_t>(res) & 31) == 0;
    auto decode = [&](const uint8_t* src, int64_t layout, int64_t g, int lane) {
        const uint8_t* vptr = p.compact ? src + g * (VB + MB) : src + g * VB;
        const uint8_t* meta = p.compact ? vptr + VB : src + layout * VB + g * MB;
        uint32_t w[4];
        vptr += lane * CB;
        load_code_words<KIND>(vptr, w, (reinterpret_cast<uintptr_t>(vptr) & (CB - 1)) == 0);
        return decode_group<T, TOPK, KIND>(w, meta, lane, lut);
    };
    for (int64_t chunk = int64_t(blockIdx.x) * kThreads + threadIdx.x; chunk < num_chunks;
         chunk += int64_t(gridDim.x) * kThreads) {
        const int64_t first = chunk * kElemsPerThread;
        const int64_t g = chunk >> shape.shift;
        const int lane = int(chunk) & (lanes - 1);
        float acc[16];
        if (p.src_shard_groups > 0) {
            // gather: the group lives in exactly one source, its owner's reduced shard
            const int64_t owner = g / p.src_shard_groups;
            unpack_elems<T>(decode(p.src[owner], p.src_shard_groups, g - owner * p.src_shard_groups, lane), acc);
        } else {
            const int64_t layout = p.layout_groups > 0 ? p.layout_groups : num_groups;
            unpack_elems<T>(decode(p.src[0], layout, g, lane), acc);
            for (int r = 1; r < p.num_src; ++r) {
                float d[16];
                unpack_elems<T>(decode(p.src[r], layout, g, lane), d);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[i] += d[i];
                round16<T>(acc);                // the sum lives in the source dtype between payloads
            }
        }
        if (p.scale != 1.0f) {
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] *= p.scale;
            round16<T>(acc);
        }
        if (prep != nullptr) {
            float e[16];
            load16<T>(prep, first, n, p_vec, e, prep != res);
#pragma unroll
            for (int i = 0; i < 16; ++i) e[i] -= acc[i];
            store16<T>(res, first, n, r_vec, e);
        }
        store16<T>(out, first, n, o_vec, acc);
    }
}

// 16 elements -> what a receiver has of them, with the places of the kept ones.  Convergent.
template <typename T, int TOPK, int KIND>
__device__ __forceinline__ Packed16<T> place_and_requantize(Packed16<T> y, int lane, int lanes, const CodeRule& rule,
                                                            int64_t first, const float* lut) {
    float v[16];
    unpack_elems<T>(y, v);
    const GroupMeta m = select_group<T, TOPK, KIND>(v, y, lane, lanes);
    if (sizeof(T) == 2 && !__all_sync(0xffffffffu, m.tame)) y = pack_elems<T>(v);          // a NaN that is kept has one pattern
    const Packed16<T> from = y;
    y = requantize<T, KIND>(v, m.stored, all_near<KIND>(m), rule, first, lut);
#pragma unroll
    for (int j = 0; j < TOPK; ++j) copy_elem<T>(y, from, int(uint32_t(m.idx[j]) & 0xffu) - lane * 16);
    return y;
}
// The same out of line, for the few warps of a 16-bit pass that need it: inline it cost every warp of them its registers.
template <typename T, int TOPK, int KIND>
__device__ __noinline__ void requantize_by_place(uint32_t* words, int lane, int lanes, const LbcRoundtripGeneral& p,
                                                 int64_t first, const float* lut) {
    const CodeRule rule = CodeRule::of<KIND>(p.book, p.quant_type, p.stochastic, p.seed);
    Packed16<T> y;
#pragma unroll
    for (int i = 0; i < Packed16<T>::kWords; ++i) y.w[i] = words[i];
    y = place_and_requantize<T, TOPK, KIND>(y, lane, lanes, rule, first, lut);
#pragma unroll
    for (int i = 0; i < Packed16<T>::kWords; ++i) words[i] = y.w[i];
}

// The all-reduce of a group of one rank: encode and decode in registers, no payload (see roundtrip_kernels.cu; here
// the decoded values are rounded to T before the residual is taken, the rule of these profiles).
// Blocks per SM, 16-bit, with a residual 4 against 5, 32 Mi bf16: one kept value 26.6 / 27.5 us, two 28.2 / 29.1; others: see the launcher.
// kFull: with a residual or two passes.  kPlain: neither.  kPlainAhead: neither, and the loads of a block's next tile are issued
// ahead of the work on the present one (which waits for its loads at four blocks per SM otherwise: ncu, long scoreboard 3.6
// per issue).
enum : int { kFull = 0, kPlain = 1, kPlainAhead = 2 };
template <typename T, int TOPK, int KIND, int kForm>
__device__ __forceinline__ void roundtrip_general(const LbcRoundtripGeneral& p) {
    constexpr bool by_magnitude = TOPK >= 1 && KIND != kBookNoise;
    const GroupShape shape = GroupShape::of<T, TOPK, KIND>(p.group_size);
    const int lanes = shape.lanes;
    __shared__ float lut[16];
    load_lut<KIND>(lut, p.quant_type);
    const T* x = static_cast<const T*>(p.x);
    const T* res = kForm == kFull ? static_cast<const T*>(p.residual) : nullptr;
    T* out = static_cast<T*>(p.out);
    T* rout = kForm == kFull ? static_cast<T*>(p.residual_out) : nullptr;
    const int passes = kForm == kFull ? p.passes : 1;
    const int64_t n = p.numel;
    const int64_t num_chunks = (n + p.group_size - 1) >> (shape.shift + 4) << shape.shift;
    const int64_t chunk_span = (num_chunks + 31) / 32 * 32;
    const bool vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(res) |
                       reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(rout)) & 31) == 0;
    const CodeRule rule = CodeRule::of<KIND>(p.book, p.quant_type, p.stochastic, p.seed);
    // 16-bit tensors: tile by tile, whole ones without a test per chunk (32 Mi bf16 elements, e2m1 40.7 -> 38.0 us; 8 Mi, one kept value
    // 9.6 -> 9.3).  fp32: chunk by chunk (by tiles it spills: 16 Mi elements, one kept value, 22.6 -> 30.4 us).
    constexpr bool tiles = sizeof(T) == 2;
    const auto whole_at = [&](int64_t at) { return tiles && vec && (at + kThreads) * kElemsPerThread <= n; };
    Packed16<T> next;
    if (kForm == kPlainAhead && whole_at(int64_t(blockIdx.x) * kThreads))
        next = load_elems<T>(x, (int64_t(blockIdx.x) * kThreads + threadIdx.x) * kElemsPerThread, n, true);
    for (int64_t at = int64_t(blockIdx.x) * kThreads + (tiles ? 0 : threadIdx.x); at < (tiles ? num_chunks : chunk_span);
         at += int64_t(gridDim.x) * kThreads) {
        const int64_t chunk = tiles ? at + threadIdx.x : at;
        const bool whole = whole_at(at);
        const bool live = whole || chunk < num_chunks;
        const int64_t first = chunk * kElemsPerThread, end = whole ? first + 16 : n;
        const int lane = tiles ? int(threadIdx.x) & (lanes - 1) : int(chunk) & (lanes - 1);
        Packed16<T> elems;
        if (kForm == kPlainAhead && whole) elems = next;
        else elems = load_elems<T>(x, first, end, vec);                 // zeros past the end
        if (kForm == kPlainAhead) {
            const int64_t then = at + int64_t(gridDim.x) * kThreads;
            const int64_t from = (then + threadIdx.x) * kElemsPerThread;
            if (whole_at(then)) next = load_elems<T>(x, from, from + 16, true);
        }
        if (res != nullptr) {
            float v[16], r[16];
            unpack_elems<T>(elems, v);
            unpack_elems<T>(load_elems<T>(res, first, end, vec), r);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += r[i];
            elems = pack_elems<T>(v);
        }
        Packed16<T> y = elems;
        for (int pass = 0; pass < passes; ++pass) {
            if constexpr (by_magnitude) {
                const GroupTop top = top_of_group<T, TOPK>(y, lanes);
                if (kept_by_magnitude<T, TOPK>(top, y, p.stochastic)) {
                    float v[16];
                    unpack_elems<T>(y, v);
                    const Packed16<T> from = y;
                    y = requantize<T, KIND>(v, top.stored, true, rule, first, lut);
                    keep_above<T>(y, from, top.stored);
                } else if constexpr (sizeof(T) == 4) {
                    y = place_and_requantize<T, TOPK, KIND>(y, lane, lanes, rule, first, lut);
                } else {
                    uint32_t words[Packed16<T>::kWords];
#pragma unroll
                    for (int i = 0; i < Packed16<T>::kWords; ++i) words[i] = y.w[i];
                    requantize_by_place<T, TOPK, KIND>(words, lane, lanes, p, first, lut);
#pragma unroll
                    for (int i = 0; i < Packed16<T>::kWords; ++i) y.w[i] = words[i];
                }
            } else {
                y = place_and_requantize<T, TOPK, KIND>(y, lane, lanes, rule, first, lut);
            }
        }
        if (!live) continue;
        if (rout != nullptr) {
            float a[16], e[16];
            unpack_elems<T>(y, a);
            unpack_elems<T>(elems, e);
#pragma unroll
            for (int i = 0; i < 16; ++i) e[i] -= a[i];
            store_elems<T>(rout, first, end, vec, pack_elems<T>(e));
        }
        store_elems<T>(out, first, end, vec, y);
    }
}

template <typename T, int TOPK, int KIND, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) roundtrip_general_kernel(const __grid_constant__ LbcRoundtripGeneral p) {
    chain_wait();
    roundtrip_general<T, TOPK, KIND, kFull>(p);
}
template <typename T, int TOPK, int KIND, int kBlocks, bool kAhead>
__global__ void __launch_bounds__(kThreads, kBlocks) roundtrip_plain_kernel(const __grid_constant__ LbcRoundtripGeneral p) {
    chain_wait();
    roundtrip_general<T, TOPK, KIND, kAhead ? kPlainAhead : kPlain>(p);
}

// A block per 4096 elements up to four times the default grid, a grid that loops above: it pays a block's set-up less
// often.  The line is where a looping grid began to win when a pass took half as long again.  (One-rank passes without a residual
// have a rule of their own, RoundtripGeneral.)  The default grid also serves blocks that meet at a flag or a counter (`shared`):
// each costs a system-scope fence or a look at the flags.
static int general_grid(int64_t groups, int group_size, int max_blocks, bool shared) {
    int64_t want = (groups * (group_size / kElemsPerThread) + kThreads - 1) / kThreads;
    if (want < 1) want = 1;
    int64_t cap = max_blocks;
    if (cap <= 0) cap = shared || want > 4 * lbc_default_max_blocks() ? lbc_default_max_blocks() : want;
    return int(want < cap ? want : cap);
}

// The thresholds of the rule "the last entry that is not above t, and the one after it when t - entry > gap / 2", searched on
// the bit patterns around the middle of two entries, and what the kernels make of them (see book_code and book_codes_far).
struct BookTable {
    LbcBook of[4];
    BookTable() {
        static const float tables[4][15] = LBC_CODEBOOKS;
        static const float nudges[4] = {0.0f, 0.0f, 2.3283064365386963e-10f, 1.862645149230957e-09f};      // 2^-32, 2^-29
        for (int q = 0; q < 4; ++q) {
            LbcBook& book = of[q];
            book.nudge = nudges[q];
            float least[14];                           // the least t whose code is above c
            for (int c = 0; c < 14; ++c) {
                const float a = tables[q][c], b = tables[q][c + 1];
                const auto above = [&](float t) {
                    if (t >= b) return true;
                    volatile float over = t - a, half = (b - a) * 0.5f;
                    return over > half;
                };
                float t = a + (b - a) * 0.5f;
                for (int i = 0; i < 64 && !above(t); ++i) t = std::nextafterf(t, 2.0f);
                for (int i = 0; i < 64 && above(std::nextafterf(t, -2.0f)); ++i) t = std::nextafterf(t, -2.0f);
                least[c] = t;
                book.thresholds[c] = -kThresholdScale * std::nextafterf(t, -2.0f);
            }
            const auto key = [&](float t) {            // as book_code forms it
                volatile float nudged = t - book.nudge;
                const float f = nudged;
                uint32_t bits;
                std::memcpy(&bits, &f, sizeof(bits));
                return bits << 1 | bits >> 31;
            };
            for (uint32_t i = 0; i < 32; ++i) {
                const uint32_t upper = (0x78000000u >> 22) + i;           // the bits of a key that name the bucket
                uint32_t below = 0u, inside = 0u;
                for (int c = 7; c < 14; ++c) {         // a threshold above zero and its mirror image
                    const uint32_t plus = key(least[c]), minus = key(std::nextafterf(least[13 - c], -2.0f));
                    const uint32_t at = plus < minus ? plus : minus;
                    if (at >> 22 < upper) ++below;
                    if (at >> 22 == upper) inside = (1u << 24) - ((at * 4u) & 0xffffffu);
                }
                book.steps[i] = (below << 24) - (upper << 24) + inside;
            }
        }
    }
};
static LbcBook book_of(int quant_type) {
    static const BookTable table;
    return quant_type == LBC_LINEAR ? LbcBook{} : table.of[quant_type - 1];
}

template <typename T, int TOPK, int KIND>
struct QuantGeneral {
    static constexpr bool noise = true;
    static void run(const LbcQuantGeneral& p, int grid, cudaStream_t s) {
        const uintptr_t at = reinterpret_cast<uintptr_t>(p.out);
        if (p.num_dst > 0 || p.signal.num_remote > 0)      // for other ranks, who wait for it
            quant_general_kernel<T, TOPK, KIND><<<grid, kThreads, 0, s>>>(p);
        else if (p.compact ? (at & 15) == 0 : (at & (Kind<KIND>::CB - 1)) == 0) {
            // Without a residual, in the kernels that know it, but where those are slower.  us with / without, encodes in a CUDA graph,
            // spread 0.2 %.  Code-books, 16 bits: up to half a default grid (bf16 e2m1 2 Mi elements 3.07 / 3.54, 3 Mi 4.61 / 4.37),
            // records that keep nothing up to a whole one (4 Mi 5.26 / 5.45, 5 Mi 6.54 / 5.98).  fp32 ones that keep nothing: outside a
            // quarter of one (1 Mi 2.34 / 2.53, 1.5 Mi 3.80 / 3.45) to a whole one (4 Mi 5.46 / 5.11, 5 Mi 5.88 / 6.04, 8 Mi 9.2 / 10.0).
            // Linear codes, 16 bits, planar, one kept value: many waves of full grids, where five blocks per SM hide more than the
            // residual's registers cost (bf16 8 Mi 7.95 / 8.00, fp16 7.80 / 7.62, bf16 12 Mi 12.7 / 13.0, 16 Mi 16.4 / 16.8); looping grids
            // have no waves (32 Mi 30.2 / 28.7).
            const int64_t tiles = (p.numel + kThreads * kElemsPerThread - 1) / (kThreads * kElemsPerThread);
            const int64_t full = lbc_default_max_blocks();
            bool plain = KIND != kBookNoise && p.residual == nullptr && p.prepared_out == nullptr;
            if (KIND == kBook && sizeof(T) == 2) plain = plain && tiles > (p.compact && TOPK == 0 ? full : full / 2);
            if (KIND == kBook && sizeof(T) == 4 && TOPK == 0) plain = plain && tiles > full / 4 && tiles <= full;
            if (KIND != kBook && sizeof(T) == 2 && TOPK == 1 && !p.compact) plain = plain && (tiles <= 2 * full || tiles > grid);
            const auto go = [&](auto prepare) {
                constexpr bool kPrepare = decltype(prepare)::value;
                if (p.compact) launch_chained(encode_general_kernel<T, TOPK, KIND, true, kPrepare>, unsigned(grid), s, p);
                else launch_chained(encode_general_kernel<T, TOPK, KIND, false, kPrepare>, unsigned(grid), s, p);
            };
            if constexpr (KIND != kBookNoise) {
                if (plain) {
                    go(std::false_type{});
                    return;
                }
            }
            go(std::true_type{});
        }
        else                    // a payload off its vectors
            launch_chained(quant_general_kernel<T, TOPK, KIND>, unsigned(grid), s, p);
    }
};
template <typename T, int TOPK, int KIND>
struct DequantGeneral {
    static constexpr bool noise = false;
    static void run(const LbcDequantGeneral& p, int grid, cudaStream_t s) {
        // Blocks per SM.  A decode waits for its loads: as many as the registers leave without the sum into `out` (64 MiB, 4 / 8,
        // bf16, one kept value 21.9 / 20.1, e2m1 19.4 / 17.1; fp32, 4 / 6, 16.6 / 15.2), but for 16-bit records with kept
        // values, whose words are read one by one (24.5 / 25.2), and fp32 up to two default grids, where six leave a short last
        // wave (16 MiB, e2m1, 5.58 / 5.89).
        const int64_t tiles = (p.numel + kThreads * kElemsPerThread - 1) / (kThreads * kElemsPerThread);
        // Five, above half a default grid and up to two: fp32 (four / five / six, e2m1, 2 Mi elements 2.94 / 3.18 / 3.45, 4 Mi
        // 4.41 / 4.11 / 4.12, 5 M 5.11 / 4.74 / 4.79), planar 16-bit payloads with kept values and linear codes (five / eight, bf16, one:
        // 2 Mi 2.57 / 2.50, 4 Mi 3.35 / 3.67, 8 Mi 5.97 / 6.14, 16 Mi 11.8 / 11.3), those in 4 bits up to one default grid (two:
        // 3 Mi 3.22 / 3.89, 4 Mi 3.86 / 3.96, 5 Mi 4.61 / 4.45, 8 Mi 6.84 / 6.43).
        const int64_t grid_tiles = lbc_default_max_blocks();
        const int64_t most = sizeof(T) == 2 && Kind<KIND>::bit == 4 ? grid_tiles : 2 * grid_tiles;
        const bool five = 2 * tiles > grid_tiles && tiles <= most &&
                          (sizeof(T) == 4 || (!p.compact && TOPK >= 1 && !Kind<KIND>::book));
        const bool many = sizeof(T) == 2 ? !(p.compact && TOPK >= 1) : tiles > 2 * grid_tiles;
        if (five && !p.accumulate)
            launch_chained(dequant_general_kernel<T, TOPK, KIND, false, 5>, unsigned(grid), s, p);
        else if (many && !p.accumulate)
            launch_chained(dequant_general_kernel<T, TOPK, KIND, false, sizeof(T) == 2 ? 8 : 6>, unsigned(grid), s, p);
        else
            launch_chained(dequant_general_kernel<T, TOPK, KIND, true, 4>, unsigned(grid), s, p);
    }
};
template <typename T, int TOPK, int KIND>
struct ReduceGeneral {
    static constexpr bool noise = false;
    static void run(const LbcReduceGeneral& p, int grid, cudaStream_t s) {
        reduce_general_kernel<T, TOPK, KIND><<<grid, kThreads, 0, s>>>(p);
    }
};
template <typename T, int TOPK, int KIND>
struct RoundtripGeneral {
    static constexpr bool noise = true;
    static void run(const LbcRoundtripGeneral& p, int grid, cudaStream_t s) {
        // No residual and one pass: kernels that know it (what the others hold for both costs registers).  Above one default
        // grid 16-bit tensors take as many blocks as are resident, each with its next tile under way: a tile per block /
        // resident blocks, bf16, one kept value, 4 Mi elements 3.62 / 3.83, 6 Mi 5.08 / 4.59, 16 Mi 14.5 / 12.0, 32 Mi 28.2 / 22.8
        // (without the next tile under way 25.4, with twice the blocks 23.1).  Books without kept values from half a grid on
        // (e2m1, 4 Mi 6.23 / 5.70, 32 Mi 37.1 / 30.0); below, the form without a residual does not pay for them.  fp32, full grids:
        // with a residual's registers / without, one kept value, 4 Mi 5.59 / 4.81, two, 16 Mi 24.2 / 21.2, e2m1 (five blocks per
        // SM) 26.7 / 23.1; looping gains nothing (16 Mi 20.9 / 22.3).
        const int64_t tiles = (p.numel + kThreads * kElemsPerThread - 1) / (kThreads * kElemsPerThread);
        const auto capped = [&](int64_t blocks) { return unsigned(p.max_blocks > 0 && p.max_blocks < blocks ? p.max_blocks : blocks); };
        if constexpr (KIND != kBookNoise) {
            // (tensors off 32 bytes keep the others: going round took 98 us instead of 86 for 16 Mi bf16 elements, one element in)
            if (p.residual == nullptr && p.passes == 1 && on_boundary(32, p.x, p.out)) {
                if constexpr (sizeof(T) == 2) {
                    constexpr bool book = KIND == kBook && TOPK == 0;
                    const int64_t resident = lbc_default_max_blocks() / 2;
                    if (tiles > (book ? resident : 2 * resident) || capped(tiles) < tiles)
                        launch_chained(roundtrip_plain_kernel<T, TOPK, KIND, 4, true>, capped(tiles < resident ? tiles : resident), s, p);
                    else if constexpr (book)
                        launch_chained(roundtrip_general_kernel<T, TOPK, KIND, 4>, unsigned(tiles), s, p);
                    else
                        launch_chained(roundtrip_plain_kernel<T, TOPK, KIND, 4, false>, unsigned(tiles), s, p);
                } else {
                    launch_chained(roundtrip_plain_kernel<T, TOPK, KIND, KIND == kBook && TOPK == 0 ? 5 : 4, false>, capped(tiles), s, p);
                }
                return;
            }
        }
        // fp32, three blocks per SM or four (64 registers, with spills).  Four are faster for two passes of one kept value without
        // a residual alone (two kept values, 16 Mi elements: 25.1 / 26.3), where three do not hold the whole grid.  Three / four
        // with a residual, one kept value, 8 bits: 1 Mi 3.75 / 5.12, 2 Mi 7.01 / 7.12, 16 Mi 40.5 / 41.4; e2m1 42.3 / 45.5, with
        // noise 107 / 116.
        if constexpr (sizeof(T) == 2) {
            launch_chained(roundtrip_general_kernel<T, TOPK, KIND, 4>, unsigned(grid), s, p);
        } else {
            if constexpr (TOPK == 1 && KIND != kBookNoise)
                if (p.residual == nullptr && grid > lbc_default_max_blocks() / 8 * 3) {
                    launch_chained(roundtrip_general_kernel<T, TOPK, KIND, 4>, unsigned(grid), s, p);
                    return;
                }
            launch_chained(roundtrip_general_kernel<T, TOPK, KIND, 3>, unsigned(grid), s, p);
        }
    }
};

template <template <typename, int, int> class Kernel, typename T, typename P>
static cudaError_t launch_typed(const P& p, int grid, cudaStream_t s) {
    constexpr bool noise = Kernel<T, 0, kBook>::noise;            // encodes
    const int kind = p.quant_type != LBC_LINEAR ? kBook : (p.bit == 8 ? kLinear8 : kLinear4);
    if constexpr (noise)
        if (kind == kBook && p.stochastic) {
            if (p.topk == 0) Kernel<T, 0, kBookNoise>::run(p, grid, s);
            else if (p.topk == 1) Kernel<T, 1, kBookNoise>::run(p, grid, s);
            else Kernel<T, 2, kBookNoise>::run(p, grid, s);
            return cudaGetLastError();
        }
#define LBC_CASE(KK, DD) if (p.topk == KK && kind == DD) Kernel<T, KK, DD>::run(p, grid, s); else
    LBC_CASE(0, kLinear8) LBC_CASE(1, kLinear8) LBC_CASE(2, kLinear8)
    LBC_CASE(0, kLinear4) LBC_CASE(1, kLinear4) LBC_CASE(2, kLinear4)
    LBC_CASE(0, kBook) LBC_CASE(1, kBook) LBC_CASE(2, kBook)
    return cudaErrorInvalidValue;
#undef LBC_CASE
    return cudaGetLastError();
}

template <template <typename, int, int> class Kernel, typename P>
static cudaError_t launch_general(const P& p, int max_blocks, bool shared, cudaStream_t s) {
    if (p.numel == 0) return cudaSuccess;
    if (p.group_size != 64 && p.group_size != 32 && p.group_size != 16) return cudaErrorInvalidValue;
    const int grid = general_grid((p.numel + p.group_size - 1) / p.group_size, p.group_size, max_blocks, shared);
    switch (p.dtype) {
        case LBC_BF16: return launch_typed<Kernel, __nv_bfloat16>(p, grid, s);
        case LBC_FP16: return launch_typed<Kernel, __half>(p, grid, s);
        case LBC_FP32: return launch_typed<Kernel, float>(p, grid, s);
        default: return cudaErrorInvalidValue;
    }
}

static bool general_args_ok(int bit, int topk, int quant_type) {
    if (bit != 4 && bit != 8) return false;
    if (topk < 0 || topk > 2) return false;
    if (quant_type < LBC_LINEAR || quant_type > LBC_E2M1) return false;
    if (quant_type != LBC_LINEAR && bit != 4) return false;
    return true;
}

}  // namespace lbc

extern "C" {

cudaError_t lbc_quant_general(const LbcQuantGeneral* p, cudaStream_t stream) {
    if (p == nullptr || p->numel < 0 || !lbc::general_args_ok(p->bit, p->topk, p->quant_type)) return cudaErrorInvalidValue;
    if (p->num_dst < 0 || p->num_dst > LBC_MAX_RANKS || (p->num_dst == 0 && p->out == nullptr)) return cudaErrorInvalidValue;
    if (p->shard_groups < 0) return cudaErrorInvalidValue;
    if (p->shard_groups > 0 && p->num_dst > 0) {      // every group must have an owner among the destinations
        const int64_t groups = (p->numel + p->group_size - 1) / p->group_size;
        if (groups > p->shard_groups * p->num_dst) return cudaErrorInvalidValue;
    }
    for (int d = 0; d < p->num_dst; ++d)
        if (p->dst[d] == nullptr) return cudaErrorInvalidValue;
    LbcQuantGeneral launch = *p;
    launch.book = lbc::book_of(p->quant_type);
    return lbc::launch_general<lbc::QuantGeneral>(launch, p->max_blocks, p->signal.num_remote > 0, stream);
}

cudaError_t lbc_dequant_general(const LbcDequantGeneral* p, cudaStream_t stream) {
    if (p == nullptr || p->numel < 0 || !lbc::general_args_ok(p->bit, p->topk, p->quant_type)) return cudaErrorInvalidValue;
    return lbc::launch_general<lbc::DequantGeneral>(*p, 0, false, stream);
}

cudaError_t lbc_reduce_general(const LbcReduceGeneral* p, cudaStream_t stream) {
    if (p == nullptr || p->numel < 0 || !lbc::general_args_ok(p->bit, p->topk, p->quant_type)) return cudaErrorInvalidValue;
    if (p->num_src < 1 || p->num_src > LBC_MAX_RANKS || p->out == nullptr) return cudaErrorInvalidValue;
    if ((p->prepared == nullptr) != (p->residual_out == nullptr)) return cudaErrorInvalidValue;
    if (p->layout_groups < 0 || p->src_shard_groups < 0) return cudaErrorInvalidValue;
    {
        const int64_t groups = (p->numel + p->group_size - 1) / p->group_size;
        if (p->src_shard_groups > 0 && groups > p->src_shard_groups * p->num_src) return cudaErrorInvalidValue;
        if (p->src_shard_groups == 0 && p->layout_groups > 0 && groups > p->layout_groups) return cudaErrorInvalidValue;
    }
    for (int r = 0; r < p->num_src; ++r)
        if (p->src[r] == nullptr) return cudaErrorInvalidValue;
    return lbc::launch_general<lbc::ReduceGeneral>(*p, p->max_blocks, p->wait.flags != nullptr, stream);
}

cudaError_t lbc_roundtrip_general(const LbcRoundtripGeneral* p, cudaStream_t stream) {
    if (p == nullptr || p->numel < 0 || !lbc::general_args_ok(p->bit, p->topk, p->quant_type)) return cudaErrorInvalidValue;
    if (p->passes < 1 || p->passes > 2 || (p->residual == nullptr && p->residual_out != nullptr)) return cudaErrorInvalidValue;
    if (p->numel > 0 && (p->x == nullptr || p->out == nullptr)) return cudaErrorInvalidValue;
    LbcRoundtripGeneral launch = *p;
    launch.book = lbc::book_of(p->quant_type);
    return lbc::launch_general<lbc::RoundtripGeneral>(launch, p->max_blocks, false, stream);
}

}  // extern "C"
