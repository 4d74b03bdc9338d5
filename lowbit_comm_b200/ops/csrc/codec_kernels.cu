// The codec on its own (encode a tensor, decode a payload, reduce the payloads a rank has gathered) for the production
// profiles: linear, no top-k, nearest-even rounding.  One payload in or out lies in this GPU's memory, nobody waits and
// nobody is signalled; what the collectives add to that (peer destinations, flags, shards) is in fast_kernels.cu.
//
// Math is identical, bit for bit, to quant_push_kernel / reduce_kernel there.
// Reference: quantization/quant_pack_kernel.cu:84-163, quantization/dequant_reduce_kernel.cu:38-69, 150-221.
//
// What bounds these kernels: memory.  A block per tile (a persistent grid moved 10-15 % less; the loops over tiles serve
// grids that a caller caps), 32 bytes of input per thread in one load, payloads read and written as 16-byte vectors in
// both layouts, the whole-tile path free of bounds and alignment tests (their registers cost occupancy); tensors and
// payloads off those boundaries have kernels of their own.
// Measured on a B200 through the public calls, passes repeated for a second, int8 groups of 64, the grid-stride kernels
// of fast_kernels.cu and now: encode of 32 Mi bf16 elements with error feedback 47.0 -> 36.0 us (6.6 TB/s), decode of
// 128 Mi 94 -> 61.5 (6.6 TB/s), mean of eight payloads of 32 Mi with error feedback 107 -> 76.4 (6.3 TB/s): that one
// draws the card's 1000 W, and its clock falls to 1.7 GHz.  Below, us in CUDA graphs.
#include <type_traits>

#include "codec_device.cuh"
#include "common.cuh"
#include "lbc_api.h"

namespace lbc {

// ---------------------------------------------------------------------------
// encode
// ---------------------------------------------------------------------------
// Quantizes and stores the thread's 16 values (`held`: the same in T).  Convergent (the group maximum shuffles); `span` is the
// warp's staging area for compact records.  kPrepared: `held` came out of a sum.  kOwnError: this rank's quantization error may be
// asked for (local_ef_out).
template <typename T, int G, int BIT, bool kCompact, bool kPrepared, bool kOwnError, int kFit>
__device__ __forceinline__ void encode_chunk(const LbcQuantPush& p, const Raw16<T>& held, float (&v)[16], int64_t chunk,
                                             uint8_t* span) {
    constexpr int lanes = G / kElemsPerThread;
    constexpr int VB = G * BIT / 8, MB = sizeof(T), CB = kElemsPerThread * BIT / 8;
    T* prep = static_cast<T*>(p.prepared_out);
    T* const lef = kOwnError ? static_cast<T*>(p.local_ef_out) : nullptr;
    uint8_t* dst = p.dst[0];
    const int64_t num_groups = (p.numel + G - 1) / G;
    const int64_t first = chunk * kElemsPerThread;
    const bool live = kFit == kFitWhole || chunk < num_groups * lanes;
    const int64_t g = chunk / lanes;
    const int lane = int(chunk) & (lanes - 1);
    const int wlane = threadIdx.x & 31;
    float stored = group_top<T, G>(held);                         // exact in T, like the values
    if (prep != nullptr && live) {
        if constexpr (kPrepared && kFit == kFitWhole) {
#pragma unroll
            for (int h = 0; h < int(sizeof(T)) / 2; ++h) st32(prep + first + 16 / (sizeof(T) / 2) * h, held.part[h]);
        } else {
            store16_fit<T, kFit>(prep, first, p.numel, v);
        }
    }
    float err[16];
    uint4 codes;
    if (scales_near(stored)) {
        codes = encode16_near<T, BIT>(v, stored, lef != nullptr ? &err : nullptr);
    } else {
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
        stored = group_max<G>(amax);
        codes = encode16<T, BIT>(v, stored, lef != nullptr ? &err : nullptr);
    }
    if (lef != nullptr && live) store16_fit<T, kFit>(lef, first, p.numel, err);
    if (kCompact && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        uint8_t* rec = span + (wlane / lanes) * (VB + MB);
        const uint32_t w[4] = {codes.x, codes.y, codes.z, codes.w};
        span_put_codes<CB>(rec + lane * CB, w);
        if (lane == 0) store_scale<T>(rec + VB, stored);
        __syncwarp();
        const int64_t g0 = (chunk - wlane) / lanes;
        const int64_t groups = min(int64_t(32 / lanes), num_groups - g0);
        if (groups > 0) span_to_global(dst + g0 * (VB + MB), span, int(groups) * (VB + MB), wlane);
        __syncwarp();
    } else if (live) {
        uint8_t* vptr = kCompact ? dst + g * (VB + MB) : dst + g * VB;
        store_codes(vptr + lane * CB, codes, CB);
        if (lane == 0) store_scale<T>(kCompact ? vptr + VB : dst + p.layout_groups * VB + g * MB, stored);
    }
}

// A tile with the tensor's end in it (kFitTail), or of unaligned tensors.
template <typename T, int G, int BIT, bool kCompact, bool kOwnError, int kFit>
__device__ __forceinline__ void encode_edge(const LbcQuantPush& p, int64_t c0, int chunks_per_thread, uint8_t* span) {
    const T* x = static_cast<const T*>(p.x);
    const T* res = static_cast<const T*>(p.residual);
    for (int j = 0; j < chunks_per_thread; ++j) {
        const int64_t chunk = c0 + j * kThreads + threadIdx.x;
        float v[16];
        load16_fit<T, kFit>(x, chunk * kElemsPerThread, p.numel, v);
        if (res != nullptr) {
            float r[16];
            load16_fit<T, kFit>(res, chunk * kElemsPerThread, p.numel, r);
            compensate16<T>(v, r);
        }
        encode_chunk<T, G, BIT, kCompact, false, kOwnError, kFit>(p, down16<T>(v), v, chunk, span);
    }
}

template <int G, int BIT, typename T>
constexpr int encode_span(bool compact) { return compact ? span_bytes(G, G * BIT / 8 + int(sizeof(T))) : 16; }

// All tensors on 32 bytes (the payload may start anywhere).  kOwnError: with local_ef_out, whose registers made the
// others spill.
// Blocks per SM: four leave a thread 64 registers, five 48.  Five where two 16-bit chunks are in flight (bf16, 4 / 5:
// 8 Mi elements 4.08 / 4.13, 16 Mi 9.50 / 9.10, 64 Mi 32.2 / 30.4) and for records, but for fp32 ones with a residual, whose
// 16 values and 16 residuals do not fit (without: bf16 16 Mi 13.3 / 12.0, fp32 14.8 / 13.8; bf16 with one, 19.5 / 18.6; fp32
// with one, 1.5 Mi 3.66 / 4.42, 16 Mi 33.3 / 33.4).  Four for the others (bf16, 1 Mi 1.44 / 1.47, with a residual
// 32 Mi 35.2 / 35.7; fp32, 2 Mi 1.95 / 2.22, with a residual 3.77 / 4.38).
template <typename T, bool kCompact, bool kResidual, int U>
constexpr int encode_kernel_blocks() {
    if (sizeof(T) == 4 && kResidual) return 4;
    return (sizeof(T) == 2 && U == 2) || (kCompact && U == 1) ? 5 : 4;
}
template <typename T, int G, int BIT, bool kCompact, bool kResidual, bool kOwnError, int U>
__global__ void __launch_bounds__(kThreads, kOwnError ? 4 : encode_kernel_blocks<T, kCompact, kResidual, U>())
encode_kernel(const __grid_constant__ LbcQuantPush p) {
    chain_wait();
    constexpr int lanes = G / kElemsPerThread;
    constexpr int tile_chunks = kThreads * U;
    const T* x = static_cast<const T*>(p.x);
    const T* res = static_cast<const T*>(p.residual);
    const int64_t chunks = (p.numel + G - 1) / G * lanes;
    __shared__ __align__(16) uint8_t spans[kThreads / 32][encode_span<G, BIT, T>(kCompact)];
    uint8_t* span = spans[threadIdx.x >> 5];
    for (int64_t c0 = int64_t(blockIdx.x) * tile_chunks; c0 < chunks; c0 += int64_t(gridDim.x) * tile_chunks) {
        if ((c0 + tile_chunks) * kElemsPerThread > p.numel) {
            encode_edge<T, G, BIT, kCompact, kOwnError, kFitTail>(p, c0, U, span);
            continue;
        }
        const int64_t mine = c0 + threadIdx.x;
        Raw16<T> rx[U], rr[kResidual ? U : 1];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            rx[j] = raw16(x + (mine + j * kThreads) * kElemsPerThread);
            if (kResidual) rr[j] = raw16(res + (mine + j * kThreads) * kElemsPerThread);
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
            float v[16];
            up16<T>(rx[j], v);
            if (kResidual) {
                float r[16];
                up16<T>(rr[j], r);
                rx[j] = compensate16<T>(v, r);
            }
            encode_chunk<T, G, BIT, kCompact, kResidual, kOwnError, kFitWhole>(p, rx[j], v, mine + j * kThreads, span);
        }
    }
}

// A tensor on another boundary (a view into a larger one), in a kernel of its own: as a branch of encode_kernel this ran
// out of line, element by element.  16 Mi elements, the input one element in, with error feedback (grid-stride kernel of
// fast_kernels.cu / that branch / here): bf16 45.8 / 41.1 / 27.1 us, fp32 45.6 / 61.7 / 43.5.  Blocks per SM, fp32, 4 / 3:
// 46.3 / 43.1 us.  kOwnError: with local_ef_out, where the launcher finds this kernel faster for aligned tensors too; and all of fp32
// on another boundary, because without it four blocks fit an SM (4 Mi elements 11.5 -> 12.6 us, 16 Mi 40.9 -> 41.0).  Measured before and
// with encode16_near: bf16 4 Mi 6.96 -> 6.38, 16 Mi 24.2 -> 22.6.
template <typename T, int G, int BIT, bool kCompact, bool kOwnError>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 4 ? 3 : 4) encode_ragged_kernel(const __grid_constant__ LbcQuantPush p) {
    chain_wait();
    const int64_t chunks = (p.numel + G - 1) / G * (G / kElemsPerThread);
    __shared__ __align__(16) uint8_t spans[kThreads / 32][encode_span<G, BIT, T>(kCompact)];
    for (int64_t c0 = int64_t(blockIdx.x) * kThreads; c0 < chunks; c0 += int64_t(gridDim.x) * kThreads)
        encode_edge<T, G, BIT, kCompact, kOwnError, kFitRagged>(p, c0, 1, spans[threadIdx.x >> 5]);
}

template <typename T, int G, int BIT>
struct EncodeLauncher {
    static cudaError_t run(const LbcQuantPush* p, cudaStream_t stream) {
        const int64_t chunks = (p->numel + G - 1) / G * (G / kElemsPerThread);
        if (chunks == 0) return cudaSuccess;
        const int64_t one = (chunks + kThreads - 1) / kThreads;
        auto grid = [&](int64_t blocks) {
            const int64_t cap = p->max_blocks > 0 ? p->max_blocks : int64_t(1) << 30;
            return unsigned(blocks < cap ? blocks : cap);
        };
        const auto go = [&](auto compact) {
            constexpr bool kCompact = decltype(compact)::value;
            const bool ragged = !on_boundary(32, p->x, p->residual, p->prepared_out);
            // Aligned tensors with local_ef_out, encode_kernel / encode_ragged_kernel: bf16, 3 Mi elements 4.95 / 4.35, 4 Mi
            // 6.54 / 5.80, 5 Mi (above one default grid) 8.08 / 8.96, 16 Mi 21.5 / 23.5, records 4 Mi 6.38 / 6.05, 5 Mi 8.41 / 9.46;
            // fp32 always the second: 1 Mi 2.92 / 3.10 (groups of 16: 3.25 / 2.99), 4 Mi 9.54 / 9.60, 32 Mi 64.0 / 64.0.
            if constexpr (sizeof(T) == 2) {
                if (p->local_ef_out != nullptr && p->residual != nullptr && !ragged && on_boundary(32, p->local_ef_out) &&
                    one > lbc_default_max_blocks()) {
                    launch_chained(encode_kernel<T, G, BIT, kCompact, true, true, 1>, grid(one), stream, *p);
                    return;
                }
            }
            if (p->local_ef_out != nullptr || (ragged && sizeof(T) == 4)) {
                launch_chained(encode_ragged_kernel<T, G, BIT, kCompact, true>, grid(one), stream, *p);
                return;
            }
            if (ragged) {
                if constexpr (sizeof(T) == 2)
                    launch_chained(encode_ragged_kernel<T, G, BIT, kCompact, false>, grid(one), stream, *p);
                return;
            }
            if (p->residual != nullptr) {
                launch_chained(encode_kernel<T, G, BIT, kCompact, true, false, 1>, grid(one), stream, *p);
                return;
            }
            // Two chunks per thread above one default grid (one / two: bf16 4 Mi elements 2.57 / 2.50, 8 Mi 4.88 / 4.08, 64 Mi 41.0 /
            // 30.4; fp32 4 Mi 2.94 / 2.84, 32 Mi 26.6 / 25.6), but for fp32 records, which gain nothing (16 Mi 13.8 / 14.1).
            if constexpr (sizeof(T) == 2 || !kCompact) {
                if (one > lbc_default_max_blocks()) {
                    launch_chained(encode_kernel<T, G, BIT, kCompact, false, false, 2>, grid((one + 1) / 2), stream, *p);
                    return;
                }
            }
            launch_chained(encode_kernel<T, G, BIT, kCompact, false, false, 1>, grid(one), stream, *p);
        };
        if (p->mode == LBC_PUSH_COMPACT_LOCAL)
            go(std::true_type{});
        else
            go(std::false_type{});
        return cudaGetLastError();
    }
};

// ---------------------------------------------------------------------------
// decode and reduce
// ---------------------------------------------------------------------------
// acc += one payload's 16 values: fma(code, scale / L, acc), one rounding per payload.  kPairs: two of them to an instruction
// (sm_100+) and the quotient without a branch; whole tiles.  Several payloads draw the card's power limit, so instructions
// are time: mean of eight of 32 Mi bf16 elements 86.5 -> 84.2 us, decode of 128 Mi 62.6 -> 61.6.  Unaligned tensors and
// tensor ends stay scalar: packed, the mean of eight of 16 Mi fp32 elements in records of 16, one payload on 8 bytes, took
// 64.4 us instead of 61.5.
template <typename T, int BIT, bool kPairs>
__device__ __forceinline__ void add_payload(float (&acc)[16], uint4 codes, float scale) {
    constexpr int lim = BIT == 8 ? 127 : 7;
    // The quotient comes ahead of the codes: after them, the sixteen decoded values lived across it, and the kernels of one payload
    // and of unaligned ones spilled (spill loads of the 36 and 72 instantiations, in sum: 10872 -> 5840 and 5388 -> 352 bytes;
    // 16 Mi bf16 elements, payload on 8 bytes 12.5 -> 9.5 us, mean of eight 54.9 -> 47.0; 4-bit decode of 128 Mi 61.5 -> 57.7).
    float step;
    if constexpr (kPairs) step = over_limit<lim>(scale);
    else step = scale / float(lim);
    float d[16];
    codes16<T, BIT>(codes, d);
    if constexpr (kPairs) {
#pragma unroll
        for (int i = 0; i < 16; i += 2)
            asm("{.reg .b64 a, b, c; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %4}; mov.b64 c, {%0, %1}; "
                "fma.rn.f32x2 c, a, b, c; mov.b64 {%0, %1}, c;}"
                : "+f"(acc[i]), "+f"(acc[i + 1]) : "f"(d[i]), "f"(d[i + 1]), "f"(step));
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = __fmaf_rn(d[i], step, acc[i]);
    }
}

// Adds payloads r0 .. r0 + K - 1 to a thread's chunk; all K loads are issued before the first is decoded.  Whole warps
// of whole groups, vector-aligned payloads.  Compact: the warp's span comes in as vectors and turns through `span`.
template <typename T, int G, int BIT, bool kCompact, int K>
__device__ __forceinline__ void add_batch(const LbcReduce& p, int r0, int64_t chunk, uint8_t* span, float (&acc)[16]) {
    constexpr int lanes = G / kElemsPerThread;
    constexpr int VB = G * BIT / 8, MB = sizeof(T), CB = kElemsPerThread * BIT / 8;
    const int lane = int(chunk) & (lanes - 1);
    const int64_t g = chunk / lanes;
    if constexpr (!kCompact) {
        uint4 codes[K];
        float scale[K];
        const int64_t voff = g * VB + lane * CB, soff = p.layout_groups * VB + g * MB;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const uint8_t* src = p.src[r0 + j];
            if constexpr (CB == 16) {
                codes[j] = ld16_once(src + voff);
            } else {
                const uint2 c = *reinterpret_cast<const uint2*>(src + voff);
                codes[j] = make_uint4(c.x, c.y, 0u, 0u);
            }
            scale[j] = load_scale<T>(src + soff);
        }
#pragma unroll
        for (int j = 0; j < K; ++j) add_payload<T, BIT, true>(acc, codes[j], scale[j]);
    } else {
        constexpr int full = span_bytes(G, VB + MB);            // 17 to 40 vectors
        const int wlane = threadIdx.x & 31;
        const int64_t at = (chunk - wlane) / lanes * (VB + MB) + wlane * 16;
        uint4 lo[K], hi[K];
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const uint8_t* src = p.src[r0 + j] + at;
            if (full >= 512 || wlane * 16 < full) lo[j] = ld16_once(src);
            if (full > 512 && wlane * 16 < full - 512) hi[j] = ld16_once(src + 512);
        }
        const uint8_t* rec = span + (wlane / lanes) * (VB + MB);
#pragma unroll
        for (int j = 0; j < K; ++j) {
            if (full >= 512 || wlane * 16 < full) *reinterpret_cast<uint4*>(span + wlane * 16) = lo[j];
            if (full > 512 && wlane * 16 < full - 512) *reinterpret_cast<uint4*>(span + wlane * 16 + 512) = hi[j];
            __syncwarp();
            uint32_t w[4];
            span_get_codes<CB>(rec + lane * CB, w);
            const float scale = load_scale<T>(rec + VB);
            __syncwarp();
            add_payload<T, BIT, true>(acc, make_uint4(w[0], w[1], w[2], w[3]), scale);
        }
    }
}

// A chunk with the tensor's end in its tile (kFitTail), or of tensors or payloads on any boundary.
template <typename T, int G, int BIT, bool kCompact, int kFit>
__device__ __forceinline__ void decode_edge(const LbcReduce& p, int64_t chunk) {
    constexpr int lanes = G / kElemsPerThread;
    constexpr int VB = G * BIT / 8, MB = sizeof(T), CB = kElemsPerThread * BIT / 8;
    if (chunk >= (p.numel + G - 1) / G * lanes) return;
    T* out = static_cast<T*>(p.out);
    T* rout = static_cast<T*>(p.residual_out);
    const T* prep = static_cast<const T*>(p.prepared);
    const int64_t first = chunk * kElemsPerThread, g = chunk / lanes;
    const int lane = int(chunk) & (lanes - 1);
    const int64_t voff = (kCompact ? g * (VB + MB) : g * VB) + lane * CB;
    const int64_t soff = kCompact ? g * (VB + MB) + VB : p.layout_groups * VB + g * MB;
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.0f;
#pragma unroll 2
    for (int r = 0; r < p.num_src; ++r)
        add_payload<T, BIT, false>(acc, load_codes(p.src[r] + voff, CB), load_scale<T>(p.src[r] + soff));
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] *= p.scale;
    if (rout != nullptr) {
        float e[16];
        load16_fit<T, kFit>(prep, first, p.numel, e);
#pragma unroll
        for (int i = 0; i < 16; ++i) e[i] -= acc[i];
        store16_fit<T, kFit>(rout, first, p.numel, e);
    }
    if (p.accumulate) {
        float prev[16];
        load16_fit<T, kFit>(static_cast<const T*>(out), first, p.numel, prev);
        round16<T>(acc);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] += prev[i];
    }
    store16_fit<T, kFit>(out, first, p.numel, acc);             // rounds to T
}

// Tensors on 32 bytes, payloads on their vectors.  B == 1: one payload without error feedback that is added to the
// output (`accumulate`), and some fp32 records in 4 bits.  B == 2: fp32 records with error feedback, two payloads in
// flight per thread.  decode_one_kernel and decode_several_kernel have the others.
// Blocks per SM as where this kernel did all of them: a decode of 128 Mi bf16 elements with 8 / 6 / 5 / 4 blocks 66 / 71 /
// 76 / 84; records, mean of eight, two in flight, with 5 / 4 / 3 blocks 105 / 101 / 113.
template <typename T, int G, int BIT, bool kCompact, int B>
__global__ void __launch_bounds__(kThreads, B == 1 ? (sizeof(T) == 2 ? 8 : 6) : (kCompact || sizeof(T) == 4 ? 4 : 5))
decode_kernel(const __grid_constant__ LbcReduce p) {
    chain_wait();
    constexpr int lanes = G / kElemsPerThread;
    constexpr int VB = G * BIT / 8, MB = sizeof(T);
    T* out = static_cast<T*>(p.out);
    const T* prep = static_cast<const T*>(p.prepared);
    T* rout = static_cast<T*>(p.residual_out);
    const int64_t chunks = (p.numel + G - 1) / G * lanes;
    const int R = B == 1 ? 1 : p.num_src;
    __shared__ __align__(16) uint8_t spans[kThreads / 32][kCompact ? span_bytes(G, VB + MB) : 16];
    uint8_t* span = spans[threadIdx.x >> 5];

    for (int64_t c0 = int64_t(blockIdx.x) * kThreads; c0 < chunks; c0 += int64_t(gridDim.x) * kThreads) {
        const int64_t chunk = c0 + threadIdx.x;
        if ((c0 + kThreads) * kElemsPerThread > p.numel) {
            decode_edge<T, G, BIT, kCompact, kFitTail>(p, chunk);
            continue;
        }
        const int64_t first = chunk * kElemsPerThread;
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.0f;
        Raw16<T> held;
        if (B > 1 && rout != nullptr) held = raw16(prep + first);      // on its way while the payloads are summed
        int r = 0;
        for (; r + B <= R; r += B) add_batch<T, G, BIT, kCompact, B>(p, r, chunk, span, acc);
        if constexpr (B > 2)
            for (; r + 2 <= R; r += 2) add_batch<T, G, BIT, kCompact, 2>(p, r, chunk, span, acc);
        if constexpr (B > 1)
            for (; r < R; ++r) add_batch<T, G, BIT, kCompact, 1>(p, r, chunk, span, acc);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] *= p.scale;
        if (B > 1 && rout != nullptr) {
            float e[16];
            up16<T>(held, e);
#pragma unroll
            for (int i = 0; i < 16; ++i) e[i] -= acc[i];
            store16<T>(rout + first, 0, 16, true, e);
        }
        if (p.accumulate) {
            float prev[16];
            up16<T>(raw16(static_cast<const T*>(out) + first), prev);
            round16<T>(acc);
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] += prev[i];
        }
        store16<T>(out + first, 0, 16, true, acc);                     // rounds to T
    }
}

// Several payloads, or one with error feedback, not added to the output: the reduction of gathered payloads, without the
// registers of the rest, which made it spill at five blocks per SM.  B payloads are in flight per thread.
// With error feedback four blocks per SM (mean of eight of 32 Mi bf16 elements, decode_kernel / five / four / six 79.7 /
// 76.1 / 72.8 / 76.2; eight of 2 Mi fp32 7.36 / 9.66 / 7.25 / 11.0), four in flight (two of 32 Mi bf16, two / four / eight
// 43.0 / 41.3 / 41.2; four of 4 Mi 8.42 / 6.85 / 7.45).  Without, five for 16 bits: two of 16 Mi 11.1 / 10.6.
template <typename T, int G, int BIT, bool kCompact, int B, bool kFeedback>
__global__ void __launch_bounds__(kThreads, kFeedback || kCompact || sizeof(T) == 4 ? 4 : 5)
decode_several_kernel(const __grid_constant__ LbcReduce p) {
    chain_wait();
    constexpr int lanes = G / kElemsPerThread;
    constexpr int VB = G * BIT / 8, MB = sizeof(T);
    T* out = static_cast<T*>(p.out);
    const T* prep = static_cast<const T*>(p.prepared);
    T* rout = static_cast<T*>(p.residual_out);
    const int64_t chunks = (p.numel + G - 1) / G * lanes;
    const int R = p.num_src;
    __shared__ __align__(16) uint8_t spans[kThreads / 32][kCompact ? span_bytes(G, VB + MB) : 16];
    uint8_t* span = spans[threadIdx.x >> 5];
    for (int64_t c0 = int64_t(blockIdx.x) * kThreads; c0 < chunks; c0 += int64_t(gridDim.x) * kThreads) {
        const int64_t chunk = c0 + threadIdx.x;
        if ((c0 + kThreads) * kElemsPerThread > p.numel) {
            decode_edge<T, G, BIT, kCompact, kFitTail>(p, chunk);
            continue;
        }
        const int64_t first = chunk * kElemsPerThread;
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.0f;
        Raw16<T> held;
        if (kFeedback) held = raw16(prep + first);                     // on its way while the payloads are summed
        int r = 0;
        for (; r + B <= R; r += B) add_batch<T, G, BIT, kCompact, B>(p, r, chunk, span, acc);
        if constexpr (B > 2)
            for (; r + 2 <= R; r += 2) add_batch<T, G, BIT, kCompact, 2>(p, r, chunk, span, acc);
        for (; r < R; ++r) add_batch<T, G, BIT, kCompact, 1>(p, r, chunk, span, acc);
        fma16(acc, p.scale, -0.0f);                                    // the product, with its sign where it is zero
        if (kFeedback) {
            float e[16];
            up16<T>(held, e);
#pragma unroll
            for (int i = 0; i < 16; ++i) e[i] -= acc[i];
            store16<T>(rout + first, 0, 16, true, e);
        }
        store16<T>(out + first, 0, 16, true, acc);                     // rounds to T
    }
}

// One payload, written as it is (no scale, nothing added to): what a decode mostly is, without the registers of the rest.
// U chunks per thread are loaded before the first is decoded.
// Small grids want five blocks per SM (48 registers), large ones eight, and planar payloads two chunks: one chunk with
// 5 / 8 blocks / two with 8, bf16 2 Mi elements 1.96 / 2.06 / 2.05, 4 Mi 2.53 / 2.56 / 3.10, 8 Mi 4.22 / 3.93 / 3.88,
// 128 Mi 70.8 / 60.9 / 61.2, in 4 bits 65.2 / 54.2 / 52.1; records 32 Mi 19.5 / 18.1 / 18.5; fp32 4 Mi 3.65 / 3.79 / 3.76,
// 16 Mi 14.4 / 13.7 / 12.8.
template <typename T, int G, int BIT, bool kCompact, int U, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) decode_one_kernel(const __grid_constant__ LbcReduce p) {
    chain_wait();
    constexpr int lanes = G / kElemsPerThread, lim = BIT == 8 ? 127 : 7;
    constexpr int VB = G * BIT / 8, MB = sizeof(T), CB = kElemsPerThread * BIT / 8;
    constexpr int tile_chunks = kThreads * U;
    T* out = static_cast<T*>(p.out);
    const uint8_t* src = p.src[0];
    const int64_t chunks = (p.numel + G - 1) / G * lanes;
    __shared__ __align__(16) uint8_t spans[kThreads / 32][kCompact ? span_bytes(G, VB + MB) : 16];
    uint8_t* span = spans[threadIdx.x >> 5];
    for (int64_t c0 = int64_t(blockIdx.x) * tile_chunks; c0 < chunks; c0 += int64_t(gridDim.x) * tile_chunks) {
        const int64_t mine = c0 + threadIdx.x;
        if ((c0 + tile_chunks) * kElemsPerThread > p.numel) {
            for (int j = 0; j < U; ++j) decode_edge<T, G, BIT, kCompact, kFitTail>(p, mine + j * kThreads);
            continue;
        }
        if constexpr (kCompact) {
#pragma unroll
            for (int j = 0; j < U; ++j) {
                float d[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) d[i] = 0.0f;
                add_batch<T, G, BIT, kCompact, 1>(p, 0, mine + j * kThreads, span, d);
                store16<T>(out + (mine + j * kThreads) * kElemsPerThread, 0, 16, true, d);
            }
        } else {
            uint4 codes[U];
            float scale[U];
#pragma unroll
            for (int j = 0; j < U; ++j) {
                const int64_t chunk = mine + j * kThreads;
                if constexpr (CB == 16) {
                    codes[j] = ld16_once(src + chunk * CB);
                } else {
                    const uint2 c = *reinterpret_cast<const uint2*>(src + chunk * CB);
                    codes[j] = make_uint4(c.x, c.y, 0u, 0u);
                }
                scale[j] = load_scale<T>(src + p.layout_groups * VB + chunk / lanes * MB);
            }
#pragma unroll
            for (int j = 0; j < U; ++j) {
                const float step = over_limit<lim>(scale[j]);      // ahead of the codes, as in add_payload
                float d[16];
                codes16<T, BIT>(codes[j], d);
                fma16(d, step, 0.0f);
                store16<T>(out + (mine + j * kThreads) * kElemsPerThread, 0, 16, true, d);
            }
        }
    }
}

// A tensor or a payload on another boundary (a view into a larger one; a row of a gather buffer whose payloads are no
// multiple of 16 bytes).  kSeveral: more than one payload, or error feedback.
// Blocks per SM, 16 Mi bf16 elements, planar 8-bit payloads of which one starts on 4 bytes, inputs beyond L2, 4 / 5 / 6
// blocks: one payload 17.6 / 16.5 / 18.5 us, mean of two with error feedback 35.2 / 32.9 / 28.8, of eight 73.8 / 67.8 /
// 61.6; 8-bit records, mean of eight 82.6 / 76.2 / 84.9.
// As a branch of decode_kernel this ran out of line, element by element.  16 Mi bf16 elements, buffers in L2 (grid-stride
// kernel of fast_kernels.cu / that branch / here): a payload on 8 bytes 14.8 / 18.8 / 9.6 us, an output one element in
// 99.7 / 107.7 / 35.8.
template <typename T, int G, int BIT, bool kCompact, bool kSeveral>
__global__ void __launch_bounds__(kThreads, kSeveral && !(kCompact && BIT == 8 && sizeof(T) == 2) ? 6 : 5)
decode_ragged_kernel(const __grid_constant__ LbcReduce p) {
    chain_wait();
    const int64_t chunks = (p.numel + G - 1) / G * (G / kElemsPerThread);
    for (int64_t c0 = int64_t(blockIdx.x) * kThreads; c0 < chunks; c0 += int64_t(gridDim.x) * kThreads)
        decode_edge<T, G, BIT, kCompact, kFitRagged>(p, c0 + threadIdx.x);
}

template <typename T, int G, int BIT>
struct DecodeLauncher {
    static cudaError_t run(const LbcReduce* p, cudaStream_t stream) {
        const int64_t chunks = (p->numel + G - 1) / G * (G / kElemsPerThread);
        if (chunks == 0) return cudaSuccess;
        const int64_t blocks = (chunks + kThreads - 1) / kThreads;
        const unsigned grid = unsigned(p->max_blocks > 0 && blocks > p->max_blocks ? p->max_blocks : blocks);
        const auto go = [&](auto compact) {
            constexpr bool kCompact = decltype(compact)::value;
            bool vectors = on_boundary(32, p->out, p->prepared, p->residual_out);
            for (int r = 0; r < p->num_src; ++r)
                vectors = vectors && on_boundary(kCompact ? 16 : kElemsPerThread * BIT / 8, p->src[r]);
            const bool alone = p->num_src == 1 && p->residual_out == nullptr;
            // (A sum of several, or one with error feedback, that is added to the output: no call of the library asks for it.
            // Eight of 16 Mi bf16 elements take 42.9 us there, 35.6 in a kernel of their own.)
            if (!vectors || (p->accumulate && !alone)) {
                if (alone)
                    launch_chained(decode_ragged_kernel<T, G, BIT, kCompact, false>, grid, stream, *p);
                else
                    launch_chained(decode_ragged_kernel<T, G, BIT, kCompact, true>, grid, stream, *p);
                return;
            }
            if (alone && p->scale == 1.0f && !p->accumulate) {
                // fp32 records in 4 bits from a block for every other SM up to three per SM, decode_kernel / decode_one_kernel:
                // 0.25 Mi elements 1.57 / 1.53, 0.5 Mi 1.69 / 1.78, 1 Mi 1.91 / 2.14, 1.5 Mi 2.17 / 2.56, 2 Mi 3.05 / 2.69; groups of
                // 16, 1 Mi, 2.07 / 2.04.  (Neither six blocks per SM nor the product with the scale bring decode_one_kernel
                // there; what does was not found.)
                if constexpr (kCompact && BIT == 4 && sizeof(T) == 4 && G > 16) {
                    const int64_t full = lbc_default_max_blocks();
                    if (blocks > full / 16 && blocks <= full / 8 * 3) {
                        launch_chained(decode_kernel<T, G, BIT, kCompact, 1>, grid, stream, *p);
                        return;
                    }
                }
                // Up to one default grid (bf16: 4 Mi small, 8 Mi large in the figures at the kernel)
                if (blocks <= lbc_default_max_blocks()) {
                    launch_chained(decode_one_kernel<T, G, BIT, kCompact, 1, 5>, grid, stream, *p);
                    return;
                }
                if constexpr (!kCompact) {
                    const int64_t pairs = (blocks + 1) / 2, cap = p->max_blocks > 0 ? p->max_blocks : pairs;
                    launch_chained(decode_one_kernel<T, G, BIT, kCompact, 2, 8>, unsigned(pairs < cap ? pairs : cap), stream, *p);
                } else {
                    launch_chained(decode_one_kernel<T, G, BIT, kCompact, 1, 8>, grid, stream, *p);
                }
                return;
            }
            // a compact payload takes two vectors per lane, so half as many are in flight
            if (p->accumulate)
                launch_chained(decode_kernel<T, G, BIT, kCompact, 1>, grid, stream, *p);
            else if (p->residual_out == nullptr)
                launch_chained(decode_several_kernel<T, G, BIT, kCompact, kCompact ? 2 : 4, false>, grid, stream, *p);
            else if constexpr (kCompact && sizeof(T) == 4)      // (16 Mi, this / the other, two 38.5 / 40.5, eight 61.6 / 69.7)
                launch_chained(decode_kernel<T, G, BIT, kCompact, 2>, grid, stream, *p);
            else
                launch_chained(decode_several_kernel<T, G, BIT, kCompact, kCompact ? 2 : 4, true>, grid, stream, *p);
        };
        if (p->compact)
            go(std::true_type{});
        else
            go(std::false_type{});
        return cudaGetLastError();
    }
};

}  // namespace lbc

extern "C" {

cudaError_t lbc_encode(const LbcQuantPush* p, cudaStream_t stream) {
    return lbc::dispatch_profile<lbc::EncodeLauncher>(p, stream);
}

cudaError_t lbc_decode(const LbcReduce* p, cudaStream_t stream) {
    return lbc::dispatch_profile<lbc::DecodeLauncher>(p, stream);
}

}  // extern "C"
