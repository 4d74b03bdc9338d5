// Collectives of a group of one rank (a one-GPU DDP job, the inter-node stage of a single node): the payload has no
// reader but its writer, so quantize and decode meet in registers and the payload never exists in memory.
//
// Math is identical, bit for bit, to the sequences of quant_push_kernel / reduce_kernel (fast_kernels.cu) and to the
// phases of pipe_allreduce_kernel (pipe_kernels.cu) on one rank:
//   prepared = T(x + residual), s = T(max |prepared|), q = clamp(rint(prepared * (L / max(s, 1e-6)))),
//   y32 = fma(q, s / L, 0), out = T(y32), residual = T(prepared - y32)          (passes == 1)
// and with passes == 2 (the two-stage all-reduce) T(y32) is quantized and decoded once more.
// Reference: quantization/quant_pack_kernel.cu:84-163, quantization/dequant_reduce_kernel.cu:38-69, 150-221.
//
// What bounds it: memory.  x is read and out written once (with error feedback the residual too), which is all that
// the result needs; the phases also wrote and read the payload, read the input's row twice and met at a grid-wide
// flag.  A block per tile and no loop over tiles: on a B200 a persistent grid of the same kernel moved 5.9 TB/s where
// the full grid moves 6.7-6.9, because the blocks of one wave end at different times and the next ones fill in.
// Measured through the public calls (bf16, int8 groups of 64): 512 Mi elements 919 -> 312 us (6.9 TB/s), 13.1 M elements
// 41.0 -> 10.2 us, 124 M elements in 7 buckets with error feedback 637 -> 186 us; then, each kernel started before the one ahead
// of it ends: 7.9 and 174-186 us.
// What stays in L2 (up to about 13 M elements) is bound by instruction issue instead: 11.5 instructions per element when every value was
// clamped and its maximum, product and sum took one each.  Now warps of finite groups take no clamp (scales_near), two elements to an
// instruction and quotients without branches, and two chunks per thread come in above one default grid.  In a CUDA graph, bf16: 1 Mi
// elements 1.92 -> 1.88 us, 4 Mi 3.18 -> 2.92, 13.1 M 7.77 -> 6.46 (8.1 TB/s), 33 Mi 22.7 -> 22.2; 13.1 M with a residual 17.8 -> 17.3;
// fp32 and what is beyond L2 stay within 1 %.
#include "codec_device.cuh"
#include "common.cuh"
#include "lbc_api.h"

namespace lbc {

// What a receiver of the codes of 16 rounded values decodes, in fp32 before the rounding to T; `p` are the same values in T.
// With `own_error` the values are replaced by this rank's quantization error, one rounding: fma(-code, step, value).
template <typename T, int G, int BIT>
__device__ __forceinline__ void roundtrip16(const Raw16<T>& p, float (&v)[16], float (&y)[16], bool own_error) {
    constexpr int lim = BIT == 8 ? 127 : 7;
    // the values are exact in T, so their largest magnitude is the stored scale without a rounding
    const float top = group_top<T, G>(p);
    if (scales_near(top)) {
        const float mul = limit_over<lim>(fmaxf(top, 1.0e-6f));
        const float step = over_limit<lim>(top);
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = v[i];
        fma16(y, mul, 0.0f);                                  // (+0 for -0, which the next sum hides anyway)
        add16(y, kRoundMagic);
        add16(y, -kRoundMagic);                               // the codes, exactly; +0 for code 0, as the decoder has it
        if (own_error) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __fmaf_rn(-y[i], step, v[i]);
        }
        fma16(y, step, 0.0f);
        return;
    }
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
    const float stored = group_max<G>(amax);
    const float mul = float(lim) / fmaxf(stored, 1.0e-6f);
    const float step = stored / float(lim);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        // the clamped sum is kRoundMagic + code exactly, and so is the difference
        const float code = __uint_as_float(quant_bits<lim>(v[i], mul)) - kRoundMagic;
        y[i] = __fmaf_rn(code, step, 0.0f);
        if (own_error) v[i] = __fmaf_rn(-code, step, v[i]);
    }
}

// From the prepared values (`held`: the same in T) to the outputs.  Convergent: the group maximum shuffles.
template <typename T, int G, int BIT, bool kResidual, int kFit>
__device__ __forceinline__ void roundtrip_chunk(const LbcRoundtrip& p, const Raw16<T>& held, float (&v)[16], int64_t first,
                                                bool live) {
    T* out = static_cast<T*>(p.out);
    T* rout = static_cast<T*>(p.residual_out);
    const bool own_error = kResidual && p.own_error != 0;
    float y[16];
    roundtrip16<T, G, BIT>(held, v, y, own_error);
    if (p.passes == 2) {
        const Raw16<T> again = down16<T>(y);
        float z[16];
        up16<T>(again, z);
        roundtrip16<T, G, BIT>(again, z, y, false);
    }
    if (!live) return;
    if (kResidual && rout != nullptr) {
        if (!own_error) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] -= y[i];
        }
        store16_fit<T, kFit>(rout, first, p.numel, v);
    }
    store16_fit<T, kFit>(out, first, p.numel, y);
}

// A chunk with the tensor's end in its tile (kFitTail), or of unaligned tensors.
template <typename T, int G, int BIT, bool kResidual, int kFit>
__device__ __forceinline__ void roundtrip_edge(const LbcRoundtrip& p, int64_t chunk, int64_t chunks) {
    const int64_t first = chunk * kElemsPerThread;
    float v[16];
    load16_fit<T, kFit>(static_cast<const T*>(p.x), first, p.numel, v);      // zeros past the end
    if (kResidual) {
        float r[16];
        load16_fit<T, kFit>(static_cast<const T*>(p.residual), first, p.numel, r);
        compensate16<T>(v, r);
    }
    roundtrip_chunk<T, G, BIT, kResidual, kFit>(p, down16<T>(v), v, first, chunk < chunks);
}

// Zeros behind the end of `out`, with the last tile (a shard is padded to 8 groups, so a padded one ends inside a tile).  As a fill of
// their own they took 7 us of the 23 that the call for the reduced shard of a ragged tensor cost.
template <typename T>
__device__ __forceinline__ void clear_pad(const LbcRoundtrip& p) {
    for (int i = threadIdx.x; i < p.pad; i += kThreads) static_cast<T*>(p.out)[p.numel + i] = T(0.0f);
}

// All tensors on 32 bytes.  kResidual: the input is T(x + residual).  U chunks of 16 elements per thread are loaded before
// the first is computed.
template <typename T, int G, int BIT, bool kResidual, int U>
__global__ void __launch_bounds__(kThreads) roundtrip_kernel(const LbcRoundtrip p) {
    chain_wait();
    constexpr int lanes = G / kElemsPerThread;
    constexpr int tile_chunks = kThreads * U;
    const T* x = static_cast<const T*>(p.x);
    const T* res = static_cast<const T*>(p.residual);
    const int64_t n = p.numel;
    const int64_t chunks = (n + G - 1) / G * lanes;

    for (int64_t c0 = int64_t(blockIdx.x) * tile_chunks; c0 < chunks; c0 += int64_t(gridDim.x) * tile_chunks) {
        const int64_t mine = (c0 + threadIdx.x) * kElemsPerThread;
        if ((c0 + tile_chunks) * kElemsPerThread <= n) {              // a whole tile
            Raw16<T> rx[U], rr[kResidual ? U : 1];
#pragma unroll
            for (int j = 0; j < U; ++j) {
                rx[j] = raw16(x + mine + j * (kThreads * kElemsPerThread));
                if (kResidual) rr[j] = raw16(res + mine + j * (kThreads * kElemsPerThread));
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
                roundtrip_chunk<T, G, BIT, kResidual, kFitWhole>(p, rx[j], v, mine + j * (kThreads * kElemsPerThread), true);
            }
        } else {
            for (int j = 0; j < U; ++j)
                roundtrip_edge<T, G, BIT, kResidual, kFitTail>(p, c0 + threadIdx.x + j * kThreads, chunks);
            clear_pad<T>(p);
        }
    }
}

// A tensor on another boundary (a view into a larger one), in a kernel of its own: as a branch of roundtrip_kernel this ran
// out of line, element by element, on all four tensors.  16 Mi elements with error feedback through the public call, the
// input one element in (phases / that branch / here): bf16 176.7 / 182.0 / 42.6 us, fp32 156.4 / 190.9 / 95.0.
template <typename T, int G, int BIT, bool kResidual>
__global__ void __launch_bounds__(kThreads) roundtrip_ragged_kernel(const LbcRoundtrip p) {
    chain_wait();
    const int64_t chunks = (p.numel + G - 1) / G * (G / kElemsPerThread);
    for (int64_t c0 = int64_t(blockIdx.x) * kThreads; c0 < chunks; c0 += int64_t(gridDim.x) * kThreads) {
        roundtrip_edge<T, G, BIT, kResidual, kFitRagged>(p, c0 + threadIdx.x, chunks);
        if (c0 + kThreads >= chunks) clear_pad<T>(p);
    }
}

template <typename T, int G, int BIT>
struct RoundtripLauncher {
    static cudaError_t run(const LbcRoundtrip* p, cudaStream_t stream) {
        const int64_t chunks = (p->numel + G - 1) / G * (G / kElemsPerThread);
        const int64_t one = (chunks + kThreads - 1) / kThreads;           // blocks of one chunk per thread
        auto grid = [&](int64_t blocks) {
            const int64_t cap = p->max_blocks > 0 ? p->max_blocks : int64_t(1) << 30;
            return unsigned(blocks < cap ? blocks : cap);
        };
        if (!on_boundary(32, p->x, p->residual, p->out, p->residual_out)) {
            if (p->residual != nullptr)
                launch_chained(roundtrip_ragged_kernel<T, G, BIT, true>, grid(one), stream, *p);
            else
                launch_chained(roundtrip_ragged_kernel<T, G, BIT, false>, grid(one), stream, *p);
            return cudaGetLastError();
        }
        if (p->residual != nullptr) {
            launch_chained(roundtrip_kernel<T, G, BIT, true, 1>, grid(one), stream, *p);
            return cudaGetLastError();
        }
        // Two chunks per thread (64 bytes in flight) above one default grid.  One chunk / two, in a CUDA graph, bf16: 2 Mi
        // elements 1.91 / 1.93 us, 2.5 Mi 2.44 / 2.69, 4.5 Mi 3.18 / 2.67, 5 Mi (above) 3.62 / 3.42, 8 Mi 4.86 / 4.13, 13.1 M 7.52 / 6.60,
        // 33 Mi 24.9 / 21.7, 128 Mi 91.1 / 78.9; fp16 3 Mi 2.63 / 3.00, 4.5 Mi 3.09 / 3.08, which is why the line is not lower, where
        // bf16 would gain (4 Mi 2.91 / 2.68).  fp32 chunks and chunks with a residual have 64 bytes in flight already.
        if constexpr (sizeof(T) == 2) {
            if (one > lbc_default_max_blocks()) {
                launch_chained(roundtrip_kernel<T, G, BIT, false, 2>, grid((one + 1) / 2), stream, *p);
                return cudaGetLastError();
            }
        }
        launch_chained(roundtrip_kernel<T, G, BIT, false, 1>, grid(one), stream, *p);
        return cudaGetLastError();
    }
};

}  // namespace lbc

extern "C" {

cudaError_t lbc_roundtrip(const LbcRoundtrip* p, cudaStream_t stream) {
    if (p == nullptr || p->numel < 0 || (p->passes != 1 && p->passes != 2)) return cudaErrorInvalidValue;
    if (p->residual == nullptr && (p->residual_out != nullptr || p->own_error)) return cudaErrorInvalidValue;
    // the pad is written with the tile that holds the tensor's end: a tensor that fills its tiles has none (see lbc_api.h)
    if (p->pad < 0 || (p->pad > 0 && p->group_size > 0 && p->numel % (8 * int64_t(p->group_size)) == 0))
        return cudaErrorInvalidValue;
    if (p->numel == 0) return cudaSuccess;
    if (p->x == nullptr || p->out == nullptr) return cudaErrorInvalidValue;
    return lbc::dispatch_profile<lbc::RoundtripLauncher>(p, stream);
}

}  // extern "C"
