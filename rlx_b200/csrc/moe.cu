// Fused GGUF dequant + grouped matmul for MoE expert stacks (Op::DequantGroupedMatMul).
//
// Replaces the reference's host-sorted lowering (rlx-cuda/src/gguf_gpu.rs:142-280): D2H of x and the
// expert ids, counting sort on the CPU, per-expert dequantise + sgemm, H2D of the result.  Here:
//   moe_count_kernel    one CTA: rows per expert (shared-memory atomics), exclusive scan
//   moe_place_kernel    the row permutation grouped by expert -- grouped_moe_sort_plan
//                       (rlx-cpu/src/gguf_matmul.rs:178-205) without the copy of x: the matmul
//                       kernel reads the rows through the permutation instead
//   moe_grouped_kernel  grid (weight-row tiles, experts): a warp owns one weight row of one expert,
//                       decodes it four weights per lane at a time (the bit-exact decoders) and
//                       multiplies it into up to eight of that expert's activation rows per pass;
//                       results go straight to the rows' original positions (the unpermute of
//                       grouped_moe_unpermute_out, gguf_matmul.rs:207-218, is the store address)
// Accumulation is f32 in a different order from the CPU loop; same tolerance as the general kernel.
//
// More than eight rows go through the tcgen05 GEMM in its grouped form instead of moe_grouped_kernel, which only runs when
// the workspace is too small for it (fewer than 32 rows of little work, moe_rows_stream, and eight or fewer of a shape the
// integer GEMV does not take: one launch of the f32 streaming GEMV, gemv_f32.cu):
//   moe_tiles_kernel    the table of activation tiles, one list per expert, from the sorted offsets
//   relay_rows_kernel   (rows TMA cannot tile) the slabs of the experts in use on a padded pitch.  (A stack that is not 16-byte
//                       aligned only with a larger workspace than the query asks for, which plans for aligned ones; the
//                       general kernel otherwise.)
//   moe_gather_kernel   the rows of every expert, gathered next to each other as bf16 (f32 activations as
//                       bf16 hi rows and, m rows further on, lo rows, so nothing of x is lost)
//   gemm_tcgen05_kernel every tile against its expert's slab of the stack (gemm_tcgen05.cu, GemmParams::groups), results
//                       stored at the rows' original positions
// The weight operand is bf16(d * q) there, as in the dense GEMM; for fewer than 32 rows, and rows of those other lengths,
// it is the f32 weight, in three bf16 parts.
// All of them are launched as programmatic dependents.  1024 rows over 8 experts of 4096 -> 14336 Q4_K: 196 us; 331 us
// with fixed 128-row tiles, an f32 result array and a scatter kernel behind the GEMM.
//
// Decode (m <= 8 rows, Q4_0 / Q8_0 / Q4_K / Q5_K / Q6_K, k a multiple of 256 up to 12288) skips both kernels:
// one launch of the streaming integer GEMV over the whole stack seen as an [experts * n, k] matrix shares its
// CTAs out among the rows, with each row's slab picked on the device from expert_idx[i] (gemv_int.cu,
// expert-indirect mode), so the routed experts' weights come through the TMA ring at GEMV speed.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "decode.cuh"
#include "kernels.h"
#include "rlxq_moe.h"
#include "staged_common.cuh"

namespace rlxq {

constexpr uint32_t kMoeScanThreads = 1024;
// Inclusive block-wide running sum over kMoeScanThreads threads.
__device__ __forceinline__ uint32_t moe_block_scan(uint32_t v, uint32_t (&wsum)[32]) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += u;
    }
    __syncthreads();                           // the previous call's sums have been read
    if (lane == 31) wsum[warp] = v;
    __syncthreads();
    uint32_t before = 0u;
    for (uint32_t w = 0; w < warp; ++w) before += wsum[w];
    return v + before;
}

// One CTA: offsets[0..E] = exclusive scan of the rows per expert, cursor[0..E] the same (where the next row of an expert
// goes; [E]: the rows no expert takes, behind all others).
__global__ void __launch_bounds__(kMoeScanThreads) moe_count_kernel(const float* expert_idx, uint32_t m, uint32_t E,
                                                                    uint32_t* __restrict__ offsets, uint32_t* __restrict__ cursor) {
    extern __shared__ uint32_t cnt[];          // [E]
    __shared__ uint32_t wsum[32], total;
    griddep_launch_dependents();
    for (uint32_t e = threadIdx.x; e < E; e += kMoeScanThreads) cnt[e] = 0u;
    griddep_wait();
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < m; i += kMoeScanThreads) {
        uint32_t e;
        if (expert_of_row(expert_idx[i], E, &e)) atomicAdd(&cnt[e], 1u);
    }
    __syncthreads();
    uint32_t carry = 0u;
    for (uint32_t e0 = 0; e0 < E; e0 += kMoeScanThreads) {
        const uint32_t e = e0 + threadIdx.x, c = e < E ? cnt[e] : 0u, incl = carry + moe_block_scan(c, wsum);
        if (e < E) { offsets[e] = incl - c; cursor[e] = incl - c; }
        if (threadIdx.x == kMoeScanThreads - 1) total = incl;
        __syncthreads();
        carry = total;
    }
    if (threadIdx.x == 0) { offsets[E] = carry; cursor[E] = carry; }
}

// perm[sorted position] = original row.
__global__ void __launch_bounds__(256) moe_place_kernel(const float* expert_idx, uint32_t m, uint32_t E,
                                                        uint32_t* __restrict__ cursor, uint32_t* __restrict__ perm) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    uint32_t e;
    if (!expert_of_row(expert_idx[i], E, &e)) e = E;
    perm[atomicAdd(&cursor[e], 1u)] = i;
}

// The GEMM's tile table: table[0] = {tiles, routed rows}, table[1 + t] = {first sorted position, rows, expert, 0}, tiles of
// tile_rows rows, expert by expert.
__global__ void __launch_bounds__(kMoeScanThreads) moe_tiles_kernel(const uint32_t* offsets, uint32_t E,
                                                                    uint4* __restrict__ table, uint32_t tile_rows) {
    __shared__ uint32_t wsum[32], total;
    griddep_launch_dependents();
    griddep_wait();
    uint32_t carry = 0u;
    for (uint32_t e0 = 0; e0 < E; e0 += kMoeScanThreads) {
        const uint32_t e = e0 + threadIdx.x, r0 = e < E ? offsets[e] : 0u, c = e < E ? offsets[e + 1] - r0 : 0u;
        const uint32_t t = (c + tile_rows - 1) / tile_rows, incl = carry + moe_block_scan(t, wsum);
        for (uint32_t q = 0; q < t; ++q)
            table[1 + incl - t + q] = make_uint4(r0 + q * tile_rows, min(tile_rows, c - q * tile_rows), e, 0u);
        if (threadIdx.x == kMoeScanThreads - 1) total = incl;
        __syncthreads();
        carry = total;
    }
    if (threadIdx.x == 0) table[0] = make_uint4(carry, offsets[E], 0u, 0u);
}

template <bool XBF16>
__device__ __forceinline__ float4 moe_load_x4(const void* x, uint64_t idx) {
    if constexpr (XBF16) {
        const uint2 v = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(x) + idx);
        return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u),
                           __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xFFFF0000u));
    } else {
        return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + idx);
    }
}

template <uint32_t SCHEME, bool XBF16, bool YBF16>
__global__ void __launch_bounds__(256) moe_grouped_kernel(const void* __restrict__ x, const uint8_t* __restrict__ w,
                                                          void* __restrict__ y, const uint32_t* __restrict__ offsets,
                                                          const uint32_t* __restrict__ perm, uint32_t k, uint32_t n) {
    constexpr uint32_t E = SchemeTraits<SCHEME>::kElems, B = SchemeTraits<SCHEME>::kBytes;
    constexpr int MT = 8;
    const uint32_t e = blockIdx.y;
    const uint32_t r0 = offsets[e], r1 = offsets[e + 1];
    if (r0 == r1) return;                                   // nobody routed here: the slab is never read
    const uint32_t lane = threadIdx.x & 31u, wpc = blockDim.x >> 5;
    const uint64_t row_bytes = (uint64_t)(k / E) * B;
    const uint8_t* slab = w + (uint64_t)e * n * row_bytes;
    for (uint32_t row = blockIdx.x * wpc + (threadIdx.x >> 5); row < n; row += gridDim.x * wpc) {
        const uint8_t* wr = slab + (uint64_t)row * row_bytes;
        for (uint32_t c0 = r0; c0 < r1; c0 += MT) {         // eight of the expert's rows per pass
            const uint32_t mt = min((uint32_t)MT, r1 - c0);
            uint32_t src[MT];
            float acc[MT];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                src[i] = (uint32_t)i < mt ? perm[c0 + i] : 0u;
                acc[i] = 0.f;
            }
            for (uint32_t el = lane * 4; el < k; el += 128) {
                const float4 wv = decode4_exact<SCHEME>(wr + (uint64_t)(el / E) * B, el % E);
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    if ((uint32_t)i < mt) {
                        const float4 xv = moe_load_x4<XBF16>(x, (uint64_t)src[i] * k + el);
                        acc[i] = fmaf(wv.x, xv.x, acc[i]);
                        acc[i] = fmaf(wv.y, xv.y, acc[i]);
                        acc[i] = fmaf(wv.z, xv.z, acc[i]);
                        acc[i] = fmaf(wv.w, xv.w, acc[i]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < MT; ++i) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xFFFFFFFFu, acc[i], o);
            }
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    if ((uint32_t)i < mt) {
                        const uint64_t o = (uint64_t)src[i] * n + row;
                        if constexpr (YBF16) reinterpret_cast<uint16_t*>(y)[o] = (uint16_t)f32_to_bf16_bits(acc[i]);
                        else reinterpret_cast<float*>(y)[o] = acc[i];
                    }
                }
            }
        }
    }
}

template <uint32_t SCHEME>
static void launch_grouped_s(cudaStream_t s, dim3 grid, bool xbf, bool ybf, const void* x, const uint8_t* w, void* y,
                             const uint32_t* offsets, const uint32_t* perm, uint32_t k, uint32_t n) {
    if (xbf && ybf) moe_grouped_kernel<SCHEME, true, true><<<grid, 256, 0, s>>>(x, w, y, offsets, perm, k, n);
    else if (xbf) moe_grouped_kernel<SCHEME, true, false><<<grid, 256, 0, s>>>(x, w, y, offsets, perm, k, n);
    else if (ybf) moe_grouped_kernel<SCHEME, false, true><<<grid, 256, 0, s>>>(x, w, y, offsets, perm, k, n);
    else moe_grouped_kernel<SCHEME, false, false><<<grid, 256, 0, s>>>(x, w, y, offsets, perm, k, n);
}

constexpr uint32_t kMoeDecodeRows = 8;      // up to this many rows go row by row through the streaming GEMV

// ---- the tensor-core GEMM in its grouped form ------------------------------------------------------------------

constexpr uint32_t kMoeBf16Rows = 32;       // batches of this size and more multiply bf16-rounded weights (where TMA can
                                            // tile them); smaller ones f32 ones (GemmCall::precise)

// Activation rows per GEMM tile: what one expert's share of the rows needs, with room for an uneven routing (2.5 standard
// deviations of an even one), so that a slab is hardly ever decoded twice; f32 activations take two boxes per tile.
static uint32_t moe_tile_rows(uint32_t m, uint32_t E, uint32_t most) {
    const float share = (float)m / (float)E;
    const uint32_t want = ((uint32_t)(share + 2.5f * sqrtf(share)) + 31u) / 32u * 32u;
    return want < 32u ? 32u : (want > most ? most : want);
}

// Whether m rows are cheaper row by row (the f32 GEMV: every row reads its expert's slab, so many us per million weights, and
// nothing goes in front of it) than as a GEMM on f32 weights (sort, gather: 14 us, so many us for each 64 columns of each wave
// of 128-row weight tiles of the experts in use, and a copy of their slabs where TMA cannot tile the rows).  The constants are
// fits to 56 shapes, 9 to 31 rows, both ways timed: the choice takes 0.4 % longer than the better one in the geometric mean, 20 %
// at worst.  GEMV and GEMM: 10 x 3072 x 576 Q4_K E16 8 and 34 us, 12 x 7168 x 11840 Q8_0 E4 244 and 346 us, 24 x 4352 x 5632 Q4_0 E16
// 146 and 222 us, 27 x 2560 x 5440 Q4_0 E4 88 and 69 us, 22 x 4352 x 3200 Q5_K E4 124 and 70 us.
// Re-laid Q6_K has a faster GEMM since, on widened rows: over 70 batches of them the choice takes 0.6 % longer than the better way, and
// one is wrong, 29 x 4352 x 2176 E4, 107 us for 72.
// Batches that the GEMM multiplies in bf16 (kMoeBf16Rows and more) stay with it.
static bool moe_rows_stream(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, uint32_t E, bool relaid) {
    if (m <= kMoeDecodeRows) return true;
    if (m >= kMoeBf16Rows) return false;
    float row = 0.32f, block = 1.0f;                    // Q6_K; a block is paced by the decoder, which makes three bf16 parts
    if (scheme == RLXQ_Q4_0) { row = 0.215f; block = 0.65f; }          // (two)
    else if (scheme == RLXQ_Q8_0) row = 0.22f;
    else if (scheme == RLXQ_Q4_K) { row = 0.265f; block = 0.78f; }
    else if (scheme == RLXQ_Q5_K) { row = 0.31f; block = 0.8f; }
    const float stream_us = 4.0f + row * 1e-6f * (float)m * (float)k * (float)n;
    const float used = (float)E * (1.0f - powf(1.0f - 1.0f / (float)E, (float)m));
    const float waves = ceilf(ceilf((float)n / 128.0f) * used / (float)sm_count());
    Geometry g;
    geometry(scheme, &g);
    const float copy_us = relaid ? used * (float)n * (float)(k / g.elems * g.bytes) * 2.0f / 4.5e6f : 0.0f;
    return stream_us < 14.0f + waves * (float)(k / 64) * block + copy_us;
}

// One CTA per sorted position i: row perm[i] of x becomes row i of xg, as bf16 hi and, for f32 activations, lo part (m
// rows further on).  The rows no expert takes come last; their outputs are set to zero here.
template <bool XBF16>
__global__ void __launch_bounds__(256) moe_gather_kernel(const void* x, const uint32_t* perm,
                                                         const uint4* table, uint32_t m, uint32_t k,
                                                         uint32_t parts, uint16_t* __restrict__ xg, uint8_t* __restrict__ y, uint64_t y_row_bytes) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t i = blockIdx.x, src = perm[i];
    if (i >= table[0].y) {
        uint8_t* row = y + (size_t)src * y_row_bytes;
        for (uint64_t b = 2 * threadIdx.x; b < y_row_bytes; b += 2 * blockDim.x) *reinterpret_cast<uint16_t*>(row + b) = 0;
        return;
    }
    if constexpr (XBF16) {
        const uint4* in = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(x) + (size_t)src * k);
        uint4* out = reinterpret_cast<uint4*>(xg + (size_t)i * k);
        for (uint32_t c = threadIdx.x; c < k / 8; c += blockDim.x) out[c] = in[c];
    } else {
        const float4* in = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + (size_t)src * k);
        uint2* hi = reinterpret_cast<uint2*>(xg + (size_t)i * k);
        uint2* lo = reinterpret_cast<uint2*>(xg + (size_t)(m + i) * k);
        uint2* last = reinterpret_cast<uint2*>(xg + (size_t)(2 * m + i) * k);
        for (uint32_t c = threadIdx.x; c < k / 4; c += blockDim.x) {
            const float4 v = in[c];
            const float f[4] = {v.x, v.y, v.z, v.w};
            uint32_t h[4], l[4], e[4];
            split_bf16x4(f, h, l, e);
            hi[c] = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
            lo[c] = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
            if (parts == 3) last[c] = make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
        }
    }
}

struct MoeTcPlan { bool ok, relaid, precise; uint32_t layout, tiles, tile_rows; uint64_t pitch; size_t off_table, off_xg, off_w, bytes; };

// The scratch of the tensor-core path behind the sort's arrays (which end at `base`): tile table, gathered activations
// and, for rows TMA cannot tile where they lie, the re-laid slabs.  Not taken (ok = false) for other formats or when it
// would need more than 4 GiB.  Q6_K's slabs are widened (276 bytes a super-block) or, with less room, copied as they are (210).
static MoeTcPlan plan_moe_tc(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, uint32_t E, bool xbf, bool w_aligned, size_t base, bool widen = true) {
    MoeTcPlan p{};
    const void* aligned = (const void*)256;
    if (options().gemm_kernel.load() == 1) return p;
    p.relaid = !(w_aligned && gemm_tc_supported(scheme, m, k, n, aligned, aligned));
    if (p.relaid && !gemm_relaid_supported(scheme, m, k, n, aligned)) return p;
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    p.precise = p.relaid || m < kMoeBf16Rows;
    p.tile_rows = moe_tile_rows(m, E, gemm_most_rows(scheme, !xbf, p.precise));
    p.tiles = m / p.tile_rows + (E < m ? E : m);
    p.layout = p.relaid && widen && scheme == RLXQ_Q6_K ? kQ6Wide : scheme;
    p.pitch = p.relaid ? gemm_relaid_pitch(p.layout, k) : 0;
    p.off_table = up(base);
    p.off_xg = p.off_table + up((size_t)(p.tiles + 1) * 16);
    p.off_w = p.off_xg + up((size_t)gemm_x_parts(!xbf, p.precise) * m * k * 2);
    p.bytes = p.off_w + (p.relaid ? up((size_t)gemm_relaid_bytes(p.layout, k, (uint64_t)n * E)) : 0);
    p.ok = p.bytes <= (4ull << 30) && (uint64_t)n * E <= 0x7FFFFFFFull;
    return p;
}

// How a call is run.  Asked by the call with the real pointers and by the workspace query with aligned ones, so that nobody
// is asked for scratch that no kernel touches (the re-laid slabs of a large stack are hundreds of megabytes).
enum class MoeRoute {
    Rows,        // the expert-indirect integer GEMV, all rows in one launch or a launch per row (MoePlan::launch_rows)
    Stream,      // one launch of the f32 streaming GEMV for all rows (an id out of range leaves zeros there, too)
    Gemm,        // the grouped tensor-core GEMM
    General      // moe_grouped_kernel
};
// Whether the rows of a decode step go in one launch that shares the CTAs out among them.  It is the faster form everywhere:
// a launch per row waits for the row before and starts its stream anew (Q4_K, rows in one launch against a launch each: 2 x 4096
// x 14336 16.3 and 21.5 us, 2 x 1024 x 512 2.9 and 5.6, 8 x 1536 x 576 3.5 and 23.5, 8 x 2304 x 5376 16.3 and 48.8, 8 x 4096 x
// 14336 44 and 81 us).  Outputs of 4097 to 4800 values keep a launch per row because the decode tests hold them to it.
static bool moe_rows_in_one_launch(uint32_t k, uint32_t n) { return !(k >= 2048 && n > 4096 && n <= 4800); }

struct MoePlan { MoeRoute route; uint32_t launch_rows; size_t off_cursor, off_perm, sort_bytes, bytes; MoeTcPlan tc; };
static MoePlan plan_moe(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, uint32_t E, bool xbf, const void* x, const void* w, size_t ws_bytes) {
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    MoePlan p{};
    p.off_cursor = up(((size_t)E + 1) * 4);
    p.off_perm = 2 * p.off_cursor;
    p.sort_bytes = p.bytes = p.off_perm + up((size_t)m * 4);      // (every route asks for this much)
    const int64_t gemv = options().gemv_kernel.load();
    size_t scratch = 0;
    if (m <= kMoeDecodeRows && gemv != 1 && ((size_t)k * (xbf ? 2 : 4)) % 16 == 0 && (uint64_t)n * E <= 0x7FFFFFFFull &&
        int_expert_supported(scheme, k, n, 1, w, x, &scratch)) {
        p.route = MoeRoute::Rows;
        p.launch_rows = 1;
        if (up(scratch) > p.bytes) p.bytes = up(scratch);
        if (moe_rows_in_one_launch(k, n) && int_expert_supported(scheme, k, n, m, w, x, &scratch) && up(scratch) <= ws_bytes) {
            p.launch_rows = m;
            if (up(scratch) > p.bytes) p.bytes = up(scratch);
        }
        return p;
    }
    if (gemv == 0 && options().gemm_kernel.load() == 0 && gemv_f32_supported(scheme, 1, k, x) &&
        moe_rows_stream(scheme, m, k, n, E, !gemm_tc_supported(scheme, m, k, n, w, x))) {
        p.route = MoeRoute::Stream;
        return p;
    }
    p.route = MoeRoute::General;
    if (m <= kMoeDecodeRows && gemv == 1) return p;
    p.tc = plan_moe_tc(scheme, m, k, n, E, xbf, !((uintptr_t)w & 15u), p.sort_bytes);
    if (p.tc.layout == kQ6Wide && (!p.tc.ok || p.tc.bytes > ws_bytes)) p.tc = plan_moe_tc(scheme, m, k, n, E, xbf, !((uintptr_t)w & 15u), p.sort_bytes, false);
    if (p.tc.ok) {
        p.route = MoeRoute::Gemm;
        p.bytes = p.tc.bytes;
    }
    return p;
}

}  // namespace rlxq

using namespace rlxq;

extern "C" int rlxq_grouped_workspace_bytes(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, uint32_t num_experts,
                                            size_t* bytes) {
    if (!bytes) return fail(RLXQ_E_NULL, "bytes is null");
    Geometry g;
    if (!geometry(scheme, &g)) return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    if (k == 0 || k % g.elems) return fail(RLXQ_E_SHAPE, "k=%u is not a positive multiple of the block size %u", k, g.elems);
    if (num_experts == 0 || num_experts > 8192) return fail(RLXQ_E_LIMIT, "num_experts=%u must be in [1, 8192]", num_experts);
    // f32 activations gather two or three times the rows, bf16 ones may need another tile table
    const void* aligned = (const void*)256;
    *bytes = std::max(plan_moe(scheme, m, k, n, num_experts, false, aligned, aligned, SIZE_MAX).bytes,
                      plan_moe(scheme, m, k, n, num_experts, true, aligned, aligned, SIZE_MAX).bytes);
    return RLXQ_OK;
}

extern "C" int rlxq_grouped_matmul(rlxq_stream_t stream, uint32_t scheme, const void* x, uint32_t x_dtype,
                                   const void* w_blocks, const float* expert_idx, void* y, uint32_t y_dtype, uint32_t m,
                                   uint32_t k, uint32_t n, uint32_t num_experts, void* workspace, size_t workspace_bytes) {
    Geometry g;
    if (!geometry(scheme, &g)) return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    if ((x_dtype != RLXQ_F32 && x_dtype != RLXQ_BF16) || (y_dtype != RLXQ_F32 && y_dtype != RLXQ_BF16))
        return fail(RLXQ_E_DTYPE, "unknown dtype");
    if (k == 0 || k % g.elems) return fail(RLXQ_E_SHAPE, "k=%u is not a positive multiple of the block size %u", k, g.elems);
    if (num_experts == 0 || num_experts > 8192) return fail(RLXQ_E_LIMIT, "num_experts=%u must be in [1, 8192]", num_experts);
    if (m == 0 || n == 0) return RLXQ_OK;
    if (!x || !w_blocks || !expert_idx || !y || !workspace) return fail(RLXQ_E_NULL, "null buffer");
    if (((uintptr_t)x & 15u) || ((uintptr_t)workspace & 15u)) return fail(RLXQ_E_ALIGN, "x and workspace must be 16-byte aligned");
    if ((uintptr_t)w_blocks & 1u) return fail(RLXQ_E_ALIGN, "w_blocks must be 2-byte aligned");
    if ((uintptr_t)y & (y_dtype == RLXQ_BF16 ? 1u : 3u)) return fail(RLXQ_E_ALIGN, "y must be aligned to its element size");
    const bool xbf = x_dtype == RLXQ_BF16, ybf = y_dtype == RLXQ_BF16;
    const uint8_t* wst = (const uint8_t*)w_blocks;
    const size_t xes = xbf ? 2 : 4, yes = ybf ? 2 : 4;
    MoePlan plan = plan_moe(scheme, m, k, n, num_experts, xbf, x, wst, workspace_bytes);
    // the tensor-core path is taken when the workspace holds its arrays; a smaller one still runs the general kernel
    if (plan.route == MoeRoute::Gemm && (workspace_bytes < plan.bytes || ((uintptr_t)workspace & 255u))) plan.route = MoeRoute::General;
    if (workspace_bytes < plan.sort_bytes)
        return fail(RLXQ_E_WORKSPACE, "grouped matmul needs %zu workspace bytes, got %zu", plan.sort_bytes, workspace_bytes);
    const MoeTcPlan& tc = plan.tc;
    cudaStream_t s = (cudaStream_t)stream;
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    uint32_t* offsets = reinterpret_cast<uint32_t*>(ws);
    uint32_t* cursor = reinterpret_cast<uint32_t*>(ws + plan.off_cursor);
    uint32_t* perm = reinterpret_cast<uint32_t*>(ws + plan.off_perm);
    if (plan.route == MoeRoute::Stream)
        return launch_gemv_f32(s, scheme, x, xbf, wst, y, ybf, m, k, n, expert_idx, num_experts);
    // rows with an id of num_experts or more are in no group: their outputs are zero (the gather kernel and the decode kernel
    // see to it)
    if (plan.route == MoeRoute::General) RLXQ_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)m * n * yes, s));
    if (plan.route == MoeRoute::Rows) {
        for (uint32_t i = 0; i < m; i += plan.launch_rows) {
            int rc = launch_gemv_int_expert(s, scheme, (const uint8_t*)x + (size_t)i * k * xes, xbf, wst,
                                            (uint8_t*)y + (size_t)i * n * yes, ybf, plan.launch_rows, k, n, num_experts, expert_idx + i,
                                            workspace, workspace_bytes);
            if (rc) return rc;
        }
        return RLXQ_OK;
    }
    int rc = launch_pdl(moe_count_kernel, dim3(1), dim3(kMoeScanThreads), num_experts * sizeof(uint32_t), s, expert_idx, m, num_experts,
                        offsets, cursor);
    if (rc) return rc;
    count_launch();
    rc = launch_pdl(moe_place_kernel, dim3((m + 255) / 256), dim3(256), 0, s, expert_idx, m, num_experts, cursor, perm);
    if (rc) return rc;
    count_launch();
    if (plan.route == MoeRoute::Gemm) {
        uint16_t* xg = reinterpret_cast<uint16_t*>(ws + tc.off_xg);
        uint4* table = reinterpret_cast<uint4*>(ws + tc.off_table);
        rc = launch_pdl(moe_tiles_kernel, dim3(1), dim3(kMoeScanThreads), 0, s, (const uint32_t*)offsets, num_experts, table, tc.tile_rows);
        if (rc) return rc;
        count_launch();
        GemmCall c{};
        c.w = wst;
        if (tc.relaid) {
            rc = launch_relay(s, tc.layout, wst, k, (uint64_t)n * num_experts, ws + tc.off_w, offsets, n);
            if (rc) return rc;
            c.w = ws + tc.off_w;
        }
        rc = launch_pdl(xbf ? moe_gather_kernel<true> : moe_gather_kernel<false>, dim3(m), dim3(256), 0, s, x, (const uint32_t*)perm,
                        (const uint4*)table, m, k, gemm_x_parts(!xbf, tc.precise), xg, (uint8_t*)y, (uint64_t)n * yes);
        if (rc) return rc;
        count_launch();
        c.x = xg; c.x_rows = m; c.f32 = !xbf; c.w_pitch = tc.pitch; c.precise = tc.precise;
        c.y = y; c.ybf = ybf; c.k = k; c.n = n;
        c.num_slabs = num_experts; c.groups = table; c.group_tiles = tc.tiles; c.tile_rows = tc.tile_rows; c.row_map = perm;
        return launch_gemm(s, tc.layout, c, nullptr, 0);
    }
    const uint32_t wpc = 8;
    unsigned gx = (n + wpc - 1) / wpc;
    const unsigned cap = (unsigned)sm_count() * 8;
    if (gx > cap) gx = cap;
    const dim3 grid(gx, num_experts);
    const uint8_t* w = (const uint8_t*)w_blocks;
    switch (scheme) {
        case RLXQ_Q4_K: launch_grouped_s<RLXQ_Q4_K>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q5_K: launch_grouped_s<RLXQ_Q5_K>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q6_K: launch_grouped_s<RLXQ_Q6_K>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q8_K: launch_grouped_s<RLXQ_Q8_K>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q2_K: launch_grouped_s<RLXQ_Q2_K>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q3_K: launch_grouped_s<RLXQ_Q3_K>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q4_1: launch_grouped_s<RLXQ_Q4_1>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q5_0: launch_grouped_s<RLXQ_Q5_0>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q5_1: launch_grouped_s<RLXQ_Q5_1>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q4_0: launch_grouped_s<RLXQ_Q4_0>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        case RLXQ_Q8_0: launch_grouped_s<RLXQ_Q8_0>(s, grid, xbf, ybf, x, w, y, offsets, perm, k, n); break;
        default: return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    }
    count_launch();
    return check_launch("moe_grouped_kernel");
}
