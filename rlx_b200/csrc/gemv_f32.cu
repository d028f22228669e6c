// Streaming decode GEMV for weight rows of any length (batch 1-8; Q4_0, Q8_0, Q4_K, Q5_K, Q6_K): the rows that TMA cannot
// tile, because they are no multiple of 16 bytes (Q6_K with k not a multiple of 2048, the 32-weight formats with k not a
// multiple of 256) or the weights do not start on a 16-byte boundary; and, in one launch, the rows of an expert batch that
// has too few of them for the GEMM (moe.cu).  (Five to eight rows of three of the formats, where there is enough work:
// gemv_parts.cu.)
//
// Activations stay f32, in registers.  A CTA's warps stand side by side over the columns: warp c owns columns
// [c * 32 * LW, (c + 1) * 32 * LW), a lane LW of them, and keeps its activations of MR batch rows for the whole kernel, while
// the CTA's weight rows stream by, RS rows a step.  Each warp fetches its own pieces of the rows into a ring of its own, in
// 16-byte asynchronous copies from the boundary below the piece, so a row may start on any even byte and no warp waits for
// another; the ring's depth keeps about 100 KB per SM in flight.  A lane decodes its LW weights (one byte-permute each,
// packed two-float arithmetic from there on), multiplies, and applies the block scale once per block; the warp's sums of a
// step's rows are reduced together and go to shared memory, where the warps' sums meet once per 32 rows.
//
// Bound: instruction issue (a weight costs 3.5 lane instructions in Q8_0, 4.5 in Q6_K, 2 of them the multiplication).  Row
// by row (RS = 1) as much again went into ring positions, copy addresses and the reduction, in a chain that left half of
// the issue slots empty; RS rows a step share that and overlap.  Batch 1, 5888 or 5920 -> 28672, RS = 1 against now: Q6_K
// 79 -> 53 us, Q8_0 63 -> 42 us (4.3 TB/s), Q4_0 61 -> 37 us; batch 4: 112 -> 92, 123 -> 79, 101 -> 78 us.  More warps per SM
// (18 for 16) and half as many weights a lane did not help.
#include "common.cuh"
#include "decode.cuh"
#include "f32x2.cuh"
#include "kernels.h"
#include "staged_common.cuh"

namespace rlxq {

constexpr uint32_t kF32Batch = 32;        // weight rows between two meetings of the warps
constexpr uint32_t kF32MaxWarps = 16;

struct F32Params {
    const void* x;
    const uint8_t* w;
    void* y;
    uint32_t x_bf16, y_bf16, m, k, n;
    uint64_t row_bytes;
    uint32_t passes;                      // column passes: more than kF32MaxWarps pieces are taken one set after the other
    uint32_t tiles, groups;               // CTA b: tile b / groups of the weight rows, batch rows MR * (b % groups) ..
    // Expert stacks: w holds num_experts slabs of n rows, groups = m, and CTA b multiplies batch row b % groups by the slab
    // that expert_idx names for it (none: the row of y is zero).
    const float* expert_idx;
    uint32_t num_experts;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint32_t s32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
// N consecutive words / the 16 bits at an even shared-memory byte address.
template <int N> __device__ __forceinline__ void s32_even(uint32_t a, uint32_t (&w)[N]) {
    const uint32_t b = a & ~3u, sh = (a & 2u) * 8u;
    uint32_t prev = s32(b);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t next = s32(b + 4 * i + 4);
        w[i] = __funnelshift_r(prev, next, sh);
        prev = next;
    }
}
__device__ __forceinline__ uint32_t s16_even(uint32_t a) { return (s32(a & ~3u) >> ((a & 2u) * 8u)) & 0xFFFFu; }

// The four bytes of u, less OFF, times x pairs xi, xi + 1 of every batch row.
template <int OFF, int MR, int NX>
__device__ __forceinline__ void mul_word(uint32_t u, const uint64_t (&x)[MR][NX], int xi, uint64_t (&acc)[MR]) {
    const uint32_t o = __float_as_uint(-(8388608.0f + (float)OFF));
    const uint64_t off = f32x2(o, o);
    const uint64_t a = add_f32x2(magic_pair<0>(u), off);
    const uint64_t b = add_f32x2(magic_pair<1>(u), off);
#pragma unroll
    for (int r = 0; r < MR; ++r) {
        acc[r] = fma_f32x2(a, x[r][xi], acc[r]);
        acc[r] = fma_f32x2(b, x[r][xi + 1], acc[r]);
    }
}

// One lane's LW weights of a row piece whose first block lies at shared-memory address p (even), in sum[].  xs: the sums of
// the lane's activations (NEEDS_SUM: formats with a minimum).
template <uint32_t SCHEME, int MR, int LW> struct F32Lane;

template <int MR, int LW> struct F32Lane<RLXQ_Q8_0, MR, LW> {
    static constexpr bool NEEDS_SUM = false;
    __device__ static __forceinline__ void run(uint32_t p, uint32_t lane, const uint64_t (&x)[MR][LW / 2], const float (&)[MR], float (&sum)[MR]) {
        const uint32_t blk = p + 34u * (lane * LW / 32);
        uint32_t q[LW / 4];
        s32_even<LW / 4>(blk + 2 + (lane * LW) % 32, q);
        const float d = f16_bits_to_f32(s16_even(blk));
        uint64_t acc[MR];
#pragma unroll
        for (int r = 0; r < MR; ++r) acc[r] = 0ull;
#pragma unroll
        for (int i = 0; i < LW / 4; ++i) mul_word<128>(q[i] ^ 0x80808080u, x, 2 * i, acc);
#pragma unroll
        for (int r = 0; r < MR; ++r) sum[r] = d * sum_f32x2(acc[r]);
    }
};

template <int MR, int LW> struct F32Lane<RLXQ_Q4_0, MR, LW> {
    static constexpr bool NEEDS_SUM = false;
    // low nibbles: weights 0..15 of the block, high nibbles: 16..31
    __device__ static __forceinline__ void run(uint32_t p, uint32_t lane, const uint64_t (&x)[MR][LW / 2], const float (&)[MR], float (&sum)[MR]) {
        const uint32_t blk = p + 18u * (lane * LW / 32);
        uint64_t acc[MR];
#pragma unroll
        for (int r = 0; r < MR; ++r) acc[r] = 0ull;
        uint32_t q[4];
        s32_even<4>(blk + 2, q);
        if constexpr (LW == 32) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                mul_word<8>(q[i] & 0x0F0F0F0Fu, x, 2 * i, acc);
                mul_word<8>((q[i] >> 4) & 0x0F0F0F0Fu, x, 8 + 2 * i, acc);
            }
        } else {
            static_assert(LW == 16, "half a block");
            const uint32_t sh = 4u * (lane & 1u);
#pragma unroll
            for (int i = 0; i < 4; ++i) mul_word<8>((q[i] >> sh) & 0x0F0F0F0Fu, x, 2 * i, acc);
        }
        const float d = f16_bits_to_f32(s16_even(blk));
#pragma unroll
        for (int r = 0; r < MR; ++r) sum[r] = d * sum_f32x2(acc[r]);
    }
};

// Q6_K (ql[128] | qh[64] | sc[16] i8 | d f16, order as rlx-gguf/src/lib.rs:1070-1114): weights 128 h + 32 g + 16 i .. of the
// super-block are nibble g >> 1 of ql bytes 64 h + 32 (g & 1) + 16 i .. and bits 2 g, 2 g + 1 of qh bytes 32 h + 16 i ..
template <int MR, int LW> struct F32Lane<RLXQ_Q6_K, MR, LW> {
    static constexpr bool NEEDS_SUM = false;
    __device__ static __forceinline__ void run(uint32_t p, uint32_t lane, const uint64_t (&x)[MR][LW / 2], const float (&)[MR], float (&sum)[MR]) {
        constexpr uint32_t PER = 256 / LW;                 // lanes per super-block
        const uint32_t sb = p + 210u * (lane / PER), j = lane % PER;
        const uint32_t e = j * LW, h = e >> 7, g = (e >> 5) & 3u, i0 = (e >> 4) & 1u;
        uint32_t ql[LW / 4], qh[LW / 4];
        s32_even<LW / 4>(sb + 64 * h + 32 * (g & 1u) + 16 * i0, ql);
        s32_even<LW / 4>(sb + 128 + 32 * h + 16 * i0, qh);
        const uint32_t sc = s16_even(sb + 192 + ((8 * h + 2 * g + i0) & ~1u)) >> (LW == 16 ? 8 * i0 : 0);
        const float d = f16_bits_to_f32(s16_even(sb + 208));
        const uint32_t nib = 4u * (g >> 1), hs = 2u * g;
#pragma unroll
        for (int r = 0; r < MR; ++r) sum[r] = 0.f;
#pragma unroll
        for (int s = 0; s < LW / 16; ++s) {
            uint64_t acc[MR];
#pragma unroll
            for (int r = 0; r < MR; ++r) acc[r] = 0ull;
#pragma unroll
            for (int i = 4 * s; i < 4 * s + 4; ++i)
                mul_word<32>(((ql[i] >> nib) & 0x0F0F0F0Fu) | (((qh[i] >> hs) << 4) & 0x30303030u), x, 2 * i, acc);
            const float ds = d * (float)(int8_t)((sc >> (8 * s)) & 0xFFu);
#pragma unroll
            for (int r = 0; r < MR; ++r) sum[r] = fmaf(ds, sum_f32x2(acc[r]), sum[r]);
        }
    }
};

// Q4_K, Q5_K (d f16 | dmin f16 | 12 bytes of 6-bit scales and minima | Q5_K: qh[32] | qs[128], order as
// rlx-gguf/src/lib.rs:988-1068): weights 32 s .. of the super-block are nibble s & 1 of qs bytes 32 (s >> 1) .., plus bit s of
// qh[0..32) as 16; the value is d * scale * q - dmin * minimum.
template <uint32_t SCHEME, int MR, int LW> struct F32LaneK45 {
    static constexpr bool NEEDS_SUM = true;
    __device__ static __forceinline__ void run(uint32_t p, uint32_t lane, const uint64_t (&x)[MR][LW / 2], const float (&xs)[MR], float (&sum)[MR]) {
        constexpr bool K5 = SCHEME == RLXQ_Q5_K;
        constexpr uint32_t PER = 256 / LW;                 // lanes per super-block
        const uint32_t sb = p + (K5 ? 176u : 144u) * (lane / PER), e = (lane % PER) * LW, s = e >> 5, i0 = e & 16u;
        uint32_t h[4], q[LW / 4], qh[LW / 4];
        s32_even<4>(sb, h);
        s32_even<LW / 4>(sb + (K5 ? 48 : 16) + 32 * (s >> 1) + i0, q);
        if constexpr (K5) s32_even<LW / 4>(sb + 16 + i0, qh);
        const uint32_t nib = 4u * (s & 1u), j = 8u * (s & 3u);
        const uint32_t a = (h[1] >> j) & 0xFFu, b = (h[2] >> j) & 0xFFu, c = (h[3] >> j) & 0xFFu;
        const uint32_t sc = s < 4 ? a & 63u : (c & 15u) | ((a >> 6) << 4), mn = s < 4 ? b & 63u : (c >> 4) | ((b >> 6) << 4);
        uint64_t acc[MR];
#pragma unroll
        for (int r = 0; r < MR; ++r) acc[r] = 0ull;
#pragma unroll
        for (int i = 0; i < LW / 4; ++i) {
            uint32_t u = (q[i] >> nib) & 0x0F0F0F0Fu;
            if constexpr (K5) u |= ((qh[i] >> s) & 0x01010101u) << 4;
            mul_word<0>(u, x, 2 * i, acc);
        }
        const float d = f16_bits_to_f32(h[0] & 0xFFFFu) * (float)sc, dm = f16_bits_to_f32(h[0] >> 16) * (float)mn;
#pragma unroll
        for (int r = 0; r < MR; ++r) sum[r] = fmaf(d, sum_f32x2(acc[r]), -dm * xs[r]);
    }
};
template <int MR, int LW> struct F32Lane<RLXQ_Q4_K, MR, LW> : F32LaneK45<RLXQ_Q4_K, MR, LW> {};
template <int MR, int LW> struct F32Lane<RLXQ_Q5_K, MR, LW> : F32LaneK45<RLXQ_Q5_K, MR, LW> {};

template <int MR> constexpr int f32_lane_weights() { return MR <= 2 ? 32 : 16; }
// bytes of a row's piece (32 * LW weights), and of its slot: from the 16-byte boundary below it to the one above
template <uint32_t SCHEME, int LW> constexpr uint32_t f32_piece_bytes() {
    return 32u * LW / SchemeTraits<SCHEME>::kElems * SchemeTraits<SCHEME>::kBytes;
}
template <uint32_t SCHEME, int LW> constexpr uint32_t f32_slot_bytes() { return (f32_piece_bytes<SCHEME, LW>() + 30) / 16 * 16 + 16; }
// RS, rows per step: 4 or 8 sums meet in one reduction; three steps of sixteen warps have to fit in shared memory
template <uint32_t SCHEME, int MR> constexpr int f32_step_rows() {
    return MR >= 2 || f32_slot_bytes<SCHEME, f32_lane_weights<MR>()>() > 1000 ? 2 : 4;
}
template <uint32_t SCHEME, int MR, int RS> constexpr int f32_depth() {             // about 128 KB over sixteen warps, 3 to 8 steps
    constexpr int d = 8192 / (int)(f32_slot_bytes<SCHEME, f32_lane_weights<MR>()>() * RS);
    return d < 3 ? 3 : d > 8 ? 8 : d;
}
// Adds OUT values over the lanes of a warp: lanes exchange halves of the values first (OUT / 2, OUT / 4, .. shuffles), then
// the rest.  Value v ends in the lanes whose upper bits spell v.
template <int OUT> __device__ __forceinline__ float warp_sums(float (&v)[OUT], uint32_t lane) {
#pragma unroll
    for (int w = OUT / 2, bit = 16; w >= 1; w /= 2, bit /= 2) {
        const bool up = lane & (uint32_t)bit;
#pragma unroll
        for (int q = 0; q < w; ++q) {
            const float mine = up ? v[q + w] : v[q], theirs = up ? v[q] : v[q + w];
            v[q] = mine + __shfl_xor_sync(0xFFFFFFFFu, theirs, bit);
        }
    }
    float r = v[0];
#pragma unroll
    for (int o = 16 / OUT; o >= 1; o /= 2) r += __shfl_xor_sync(0xFFFFFFFFu, r, o);
    return r;
}

template <uint32_t SCHEME, int MR, int RS>
__global__ void __launch_bounds__(kF32MaxWarps * 32, 1) gemv_f32_kernel(const __grid_constant__ F32Params P) {
    constexpr int LW = f32_lane_weights<MR>(), D = f32_depth<SCHEME, MR, RS>(), OUT = RS * MR;
    constexpr uint32_t COLS = 32 * LW, PIECE = f32_piece_bytes<SCHEME, LW>(), SLOT = f32_slot_bytes<SCHEME, LW>();
    constexpr uint32_t LPR = 32 / RS;                      // lanes that copy one row of a step
    constexpr int COPIES = (int)((PIECE + 14 + 15) / 16 + LPR - 1) / (int)LPR;
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nwarps = blockDim.x >> 5;
    float* red = reinterpret_cast<float*>(smem);                                   // [2][kF32Batch][nwarps][MR]
    const uint32_t ring = smem_u32(smem) + 2 * kF32Batch * nwarps * MR * 4 + warp * (D * RS * SLOT);
    griddep_launch_dependents();

    const uint32_t tile = blockIdx.x / P.groups, m0 = (blockIdx.x - tile * P.groups) * MR;
    const uint32_t r0 = (uint32_t)((uint64_t)tile * P.n / P.tiles), r1 = (uint32_t)((uint64_t)(tile + 1) * P.n / P.tiles);
    const uint32_t rows = r1 - r0;
    const uint8_t* w = P.w;
    bool none = false;
    if (P.expert_idx) {                   // which slab is known only after the kernel in front
        griddep_wait();
        uint32_t e = 0;
        none = !expert_of_row(P.expert_idx[m0], P.num_experts, &e);
        w += (uint64_t)e * P.n * P.row_bytes;
    }
    // A step: RS rows of a batch of up to kF32Batch rows, in one column pass.  Rows past the last are the last row again.
    const uint32_t batches = (rows + kF32Batch - 1) / kF32Batch;
    struct Pos { uint32_t b, pass, i; };
    auto batch_rows = [&](uint32_t b) { return min(kF32Batch, rows - b * kF32Batch); };
    const uint32_t crow = lane / LPR, cchunk = lane % LPR;                         // this lane's share of the copies
    auto fetch = [&](const Pos& p, uint32_t slot) {
        const uint64_t off = (uint64_t)(p.pass * nwarps + warp) * PIECE;
        if (off < P.row_bytes && !none) {
            const uint32_t row = min(p.b * kF32Batch + p.i + crow, rows - 1);
            const uint8_t* src = w + (uint64_t)(r0 + row) * P.row_bytes + off;
            const uint32_t lead = (uint32_t)((uintptr_t)src & 15u);
            const uint32_t chunks = (lead + (uint32_t)min((uint64_t)PIECE, P.row_bytes - off) + 15u) / 16u;
            const uint8_t* from = src - lead + 16 * cchunk;
            const uint32_t to = ring + (slot * RS + crow) * SLOT + 16 * cchunk;
#pragma unroll
            for (int c = 0; c < COPIES; ++c)
                if (cchunk + c * LPR < chunks) cp_async16(to + 16 * LPR * c, from + 16 * LPR * c);
        }
        cp_async_commit();
    };
    auto advance = [&](Pos& p) {
        p.i += RS;
        if (p.i >= batch_rows(p.b)) {
            p.i = 0;
            if (++p.pass == P.passes) { p.pass = 0; ++p.b; }
        }
    };
    Pos next{0, 0, 0};
    uint32_t slot_in = 0, slot = 0;
#pragma unroll 1
    for (int s = 0; s < D - 1; ++s) {
        if (next.b < batches) { fetch(next, slot_in); advance(next); }
        else cp_async_commit();
        if (++slot_in == (uint32_t)D) slot_in = 0;
    }
    if (!P.expert_idx) griddep_wait();    // the weights are on their way; x and y belong to the kernel in front until here

    uint64_t x[MR][LW / 2];
    float xs[MR] = {};
    uint32_t loaded = 0xFFFFFFFFu;        // the column pass whose activations are in x
    for (uint32_t b = 0; b < batches; ++b) {
        const uint32_t nb = batch_rows(b);
        float* rb = red + (b & 1u) * (kF32Batch * nwarps * MR);
        for (uint32_t pass = 0; pass < P.passes; ++pass) {
            const uint32_t c0 = (pass * nwarps + warp) * COLS + lane * LW;
            const bool in = c0 < P.k && !none;
            if (loaded != pass) {
                loaded = pass;
#pragma unroll
                for (int r = 0; r < MR; ++r) {
                    const bool have = in && m0 + r < P.m;
                    if (P.x_bf16) {
                        const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(P.x) + (size_t)(m0 + r) * P.k + c0);
#pragma unroll
                        for (int t = 0; t < LW / 8; ++t) {
                            const uint4 v = have ? src[t] : make_uint4(0u, 0u, 0u, 0u);
                            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int q = 0; q < 4; ++q) x[r][4 * t + q] = f32x2(u[q] << 16, u[q] & 0xFFFF0000u);
                        }
                    } else {
                        const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(P.x) + (size_t)(m0 + r) * P.k + c0);
#pragma unroll
                        for (int t = 0; t < LW / 4; ++t) {
                            const uint4 v = have ? src[t] : make_uint4(0u, 0u, 0u, 0u);
                            x[r][2 * t] = f32x2(v.x, v.y);
                            x[r][2 * t + 1] = f32x2(v.z, v.w);
                        }
                    }
                }
            }
            if constexpr (F32Lane<SCHEME, MR, LW>::NEEDS_SUM) {
#pragma unroll
                for (int r = 0; r < MR; ++r) {
                    uint64_t t = 0ull;
#pragma unroll
                    for (int q = 0; q < LW / 2; ++q) t = add_f32x2(t, x[r][q]);
                    xs[r] = sum_f32x2(t);
                }
            }
            uint32_t at = (uint32_t)(uintptr_t)w + (r0 + b * kF32Batch) * (uint32_t)P.row_bytes + (pass * nwarps + warp) * PIECE;
#pragma unroll 1
            for (uint32_t i = 0; i < nb; i += RS) {
                cp_async_wait<D - 2>();
                __syncwarp();             // every lane's copies of this step have landed, and the slot refilled below is read
                float v[OUT];
#pragma unroll
                for (int o = 0; o < OUT; ++o) v[o] = 0.f;
                if (in) {
#pragma unroll
                    for (int q = 0; q < RS; ++q) {
                        // (a row past the batch's last holds the last row's bytes; its sums are not stored)
                        const uint32_t lead = (at + min((uint32_t)q, nb - 1 - i) * (uint32_t)P.row_bytes) & 15u;
                        float sum[MR];
                        F32Lane<SCHEME, MR, LW>::run(ring + (slot * RS + q) * SLOT + lead, lane, x, xs, sum);
#pragma unroll
                        for (int r = 0; r < MR; ++r) v[q * MR + r] = sum[r];
                    }
                }
                at += RS * (uint32_t)P.row_bytes;
                if (next.b < batches) { fetch(next, slot_in); advance(next); }
                else cp_async_commit();
                if (++slot_in == (uint32_t)D) slot_in = 0;
                if (++slot == (uint32_t)D) slot = 0;
                const float t = warp_sums<OUT>(v, lane);
                constexpr uint32_t SP = 32 / OUT;
                const uint32_t o = lane / SP, q = o / MR;
                if (lane % SP == 0 && i + q < nb) {
                    float* dst = rb + ((i + q) * nwarps + warp) * MR + o % MR;
                    *dst = pass ? *dst + t : t;
                }
            }
        }
        __syncthreads();                  // (the buffers alternate: the next batch writes the other one)
        for (uint32_t o = tid; o < nb * MR; o += blockDim.x) {
            const uint32_t i = o / MR, r = o - i * MR;
            float v = 0.f;
            for (uint32_t c = 0; c < nwarps; ++c) v += rb[(i * nwarps + c) * MR + r];
            if (m0 + r < P.m) {
                if constexpr (F32Lane<SCHEME, MR, LW>::NEEDS_SUM) {
                    // An infinite activation makes infinities of the products and of the minima, and NaN of their difference.
                    // Weight by weight it is the infinity of its weight's sign: once more, out of the way of the main loop.
                    if (v != v && !none) {
                        v = 0.f;
                        const uint8_t* row = w + (uint64_t)(r0 + b * kF32Batch + i) * P.row_bytes;
                        constexpr uint32_t E = SchemeTraits<SCHEME>::kElems, B = SchemeTraits<SCHEME>::kBytes;
#pragma unroll 1
                        for (uint32_t el = 0; el < P.k; el += 4) {
                            const float4 wv = decode4_exact<SCHEME>(row + (uint64_t)(el / E) * B, el % E);
                            const float wf[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                            for (uint32_t q = 0; q < 4; ++q) {
                                const size_t xi = (size_t)(m0 + r) * P.k + el + q;
                                v = fmaf(wf[q], P.x_bf16 ? bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(P.x)[xi])
                                                         : reinterpret_cast<const float*>(P.x)[xi], v);
                            }
                        }
                    }
                }
                const size_t out = (size_t)(m0 + r) * P.n + r0 + b * kF32Batch + i;
                if (P.y_bf16) reinterpret_cast<uint16_t*>(P.y)[out] = (uint16_t)f32_to_bf16_bits(v);
                else reinterpret_cast<float*>(P.y)[out] = v;
            }
        }
    }
}

template <uint32_t SCHEME, int MR, int RS>
static int launch_f32_t(cudaStream_t stream, F32Params P) {
    constexpr int LW = f32_lane_weights<MR>(), D = f32_depth<SCHEME, MR, RS>();
    constexpr uint32_t COLS = 32 * LW, SLOT = f32_slot_bytes<SCHEME, LW>();
    const uint32_t pieces = (P.k + COLS - 1) / COLS;
    P.passes = (pieces + kF32MaxWarps - 1) / kF32MaxWarps;
    const uint32_t warps = (pieces + P.passes - 1) / P.passes;
    // sixteen warps per SM, all of them resident at once
    const uint32_t per_sm = kF32MaxWarps / warps, ctas = (uint32_t)sm_count() * per_sm;
    P.tiles = ctas / P.groups;
    if (P.tiles < 1) P.tiles = 1;
    if (P.tiles > P.n) P.tiles = P.n;
    if constexpr (RS > 1)                 // tiles of fewer rows than a step takes would multiply rows they do not have
        if (P.n / P.tiles < (uint32_t)RS) return launch_f32_t<SCHEME, MR, 1>(stream, P);
    const uint32_t smem = 2 * kF32Batch * warps * MR * 4 + warps * D * RS * SLOT;
    static std::atomic<uint32_t> attr_set[64];
    int dev = 0;
    RLXQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && attr_set[dev].load() == 0) {
        RLXQ_CUDA_TRY(cudaFuncSetAttribute(gemv_f32_kernel<SCHEME, MR, RS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_set[dev].store(1);
    }
    int rc = launch_pdl(gemv_f32_kernel<SCHEME, MR, RS>, dim3(P.tiles * P.groups), dim3(warps * 32), smem, stream, P);
    if (rc) return rc;
    count_launch();
    return check_launch("gemv_f32_kernel");
}

template <uint32_t SCHEME>
static int launch_f32_s(cudaStream_t stream, const F32Params& P) {
    if (P.expert_idx || P.m == 1) return launch_f32_t<SCHEME, 1, f32_step_rows<SCHEME, 1>()>(stream, P);
    if (P.m == 2) return launch_f32_t<SCHEME, 2, f32_step_rows<SCHEME, 2>()>(stream, P);
    return launch_f32_t<SCHEME, 4, f32_step_rows<SCHEME, 4>()>(stream, P);
}

bool gemv_f32_supported(uint32_t scheme, uint32_t m, uint32_t k, const void* x) {
    const bool known = scheme == RLXQ_Q4_0 || scheme == RLXQ_Q8_0 || scheme == RLXQ_Q6_K || scheme == RLXQ_Q4_K || scheme == RLXQ_Q5_K;
    return known && m >= 1 && m <= 8 && !((uintptr_t)x & 15u) && k % 32 == 0;
}

int launch_gemv_f32(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y, bool ybf, uint32_t m,
                    uint32_t k, uint32_t n, const float* expert_idx, uint32_t num_experts) {
    Geometry g;
    if (!geometry(scheme, &g)) return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    F32Params P{};
    P.x = x; P.w = w; P.y = y; P.x_bf16 = xbf; P.y_bf16 = ybf; P.m = m; P.k = k; P.n = n;
    P.row_bytes = (uint64_t)k / g.elems * g.bytes;
    P.expert_idx = expert_idx; P.num_experts = num_experts;
    P.groups = expert_idx ? m : m <= 2 ? 1u : (m + 3) / 4;
    switch (scheme) {
        case RLXQ_Q4_0: return launch_f32_s<RLXQ_Q4_0>(stream, P);
        case RLXQ_Q8_0: return launch_f32_s<RLXQ_Q8_0>(stream, P);
        case RLXQ_Q6_K: return launch_f32_s<RLXQ_Q6_K>(stream, P);
        case RLXQ_Q4_K: return launch_f32_s<RLXQ_Q4_K>(stream, P);
        case RLXQ_Q5_K: return launch_f32_s<RLXQ_Q5_K>(stream, P);
        default: return fail(RLXQ_E_SCHEME, "no f32 streaming GEMV for scheme %u", scheme);
    }
}

}  // namespace rlxq
