// Prefill GEMM (m > 8 activation rows) on the 5th-generation tensor cores: tcgen05.mma with
// the accumulator AND the dequantised weight operand in tensor memory, activations by TMA.
//
// y[m,n] = x[m,k] . W^T is computed transposed, tile by tile: D[128 weight rows, 32 to 256 activation
// rows] += A[128, 64] . B[rows, 64]^T per 64-wide k block.
//   * A (weights) never exists in memory.  The raw GGUF blocks of 128 rows x 256 weights arrive in
//     shared memory through one 2-D TMA box; eight decode warps, twelve for Q3_K (one thread per weight row, which
//     is also that thread's tensor-memory lane) turn 64 weights at a time into bf16(d * q) in
//     registers and store them to tensor memory with tcgen05.st.  d * q is formed in f32 exactly as
//     the reference decoder does (rlx-gguf/src/lib.rs:574-597, 974-1013) and rounded once to bf16.
//   * B (activations, bf16, K-major) comes through TMA with the 128-byte swizzle the MMA's
//     shared-memory descriptor expects.
//   * One thread issues four tcgen05.mma (k = 16 each) per stage and tcgen05.commit releases the
//     stage's shared memory and tensor-memory columns through an mbarrier.
//   * Four epilogue warps read the 128 x 256 f32 accumulator with tcgen05.ld and write y (f32 or
//     bf16, round to nearest even); consecutive lanes hold consecutive n, so stores coalesce.
// Persistent CTAs, one per SM, walk the tiles with the activation tile index fastest so that the
// CTAs working at any moment share a handful of weight tiles (L2 reuse) and x stays L2 resident.
//
// Every wait is bounded: on a timeout the kernel records an error word, stops issuing, lets the
// copies in flight land, frees its tensor memory and returns.
//
// Replaces the reference's dequantise-to-f32-scratch + cublasSgemm for m > 8
// (rlx-cuda/src/gguf_gpu.rs:62-134), which also reads the scratch with the wrong leading
// dimension for n > 1.
#include <algorithm>
#include <chrono>

#include "arrival.h"
#include "common.cuh"
#include "decode.cuh"
#include "f32x2.cuh"
#include "kernels.h"
#include "staged_common.cuh"
#include "tc_common.cuh"
#include "tensormap.cuh"

namespace rlxq {

constexpr uint32_t kGemmTileW = 128;    // weight rows per tile (MMA M, tensor-memory lanes)
constexpr uint32_t kGemmBK = 64;        // k per pipeline stage (one 128-byte swizzled row of bf16)
constexpr uint32_t kGemmMaxStages = 8;  // B shared-memory stages == A tensor-memory stages (8 x 32 columns)
constexpr uint32_t kGemmMaxRaw = 8;     // raw weight boxes (256 weights of 128 rows each): what shared memory is left for
constexpr uint32_t kGemmRawStages = 2;  // the paired kernel's

// ---- weight decode: 64 consecutive weights of one row -> 32 bf16 pairs ------------------------
// The raw box holds 256 weights of 128 rows; RAW_ROW bytes per row (an odd number of 16-byte
// chunks, so one-row-per-lane 128-bit reads do not conflict).  `S` = which 64 of the 256.
template <uint32_t SCHEME> struct GemmRaw;
// GROUPS: decode warp groups (four warps each).  Two keep pace with the MMA for the cheap decoders (more only
// add contention: measured 917 against 950 TFLOP/s for Q8_0); Q3_K's decoder is the slow one and gains from three.
template <> struct GemmRaw<RLXQ_Q4_0> { static constexpr uint32_t ROW = 144, GROUPS = 2; };
template <> struct GemmRaw<RLXQ_Q8_0> { static constexpr uint32_t ROW = 272, GROUPS = 2; };
template <> struct GemmRaw<RLXQ_Q4_K> { static constexpr uint32_t ROW = 144, GROUPS = 2; };
template <> struct GemmRaw<RLXQ_Q5_K> { static constexpr uint32_t ROW = 176, GROUPS = 2; };
// Q6_K super-blocks are 210 bytes: group g of a row starts at byte 210 g, which is only 2-byte aligned.
// The box starts at the 16-byte boundary below it and is 240 bytes wide (15 chunks: conflict-free, and
// 14 + 210 <= 240); the decoder moves the words by the offset.
template <> struct GemmRaw<RLXQ_Q6_K> { static constexpr uint32_t ROW = 240, GROUPS = 2; };
// Q2_K super-blocks are 84 bytes (group g starts 4 (g mod 4) bytes past a 16-byte boundary: a 112-byte box covers
// 12 + 84), Q3_K's 110 bytes (2-byte aligned only, like Q6_K: a 144-byte box covers 14 + 110).
template <> struct GemmRaw<RLXQ_Q2_K> { static constexpr uint32_t ROW = 112, GROUPS = 2; };
// The 32-weight container types: Q4_1 (20-byte blocks: 160 bytes per 256 weights, fetched as 176 so that a row of the
// box is an odd number of 16-byte chunks), Q5_0 (22: 176), Q5_1 (24: 192, fetched as 208).
template <> struct GemmRaw<RLXQ_Q4_1> { static constexpr uint32_t ROW = 176, GROUPS = 2; };
template <> struct GemmRaw<RLXQ_Q5_0> { static constexpr uint32_t ROW = 176, GROUPS = 2; };
template <> struct GemmRaw<RLXQ_Q5_1> { static constexpr uint32_t ROW = 208, GROUPS = 2; };
// Q8_K: 292 bytes (f32 d, 256 int8, 16 int16 block sums that the decoder does not read); 4 (g mod 4) bytes past a
// boundary, a 304-byte box (19 chunks) covers 12 + 292.
template <> struct GemmRaw<RLXQ_Q8_K> { static constexpr uint32_t ROW = 304, GROUPS = 2; };
template <> struct GemmRaw<RLXQ_Q3_K> { static constexpr uint32_t ROW = 144, GROUPS = 3; };
template <> struct GemmRaw<kQ6Wide> { static constexpr uint32_t ROW = 272, GROUPS = 2; };
template <uint32_t SCHEME> __device__ __forceinline__ uint32_t gemm_raw_x(uint32_t g) {   // box start, 8-byte elements
    if (SCHEME == RLXQ_Q6_K) return ((210u * g) & ~15u) / 8u;
    if (SCHEME == RLXQ_Q2_K) return ((84u * g) & ~15u) / 8u;
    if (SCHEME == RLXQ_Q8_K) return ((292u * g) & ~15u) / 8u;
    if (SCHEME == RLXQ_Q4_1) return g * (160u / 8u);
    if (SCHEME == RLXQ_Q5_1) return g * (192u / 8u);
    if (SCHEME == RLXQ_Q3_K) return ((110u * g) & ~15u) / 8u;
    return g * (GemmRaw<SCHEME>::ROW / 8u);
}

// float(b) for b in 0..255 without the conversion unit: 0x4B000000 | b is 2^23 + b
__device__ __forceinline__ float u8_to_f32(uint32_t b) { return __uint_as_float(0x4B000000u | b) - 8388608.0f; }
// float(b) - OFF in one exact subtraction (OFF a small integer)
template <int OFF>
__device__ __forceinline__ float u8_minus(uint32_t b) { return __uint_as_float(0x4B000000u | b) - (8388608.0f + (float)OFF); }

// The decoders are bound by instruction issue (two decode warps share a scheduler with the MMA pace of one
// k block per 512 cycles), so they work on pairs: one byte-permute per weight builds the float 2^23 + byte
// straight from the raw word, and the arithmetic uses the packed two-float instructions of this architecture.
// Every step rounds exactly as the scalar f32 expression it replaces.
// two floats -> bf16 pair, the first in the low half
__device__ __forceinline__ uint32_t bf16x2_of(uint64_t v) {
    uint32_t lo, hi, d;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
    return d;
}
// (byte - OFF) * scale for bytes 2 H, 2 H + 1 of u
template <int H> __device__ __forceinline__ uint64_t scaled_pair(uint32_t u, uint64_t neg_off, uint64_t scale) {
    return mul_f32x2(add_f32x2(magic_pair<H>(u), neg_off), scale);
}
// Where a decoder puts its 64 weights, two f32 at a time: rounded to bf16 pairs, or kept as they are (PRECISE).
template <bool PRECISE> struct GemmOut {
    uint32_t hi[32];
    __device__ __forceinline__ void put(int i, uint64_t pair) { hi[i] = bf16x2_of(pair); }
};
// An f32 weight is the sum of three bf16 values: the upper half of its bits, of what that leaves behind, and of what is
// left then, all of it exact (one byte-permute per pair and part; a conversion instruction would pace the decoder).
// Q4_0's weights (f16 scale times four bits: 15) are two such parts, and so are re-laid Q6_K's without the
// super-block's scale (sub-block scale times six bits: 13), which is left to the epilogue (gemm_late_scale).
constexpr bool gemm_late_scale(uint32_t scheme) { return scheme == kQ6Wide; }
constexpr uint32_t gemm_weight_parts(uint32_t scheme) { return scheme == RLXQ_Q4_0 || gemm_late_scale(scheme) ? 2u : 3u; }
template <> struct GemmOut<true> {
    uint64_t f[32];
    __device__ __forceinline__ void put(int i, uint64_t pair) { f[i] = pair; }
    __device__ __forceinline__ void part(uint32_t (&p)[32]) {          // the next part
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            uint32_t a, b;
            asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(f[i]));
            p[i] = __byte_perm(a, b, 0x7632);
            f[i] = add_f32x2(f[i], f32x2((a & 0xFFFF0000u) ^ 0x80000000u, (b & 0xFFFF0000u) ^ 0x80000000u));
        }
    }
};

// Weights without a scale of their group, as two bf16 parts that the decoder forms itself, 32 at a time.
struct GemmOutTwo { uint32_t hi[16], lo[16]; };
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
template <uint32_t SCHEME, int S> struct Decode64;

// Words of a row buffer at compile-time byte offsets: loads the 16-byte chunks covering [B0, B0 + LEN)
// and hands out the 32-bit little-endian word at any even byte offset inside.
template <int B0, int LEN> struct Span {
    static constexpr int C0 = B0 / 16, C1 = (B0 + LEN + 15) / 16;
    uint32_t w[4 * (C1 - C0) + 1];
    __device__ __forceinline__ void load(const uint8_t* row) {
#pragma unroll
        for (int c = C0; c < C1; ++c) {
            const uint4 t = *reinterpret_cast<const uint4*>(row + 16 * c);
            w[4 * (c - C0)] = t.x; w[4 * (c - C0) + 1] = t.y; w[4 * (c - C0) + 2] = t.z; w[4 * (c - C0) + 3] = t.w;
        }
        w[4 * (C1 - C0)] = 0;
    }
    template <int B> __device__ __forceinline__ uint32_t word() const {
        constexpr int rel = B - 16 * C0;
        if (rel % 4 == 0) return w[rel / 4];
        return __funnelshift_r(w[rel / 4], w[rel / 4 + 1], 16);
    }
};

// Words [0, N) behind byte `off` (even, below 16) of the 16-byte aligned row piece p: the chunks that cover them, moved by
// whole words where bits 2 and 3 of off say so and by half a word where bit 1 does.  The offset stays a run-time value: one
// copy of the decoder instead of one per offset, whose eight copies did not stay in the instruction cache.
template <int N> __device__ __forceinline__ void words_at(const uint8_t* p, uint32_t off, uint32_t (&q)[N]) {
    constexpr int C = (4 * N + 14 + 15) / 16;
    uint32_t w[4 * C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const uint4 t = *reinterpret_cast<const uint4*>(p + 16 * c);
        w[4 * c] = t.x; w[4 * c + 1] = t.y; w[4 * c + 2] = t.z; w[4 * c + 3] = t.w;
    }
    const bool one = off & 4u, two = off & 8u;
    const uint32_t sh = (off & 2u) * 8u;
#pragma unroll
    for (int i = 0; i + 1 < 4 * C; ++i) w[i] = one ? w[i + 1] : w[i];
#pragma unroll
    for (int i = 0; i + 2 < 4 * C; ++i) w[i] = two ? w[i + 2] : w[i];
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = __funnelshift_r(w[i], w[i + 1], sh);
}

// Q6_K: ql[128] | qh[64] | sc[16] (i8) | d (f16), element order as rlx-gguf/src/lib.rs:1070-1114.  Half h (128 weights)
// reads 64 bytes of ql and 32 of qh; its part p takes the low (p = 0) or high nibbles and two bits of qh for two
// interleaved 32-weight groups, so both parts come from the same words.  Group g of a row starts at byte 210 g, `off` =
// 210 g mod 16 behind the start of the row's 240-byte buffer.
struct Q6Half {
    uint32_t ql[16], qh[8], sc[2];
    float d;
    __device__ __forceinline__ void load(const uint8_t* row, uint32_t off, uint32_t h) {
        words_at<16>(row + 64 * h, off, ql);
        words_at<8>(row + 128 + 32 * h, off, qh);
        uint32_t tail[5];                                                 // sc[16], d
        words_at<5>(row + 192, off, tail);
        sc[0] = h ? tail[2] : tail[0];
        sc[1] = h ? tail[3] : tail[1];
        d = f16_bits_to_f32(tail[4] & 0xFFFFu);
    }
    template <typename Out> __device__ __forceinline__ void decode(uint32_t part, Out& v) const {
        const uint64_t off = f32x2_splat(-(8388608.0f + 32.0f));
        const uint32_t scw = part ? sc[1] : sc[0];
#pragma unroll
        for (int gsel = 0; gsel < 2; ++gsel) {
            // int8 -> (s + 128) unsigned -> float, minus 128
            const float s0 = d * u8_minus<128>(((scw >> (16 * gsel)) & 0xFFu) ^ 0x80u), s1 = d * u8_minus<128>(((scw >> (16 * gsel + 8)) & 0xFFu) ^ 0x80u);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t ds = f32x2_splat(i < 4 ? s0 : s1);
                const uint32_t lo = (ql[8 * gsel + i] >> (4 * part)) & 0x0F0F0F0Fu;
                const uint32_t hi = ((qh[i] >> (4 * part)) << (4 - 2 * gsel)) & 0x30303030u;
                v.put(16 * gsel + 2 * i, scaled_pair<0>(lo | hi, off, ds));
                v.put(16 * gsel + 2 * i + 1, scaled_pair<1>(lo | hi, off, ds));
            }
        }
    }
};
// Q2_K as the reference reads it (rlx-gguf/src/lib.rs:857-886): d, dmin (f16) | 16 scale bytes (low nibble scale,
// high nibble min) | 64 quant bytes.  Weights [64 S, 64 S + 64) are two 2-bit planes (shift 4 (S % 2), + 2) of the
// 32 quant bytes of half S / 2, sixteen weights per scale byte: w = (d * sc) * q - dmin * mn, product and
// difference rounded separately.  O = byte offset of the super-block in the row buffer (a multiple of 4).
template <int S, int O> struct Decode64Q2 {
    template <typename Out> __device__ static __forceinline__ void run(const uint8_t* row, Out& v) {
        constexpr int h = S / 2;
        Span<O, 4> hd;
        Span<O + 4 + 8 * h + 4 * (S % 2), 4> sc;
        Span<O + 20 + 32 * h, 32> qs;
        hd.load(row); sc.load(row); qs.load(row);
        const uint32_t hw = hd.template word<O>();
        const float d = f16_bits_to_f32(hw & 0xFFFFu), dmin = f16_bits_to_f32(hw >> 16);
        const uint32_t scw = sc.template word<O + 4 + 8 * h + 4 * (S % 2)>();    // scale bytes of (plane, sixteen) = (0,0) (0,1) (1,0) (1,1)
        const uint64_t off = f32x2_splat(-8388608.0f);
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
            const int shift = 4 * (S % 2) + 2 * pl;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t sb = (scw >> (16 * pl + 8 * (i >> 2))) & 0xFFu;
                const uint64_t dl2 = f32x2_splat(d * (float)(sb & 0xFu)), ml2 = f32x2_splat(-(dmin * (float)(sb >> 4)));
                const uint32_t q = (word_at(qs, i) >> shift) & 0x03030303u;
                v.put(16 * pl + 2 * i, add_f32x2(mul_f32x2(dl2, add_f32x2(magic_pair<0>(q), off)), ml2));
                v.put(16 * pl + 2 * i + 1, add_f32x2(mul_f32x2(dl2, add_f32x2(magic_pair<1>(q), off)), ml2));
            }
        }
    }
    __device__ static __forceinline__ uint32_t word_at(const Span<O + 20 + 32 * (S / 2), 32>& qs, int i) {
        constexpr int base = O + 20 + 32 * (S / 2);
        switch (i) {
            case 0: return qs.template word<base>();      case 1: return qs.template word<base + 4>();
            case 2: return qs.template word<base + 8>();  case 3: return qs.template word<base + 12>();
            case 4: return qs.template word<base + 16>(); case 5: return qs.template word<base + 20>();
            case 6: return qs.template word<base + 24>(); default: return qs.template word<base + 28>();
        }
    }
};
template <int S, typename Out>
__device__ __forceinline__ void decode64_q2(const uint8_t* row, uint32_t g, Out& v) {
    switch (g & 3u) {      // 84 g mod 16 = 4 (g mod 4)
        case 0: Decode64Q2<S, 0>::run(row, v); break;   case 1: Decode64Q2<S, 4>::run(row, v); break;
        case 2: Decode64Q2<S, 8>::run(row, v); break;   default: Decode64Q2<S, 12>::run(row, v); break;
    }
}

// The 32-bit word at even byte offset `rel` of a word array (offsets are constants once the loops are unrolled).
__device__ __forceinline__ uint32_t word_of(const uint32_t* w, int rel) {
    return (rel % 4 == 0) ? w[rel / 4] : __funnelshift_r(w[rel / 4], w[rel / 4 + 1], 16);
}
// four bits -> bit 0 of four bytes
__device__ __forceinline__ uint32_t spread4(uint32_t x) { return ((x & 0xFu) * 0x00204081u) & 0x01010101u; }

// Q4_1 / Q5_0 / Q5_1 (rlx-gguf/src/lib.rs:635-729): blocks of 32 weights, d (f16) [m (f16)] [qh (u32)] 16 nibble
// bytes; low nibbles are weights 0..15, high nibbles 16..31, bit j (j + 16) of qh the fifth bit of weight j (16 + j).
// Q4_1, Q5_1: d * q + m (product and sum rounded separately); Q5_0: d * (q - 16).
template <int S, int BB, bool HAS_M, bool HAS_H> struct Decode64Blk32 {
    template <typename Out> __device__ static __forceinline__ void run(const uint8_t* row, Out& v) {
        constexpr int B0 = 2 * BB * S;
        Span<B0, 2 * BB> sp;
        sp.load(row);
        constexpr int R0 = B0 - 16 * Span<B0, 2 * BB>::C0;
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
            const int base = R0 + BB * blk;
            const uint32_t hw = word_of(sp.w, base);
            const uint64_t d2 = f32x2_splat(f16_bits_to_f32(hw & 0xFFFFu));
            const uint64_t m2 = HAS_M ? f32x2_splat(f16_bits_to_f32(hw >> 16)) : 0ull;
            const int oh = HAS_M ? 4 : 2, oq = oh + (HAS_H ? 4 : 0);
            const uint32_t qh = HAS_H ? word_of(sp.w, base + oh) : 0u;
            const uint64_t off = f32x2_splat(HAS_M ? -8388608.0f : -(8388608.0f + 16.0f));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t q = word_of(sp.w, base + oq + 4 * i);
                uint32_t lo = q & 0x0F0F0F0Fu, hi = (q >> 4) & 0x0F0F0F0Fu;
                if (HAS_H) { lo |= spread4(qh >> (4 * i)) << 4; hi |= spread4(qh >> (16 + 4 * i)) << 4; }
                if (HAS_M) {
                    v.put(16 * blk + 2 * i, add_f32x2(mul_f32x2(d2, add_f32x2(magic_pair<0>(lo), off)), m2));
                    v.put(16 * blk + 2 * i + 1, add_f32x2(mul_f32x2(d2, add_f32x2(magic_pair<1>(lo), off)), m2));
                    v.put(16 * blk + 8 + 2 * i, add_f32x2(mul_f32x2(d2, add_f32x2(magic_pair<0>(hi), off)), m2));
                    v.put(16 * blk + 8 + 2 * i + 1, add_f32x2(mul_f32x2(d2, add_f32x2(magic_pair<1>(hi), off)), m2));
                } else {
                    v.put(16 * blk + 2 * i, scaled_pair<0>(lo, off, d2));
                    v.put(16 * blk + 2 * i + 1, scaled_pair<1>(lo, off, d2));
                    v.put(16 * blk + 8 + 2 * i, scaled_pair<0>(hi, off, d2));
                    v.put(16 * blk + 8 + 2 * i + 1, scaled_pair<1>(hi, off, d2));
                }
            }
        }
    }
};
template <int S> struct Decode64<RLXQ_Q4_1, S> : Decode64Blk32<S, 20, true, false> {};
template <int S> struct Decode64<RLXQ_Q5_0, S> : Decode64Blk32<S, 22, false, true> {};
template <int S> struct Decode64<RLXQ_Q5_1, S> : Decode64Blk32<S, 24, true, true> {};

// Q8_K (rlx-gguf/src/lib.rs:848-854, 1121-1140): w = d * q with an f32 d.
template <int S, int O> struct Decode64Q8K {
    template <typename Out> __device__ static __forceinline__ void run(const uint8_t* row, Out& v) {
        Span<O, 4> hd;
        Span<O + 4 + 64 * S, 64> qs;
        hd.load(row); qs.load(row);
        const uint64_t d2 = f32x2_splat(__uint_as_float(hd.template word<O>())), off = f32x2_splat(-(8388608.0f + 128.0f));
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t u = qs.w[(O + 4 + 64 * S) / 4 - 4 * Span<O + 4 + 64 * S, 64>::C0 + i] ^ 0x80808080u;   // int8 -> q + 128
            v.put(2 * i, scaled_pair<0>(u, off, d2));
            v.put(2 * i + 1, scaled_pair<1>(u, off, d2));
        }
    }
};
template <int S, typename Out>
__device__ __forceinline__ void decode64_q8k(const uint8_t* row, uint32_t g, Out& v) {
    switch (g & 3u) {      // 292 g mod 16 = 4 (g mod 4)
        case 0: Decode64Q8K<S, 0>::run(row, v); break;   case 1: Decode64Q8K<S, 4>::run(row, v); break;
        case 2: Decode64Q8K<S, 8>::run(row, v); break;   default: Decode64Q8K<S, 12>::run(row, v); break;
    }
}

// Q3_K as the reference reads it (rlx-gguf/src/lib.rs:889-930): d (f16) | 12 scale bytes (sixteen 6-bit scales) |
// 32 high-mask bytes | 64 quant bytes.  Weights [64 S, 64 S + 64): planes 2 (S % 2), + 1 of the 32 quant bytes of
// half S / 2; weight = (d * (scale - 32)) * (q - (mask bit ? 0 : 4)), mask bit 4 (S / 2) + plane of the weight's
// mask byte.  The four scales of the group are the bytes of word S of the unpacked scale words.
template <int S, int O> struct Decode64Q3 {
    template <typename Out> __device__ static __forceinline__ void run(const uint8_t* row, Out& v) {
        constexpr int h = S / 2;
        Span<O, 14> hd;
        Span<O + 14, 32> hm;
        Span<O + 46 + 32 * h, 32> qs;
        hd.load(row); hm.load(row); qs.load(row);
        const float d = f16_bits_to_f32(hd.template word<O>() & 0xFFFFu);
        const uint32_t a0 = hd.template word<O + 2>(), a1 = hd.template word<O + 6>(), tmp = hd.template word<O + 10>();
        uint32_t scw;
        if (S == 0) scw = (a0 & 0x0F0F0F0Fu) | ((tmp & 0x03030303u) << 4);
        else if (S == 1) scw = (a1 & 0x0F0F0F0Fu) | (((tmp >> 2) & 0x03030303u) << 4);
        else if (S == 2) scw = ((a0 >> 4) & 0x0F0F0F0Fu) | (((tmp >> 4) & 0x03030303u) << 4);
        else scw = ((a1 >> 4) & 0x0F0F0F0Fu) | (((tmp >> 6) & 0x03030303u) << 4);
        const uint64_t off = f32x2_splat(-(8388608.0f + 4.0f));
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
            const int plane = 2 * (S % 2) + pl;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int sb = (int)((scw >> (16 * pl + 8 * (i >> 2))) & 0xFFu) - 32;
                const uint64_t dl2 = f32x2_splat(d * (float)sb);
                const uint32_t q = (word_q(qs, i) >> (2 * plane)) & 0x03030303u;
                const uint32_t hb = (word_h(hm, i) >> (4 * h + plane)) & 0x01010101u;
                const uint32_t u = q | (hb << 2);                 // q + 4 where the mask bit is set: weight = u - 4
                v.put(16 * pl + 2 * i, scaled_pair<0>(u, off, dl2));
                v.put(16 * pl + 2 * i + 1, scaled_pair<1>(u, off, dl2));
            }
        }
    }
    __device__ static __forceinline__ uint32_t word_q(const Span<O + 46 + 32 * (S / 2), 32>& qs, int i) {
        constexpr int base = O + 46 + 32 * (S / 2);
        switch (i) {
            case 0: return qs.template word<base>();      case 1: return qs.template word<base + 4>();
            case 2: return qs.template word<base + 8>();  case 3: return qs.template word<base + 12>();
            case 4: return qs.template word<base + 16>(); case 5: return qs.template word<base + 20>();
            case 6: return qs.template word<base + 24>(); default: return qs.template word<base + 28>();
        }
    }
    __device__ static __forceinline__ uint32_t word_h(const Span<O + 14, 32>& hm, int i) {
        constexpr int base = O + 14;
        switch (i) {
            case 0: return hm.template word<base>();      case 1: return hm.template word<base + 4>();
            case 2: return hm.template word<base + 8>();  case 3: return hm.template word<base + 12>();
            case 4: return hm.template word<base + 16>(); case 5: return hm.template word<base + 20>();
            case 6: return hm.template word<base + 24>(); default: return hm.template word<base + 28>();
        }
    }
};
template <int S, typename Out>
__device__ __forceinline__ void decode64_q3(const uint8_t* row, uint32_t g, Out& v) {
    switch (g & 7u) {      // 110 g mod 16 = (16 - 2 (g mod 8)) mod 16
        case 0: Decode64Q3<S, 0>::run(row, v); break;   case 1: Decode64Q3<S, 14>::run(row, v); break;
        case 2: Decode64Q3<S, 12>::run(row, v); break;  case 3: Decode64Q3<S, 10>::run(row, v); break;
        case 4: Decode64Q3<S, 8>::run(row, v); break;   case 5: Decode64Q3<S, 6>::run(row, v); break;
        case 6: Decode64Q3<S, 4>::run(row, v); break;   default: Decode64Q3<S, 2>::run(row, v); break;
    }
}

template <uint32_t SCHEME, int S, typename Out>
__device__ __forceinline__ void decode64(const uint8_t* row, uint32_t g, Out& v) {
    if constexpr (SCHEME == RLXQ_Q2_K) decode64_q2<S>(row, g, v);
    else if constexpr (SCHEME == RLXQ_Q8_K) decode64_q8k<S>(row, g, v);
    else if constexpr (SCHEME == RLXQ_Q3_K) decode64_q3<S>(row, g, v);
    else Decode64<SCHEME, S>::run(row, v);
}

// ---- one 64-weight part, its number known at run time -------------------------------------------
// The decode warps run a loop over parts whose body exists once (Q4_K, Q5_K, Q6_K) or once per warp group (the 32-weight
// formats, whose odd parts start one word later): four unrolled copies of 250 instructions left a quarter of the decode
// warps' time to instruction fetch.  The other formats keep unrolled copies (Decode64).
constexpr bool gemm_part_loop(uint32_t scheme) {
    return scheme == RLXQ_Q4_0 || scheme == RLXQ_Q8_0 || scheme == RLXQ_Q4_K || scheme == RLXQ_Q5_K || scheme == RLXQ_Q6_K || scheme == kQ6Wide;
}
// Words [0, N) from word GRP + 2 * high on of the chunks at p.
template <int N, uint32_t GRP> __device__ __forceinline__ void words_from(const uint8_t* p, bool high, uint32_t (&q)[N]) {
    constexpr int C = (N + 3 + 3) / 4;
    uint32_t w[4 * C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const uint4 t = *reinterpret_cast<const uint4*>(p + 16 * c);
        w[4 * c] = t.x; w[4 * c + 1] = t.y; w[4 * c + 2] = t.z; w[4 * c + 3] = t.w;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = high ? w[i + GRP + 2] : w[i + GRP];
}
// Q4_0 and Q8_0: part S = GRP + 2 p, blocks 2 S and 2 S + 1.  The first starts on a word (d, quants two bytes on), the second
// two bytes into one (d in its upper half, quants aligned behind it).
template <uint32_t SCHEME, uint32_t GRP, typename Out>
__device__ __forceinline__ void decode_blocks32(const uint8_t* row, uint32_t p, Out& v) {
    constexpr int QW = SCHEME == RLXQ_Q4_0 ? 4 : 8, N = 2 * QW + 1;
    constexpr uint32_t STEP = SCHEME == RLXQ_Q4_0 ? 32 : 64;              // 36 S or 68 S, less the S words
    uint32_t w[N];
    words_from<N, GRP>(row + STEP * (GRP + 2 * p), p != 0, w);
#pragma unroll
    for (int blk = 0; blk < 2; ++blk) {
        const uint32_t dbits = blk == 0 ? w[0] & 0xFFFFu : w[QW] >> 16;
        const uint64_t d2 = f32x2_splat(f16_bits_to_f32(dbits));
        const uint64_t off = f32x2_splat(-(8388608.0f + (SCHEME == RLXQ_Q4_0 ? 8.0f : 128.0f)));
#pragma unroll
        for (int i = 0; i < QW; ++i) {
            const uint32_t q = blk == 0 ? __funnelshift_r(w[i], w[i + 1], 16) : w[QW + 1 + i];
            if (SCHEME == RLXQ_Q4_0) {       // weights 4i..: low nibbles; 16 + 4i..: high nibbles
                const uint32_t lo = q & 0x0F0F0F0Fu, hi = (q >> 4) & 0x0F0F0F0Fu;
                v.put(16 * blk + 2 * i, scaled_pair<0>(lo, off, d2));
                v.put(16 * blk + 2 * i + 1, scaled_pair<1>(lo, off, d2));
                v.put(16 * blk + 8 + 2 * i, scaled_pair<0>(hi, off, d2));
                v.put(16 * blk + 8 + 2 * i + 1, scaled_pair<1>(hi, off, d2));
            } else {                         // int8 -> (q + 128) unsigned -> float, minus 128
                const uint32_t u = q ^ 0x80808080u;
                v.put(16 * blk + 2 * i, scaled_pair<0>(u, off, d2));
                v.put(16 * blk + 2 * i + 1, scaled_pair<1>(u, off, d2));
            }
        }
    }
}
// Q4_K and Q5_K: part S, sub-blocks 2 S (low nibbles) and 2 S + 1 (high nibbles) of 32 bytes; bit j of qh[l] adds 16 to
// weight l of sub-block j (Q5_K).
template <uint32_t SCHEME, typename Out>
__device__ __forceinline__ void decode_k45(const uint8_t* row, uint32_t S, Out& v) {
    constexpr bool FIVE = SCHEME == RLXQ_Q5_K;
    const uint4 hd = *reinterpret_cast<const uint4*>(row);   // d, dmin, 12 scale bytes
    const uint8_t* qp = row + (FIVE ? 48 : 16) + 32 * S;
    const uint4 a = *reinterpret_cast<const uint4*>(qp), b = *reinterpret_cast<const uint4*>(qp + 16);
    const uint32_t qs[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t qh[8];
    if (FIVE) {
        const uint4 ha = *reinterpret_cast<const uint4*>(row + 16), hb = *reinterpret_cast<const uint4*>(row + 32);
        qh[0] = ha.x; qh[1] = ha.y; qh[2] = ha.z; qh[3] = ha.w; qh[4] = hb.x; qh[5] = hb.y; qh[6] = hb.z; qh[7] = hb.w;
    }
    const bool upper = S >= 2;
    const uint32_t scb = upper ? (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u) : hd.y & 0x3F3F3F3Fu;
    const uint32_t mnb = upper ? ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u) : hd.z & 0x3F3F3F3Fu;
    const uint32_t sc = scb >> (16 * (S & 1u)), mn = mnb >> (16 * (S & 1u));
    const float d = f16_bits_to_f32(hd.x & 0xFFFFu), dmin = f16_bits_to_f32(hd.x >> 16);
    const float dl = d * u8_to_f32(sc & 0xFFu), ml = dmin * u8_to_f32(mn & 0xFFu);
    const float dh = d * u8_to_f32((sc >> 8) & 0xFFu), mh = dmin * u8_to_f32((mn >> 8) & 0xFFu);
    const uint64_t off = f32x2_splat(-8388608.0f);
    const uint64_t dl2 = f32x2_splat(dl), ml2 = f32x2_splat(-ml), dh2 = f32x2_splat(dh), mh2 = f32x2_splat(-mh);
#pragma unroll
    for (int i = 0; i < 8; ++i) {       // scale * quant - min, rounded after each step as the dequantiser does
        uint32_t lo = qs[i] & 0x0F0F0F0Fu, hi = (qs[i] >> 4) & 0x0F0F0F0Fu;
        if (FIVE) {
            const uint32_t t = qh[i] >> (2 * S);
            lo |= (t << 4) & 0x10101010u;
            hi |= (t << 3) & 0x10101010u;
        }
        v.put(2 * i, add_f32x2(mul_f32x2(dl2, add_f32x2(magic_pair<0>(lo), off)), ml2));
        v.put(2 * i + 1, add_f32x2(mul_f32x2(dl2, add_f32x2(magic_pair<1>(lo), off)), ml2));
        v.put(16 + 2 * i, add_f32x2(mul_f32x2(dh2, add_f32x2(magic_pair<0>(hi), off)), mh2));
        v.put(16 + 2 * i + 1, add_f32x2(mul_f32x2(dh2, add_f32x2(magic_pair<1>(hi), off)), mh2));
    }
}

// Half H of part S of a widened Q6_K row, without d and times 2^-12: sub-block scale (8 bits) times quant (6 bits), rounded to
// bf16, and what the rounding left (4 bits): a product, and a fused multiply-add that takes the rounded one off again, both
// exact.  2^-12 keeps a product within the activation's range.
__device__ __forceinline__ void decode_q6_wide(const uint8_t* row, uint32_t S, int H, GemmOutTwo& v) {
    const uint32_t scw = *reinterpret_cast<const uint16_t*>(row + 256 + 4 * S + 2 * H) ^ 0x8080u;  // int8 -> s + 128
#pragma unroll
    for (int i = 0; i < 2; ++i) {                            // sixteen weights of one scale
        const float f = u8_minus<128>((scw >> (8 * i)) & 0xFFu) * 0x1p-12f;
        const uint32_t s2 = __byte_perm(__float_as_uint(f), 0u, 0x3232);
        const uint4 t = *reinterpret_cast<const uint4*>(row + 64 * S + 32 * H + 16 * i);
        const uint32_t q[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            // 0x43 over a byte below 128 is the bf16 128 + byte; less 160
            const uint32_t w = sub_bf16x2(__byte_perm(q[j / 2], 0x43434343u, j & 1 ? 0x4342 : 0x4140), 0x43204320u);
            const uint32_t r = mul_bf16x2(s2, w);
            v.hi[8 * i + j] = r;
            v.lo[8 * i + j] = fma_bf16x2(s2, w, r ^ 0x80008000u);
        }
    }
}

// ---- kernel -----------------------------------------------------------------------------------
// B TMA, MMA, raw TMA, spare | decode | epilogue.  The block's real size goes into the launch bounds: with two decode
// groups a thread may then use 128 registers, and the decoders keep a row's loads and 32 (PRECISE: 64) results in flight.
constexpr uint32_t gemm_threads(uint32_t groups, uint32_t epilogue = 4) { return (4 + 4 * groups + epilogue) * 32; }
// Epilogue warps: two for each quarter of the rows, half of the tile's columns each, where every fourth block's products have to
// be scaled and added (gemm_late_scale); their decoder fits the 96 registers a thread that leaves.
constexpr uint32_t gemm_epilogue_warps(uint32_t scheme, bool precise) { return precise && gemm_late_scale(scheme) ? 8u : 4u; }
// warp roles: 0 = activation (B) TMA producer, 1 = MMA issuer and tensor-memory owner,
// 2 = raw weight TMA producer, 3 = the second MMA issuer (gemm_late_scale; idle otherwise), then GROUPS x 4 decode warps
// (tensor-memory lane quarter = warp % 4), then 4 (gemm_late_scale: 8) epilogue warps (lane quarter = warp % 4).

struct GemmParams {
    CUtensorMap xmap;      // x[rows, k] bf16, box tx rows x 64 columns, 128-byte swizzle
    CUtensorMap wmap;      // W[n, row_bytes / 8] eight-byte elements, box 128 rows x one 256-weight group
    void* y;
    int* err;
    uint32_t m, n, k, y_bf16, y_vec;      // y_vec: y rows can be written in aligned 16-byte pieces
    uint32_t wtiles, xtiles;
    uint32_t tx;           // activation rows per tile: a multiple of 32, at most 256
    // f32 activations (lo_row != 0): x holds bf16(x) in rows [0, lo_row) and bf16(x - bf16(x)) in the same number of
    // rows behind them; a stage carries both boxes and both are multiplied by the same decoded weights into the same
    // accumulator, so a weight is decoded once for the two halves.
    uint32_t lo_row, xparts;
    // PRECISE: k blocks a main accumulator takes at a time, the accumulator of the lower products, and the sums; powers of two
    // (gemm_main_run).  nmain, ncross: accumulators of either kind, used in turn.
    uint32_t main_run, cross_run, sum_run, nmain, ncross;
    const float* late;      // gemm_late_scale: 2^12 d of the groups of the stack's rows, [k group][row], late_rows rows
    size_t late_rows;
    const uint16_t* x;      // gemm_late_scale: what xmap and wmap describe, for gemm_late_infinite
    const uint8_t* w;
    uint32_t nstages, nraw;               // depth of the operand ring (B in shared memory, A in tensor memory) and of the raw ring
    uint32_t b_bytes;                     // bytes of a B stage: tx * 128, twice that with lo_row
    uint32_t w_late;       // the weights are written by a kernel in front (re-laid rows): read them after the dependency wait
    // Work split.  streamk == 0: CTA c takes whole tiles c, c + grid, ...  streamk == 1: the units
    // (tile, 256-weight k group), tile-major, are dealt as contiguous ranges of units_q units (the first
    // units_r CTAs one more), so every SM gets the same work however many tiles there are; a tile cut
    // by range boundaries is completed by the last of its contributors to arrive (partial tiles in
    // `partial`, one slot per CTA and end of its range).  Arrivals are counted in `counters` under the call's tag
    // (arrival.h), so the words need no zeroing before the call; the last arrival clears its word for a replay of the
    // same launch.
    // slices > 1 (never with streamk): unit (tile, slice) covers an equal part of the tile's k groups and stores its
    // sums to slice `slice` of an f32 array of y's shape (y points at it, slice_elems apart); a kernel behind this one
    // adds the slices in order.
    uint32_t streamk, kgroups, units_q, units_r, slices;
    size_t slice_elems;
    float* partial;
    unsigned long long* counters;
    unsigned long long tag;
    // Grouped mode (MoE expert stacks; null = one dense matrix): W is a stack of [n, k] slabs and activation
    // tile xt is described by groups[1 + xt] = {first row in x, rows, expert, -}: the tile multiplies those rows by slab
    // `expert`.  groups[0].x is the number of tiles.  The table is written on the device by the kernels in front.  Never
    // combined with a k split.  row_map[r]: the row of y that row r of x belongs to.
    const uint4* groups;
    const uint32_t* row_map;
};

// Where tile `tile` reads and writes: activation rows [xrow0, xlim), weight rows from wrow0 (in the stack).
struct GemmTileRows { uint32_t wt, xrow0, xlim, wrow0; };
__device__ __forceinline__ GemmTileRows gemm_tile_rows(const GemmParams& P, uint32_t xtiles, uint32_t tile) {
    GemmTileRows t;
    t.wt = tile / xtiles;
    const uint32_t xt = tile - t.wt * xtiles;
    if (P.groups) {
        const uint4 g = __ldg(&P.groups[1 + xt]);
        t.xrow0 = g.x; t.xlim = g.x + g.y; t.wrow0 = g.z * P.n + t.wt * kGemmTileW;
    } else {
        t.xrow0 = xt * P.tx; t.xlim = min(P.m, t.xrow0 + P.tx); t.wrow0 = t.wt * kGemmTileW;
    }
    return t;
}

struct GemmSeg { uint32_t tile, g0, g1, slice; };     // k groups [g0, g1) of one tile

__device__ __forceinline__ uint32_t gemm_range_start(const GemmParams& P, uint32_t c) {
    return c * P.units_q + min(c, P.units_r);
}
// The CTA whose range holds unit u.
__device__ __forceinline__ uint32_t gemm_owner(const GemmParams& P, uint32_t u) {
    const uint32_t big = P.units_r * (P.units_q + 1);
    return u < big ? u / (P.units_q + 1) : P.units_r + (u - big) / P.units_q;
}
// Iteration over this CTA's segments, in the order every warp role walks them.
__device__ __forceinline__ void gemm_seg_init(const GemmParams& P, uint32_t xtiles, uint32_t& cur, uint32_t& lim) {
    if (P.streamk) { cur = gemm_range_start(P, blockIdx.x); lim = gemm_range_start(P, blockIdx.x + 1); }
    else { cur = blockIdx.x; lim = P.wtiles * xtiles * P.slices; }
}
__device__ __forceinline__ bool gemm_seg_next(const GemmParams& P, uint32_t& cur, uint32_t lim, GemmSeg& sg) {
    if (cur >= lim) return false;
    sg.slice = 0;
    if (P.streamk) {
        sg.tile = cur / P.kgroups;
        sg.g0 = cur - sg.tile * P.kgroups;
        sg.g1 = min(P.kgroups, sg.g0 + (lim - cur));
        cur += sg.g1 - sg.g0;
    } else {
        sg.tile = cur; sg.g0 = 0; sg.g1 = P.kgroups;
        if (P.slices > 1) {
            sg.tile = cur / P.slices;
            sg.slice = cur - sg.tile * P.slices;
            sg.g0 = sg.slice * P.kgroups / P.slices;
            sg.g1 = (sg.slice + 1) * P.kgroups / P.slices;
        }
        cur += gridDim.x;
    }
    return true;
}
// Counts one contributor in and returns how many came before it.  Only the first arrival finds another call's (or
// anybody's) bits in the word and has to install the tag.
__device__ __forceinline__ uint32_t gemm_arrive(unsigned long long* word, unsigned long long tag) {
    unsigned long long old = *reinterpret_cast<volatile unsigned long long*>(word);
    for (;;) {
        if (arrival_count(old, tag)) return arrival_count(atomicAdd(word, 1ull), tag);
        const unsigned long long prev = atomicCAS(word, old, arrival_word(tag, 1u));
        if (prev == old) return 0u;
        old = prev;
    }
}
// Barrier of the epilogue warps that tells all of them whether any thread passed true.
template <uint32_t THREADS = 128> __device__ __forceinline__ bool epilogue_any(bool v) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)v), "n"(THREADS) : "memory");
    return r != 0u;
}

// Where an epilogue pass writes: y (bf16 or f32, row pitch n) or a partial tile (f32, row pitch 128).
struct GemmDst {
    uint8_t* base;
    size_t ld;                        // elements per activation row
    uint32_t m0, mlim, n0, nlim;      // first row / column of the tile in the destination, and its extents
    const uint32_t* map;              // the destination row of activation row r is map[r] (null: r)
};
constexpr uint32_t kGemmEpiStage = 2 * 8192;   // two 8 KB transposition buffers

// Thirty-two accumulator columns (activation rows 32 c ..) of the 128 weight rows -> destination.  A thread
// owns one weight row, so its values lie one destination row apart; written directly, a warp's store is
// 64 or 128 bytes and each thread issues one store per value.  Here the columns are transposed through
// shared memory 8 KB at a time and leave as 16-byte pieces, a warp covering whole 256- or 512-byte row
// segments.  One named barrier per pass: the two buffers alternate, and a thread can only write a
// buffer again after the barrier of the pass in between, which everybody reaches after reading it.
template <bool F32>
__device__ __forceinline__ void gemm_store_vec(uint8_t* stage, uint32_t epi_tid, uint32_t row, const uint32_t (&v)[32],
                                               const GemmDst& d, uint32_t c) {
    constexpr uint32_t ES = F32 ? 4u : 2u, CP = 8192u / (kGemmTileW * ES), PR = kGemmTileW * ES / 16u, NPASS = 32u / CP;
#pragma unroll
    for (uint32_t h = 0; h < NPASS; ++h) {
        uint8_t* buf = stage + ((NPASS == 1u ? c : h) & 1u) * 8192u;
        if (F32) {
#pragma unroll
            for (uint32_t j = 0; j < CP; ++j) *reinterpret_cast<uint32_t*>(buf + (j * kGemmTileW + row) * 4u) = v[h * CP + j];
        } else {
            // one conversion instruction per two values (round to nearest even; a NaN becomes the canonical
            // quiet NaN), the halves stored to the two output rows they belong to
#pragma unroll
            for (uint32_t j = 0; j < CP; j += 2) {
                const uint32_t pr = bf16x2_of(f32x2(v[h * CP + j], v[h * CP + j + 1]));
                *reinterpret_cast<uint16_t*>(buf + (j * kGemmTileW + row) * 2u) = (uint16_t)pr;
                *reinterpret_cast<uint16_t*>(buf + ((j + 1) * kGemmTileW + row) * 2u) = (uint16_t)(pr >> 16);
            }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t p = epi_tid + 128u * q, j = p / PR, pc = p % PR;
            const uint32_t mi = d.m0 + 32u * c + h * CP + j, ni = d.n0 + pc * (16u / ES);
            if (mi < d.mlim && ni < d.nlim) {
                const uint4 t = *reinterpret_cast<const uint4*>(buf + j * (kGemmTileW * ES) + pc * 16u);
                *reinterpret_cast<uint4*>(d.base + ((size_t)(d.map ? __ldg(d.map + mi) : mi) * d.ld + ni) * ES) = t;
            }
        }
    }
}

// Four values of activation row mi, weight rows ni .. ni + 3, into y.
__device__ __forceinline__ void gemm_store4(const GemmParams& P, uint32_t mi, uint32_t ni, float4 a) {
    if (mi >= P.m || ni >= P.n) return;
    const size_t o = (size_t)mi * P.n + ni;
    if (P.y_vec) {                       // n is a multiple of 4 at least and the rows are aligned
        if (P.y_bf16) {
            uint2 t;
            t.x = bf16x2_of(f32x2(__float_as_uint(a.x), __float_as_uint(a.y)));
            t.y = bf16x2_of(f32x2(__float_as_uint(a.z), __float_as_uint(a.w)));
            *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(P.y) + o) = t;
        } else {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(P.y) + o) = a;
        }
        return;
    }
    const float e[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        if (ni + i < P.n) {
            if (P.y_bf16) reinterpret_cast<uint16_t*>(P.y)[o + i] = (uint16_t)bf16x2_of(f32x2(__float_as_uint(e[i]), 0u));
            else reinterpret_cast<float*>(P.y)[o + i] = e[i];
        }
    }
}

// Thirty-two accumulator columns plus the same columns of another contributor's published part -> y.  The
// other part's 16-byte pieces follow the piece order of the transposition buffers: piece p of a 16-column
// pass is floats [4 p, 4 p + 4) of that pass, in the buffer and in the part alike.
__device__ __forceinline__ void gemm_add_store(uint8_t* stage, uint32_t epi_tid, uint32_t row, const uint32_t (&v)[32],
                                               const uint4* other, const GemmParams& P, uint32_t m0, uint32_t n0) {
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        uint8_t* buf = stage + h * 8192u;
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) *reinterpret_cast<uint32_t*>(buf + (j * kGemmTileW + row) * 4u) = v[16 * h + j];
        asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t p = epi_tid + 128u * q;
            const float4 own = *reinterpret_cast<const float4*>(buf + p * 16u);
            const uint4 ot = __ldcg(other + 512u * h + p);
            float4 r;
            r.x = own.x + __uint_as_float(ot.x); r.y = own.y + __uint_as_float(ot.y);
            r.z = own.z + __uint_as_float(ot.z); r.w = own.w + __uint_as_float(ot.w);
            gemm_store4(P, m0 + 16 * h + (p >> 5), n0 + 4 * (p & 31u), r);
        }
    }
}

// The last contributor of a cut tile adds all parts in contributor order (its own included, re-read from
// memory: the sum then never depends on who came last).  Sixteen activation rows (8 KB of every part) at a
// time, in 16-byte pieces: a warp reads 512 contiguous bytes of each part.  Kept out of line: it runs once
// per cut tile and would otherwise raise the register need of the whole kernel.
__device__ __noinline__ void gemm_reduce_parts(const GemmParams& P, uint32_t tile_x, uint32_t c_first, uint32_t c_last,
                                               uint32_t u0, uint32_t m0, uint32_t n0, uint32_t epi_tid) {
    for (uint32_t col0 = 0; col0 < tile_x && m0 + col0 < P.m; col0 += 16) {
        float4 acc[4];
        for (uint32_t cc = c_first; cc <= c_last; ++cc) {
            const uint32_t sid = 2 * cc + (gemm_range_start(P, cc) > u0 ? 0u : 1u);
            const uint4* src = reinterpret_cast<const uint4*>(P.partial + (size_t)sid * (kGemmTileW * tile_x) + (size_t)col0 * kGemmTileW) + epi_tid;
            uint4 pv[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) pv[q] = __ldcg(src + 128u * q);
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const float4 f = make_float4(__uint_as_float(pv[q].x), __uint_as_float(pv[q].y), __uint_as_float(pv[q].z), __uint_as_float(pv[q].w));
                if (cc == c_first) acc[q] = f;
                else { acc[q].x += f.x; acc[q].y += f.y; acc[q].z += f.z; acc[q].w += f.w; }
            }
        }
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t p = epi_tid + 128u * q;
            gemm_store4(P, m0 + col0 + (p >> 5), n0 + 4 * (p & 31u), acc[q]);
        }
    }
}

// tensor-memory columns of a weight stage
constexpr uint32_t gemm_a_cols(uint32_t scheme, bool precise) { return precise ? 32u * gemm_weight_parts(scheme) : 32u; }

struct GemmBars {
    // full: a stage's activations (their bytes) and its weights (four decode warps) are there: one barrier to look at for both.
    // (f32 weights in three parts, and Q4_0's in two, have a_full for the weights: with one barrier Q4_0 300 x 11040 x 14336
    // bf16 took 489 us instead of 463, f32 in the mean 3 % less.)
    uint64_t full[kGemmMaxStages], a_full[kGemmMaxStages], stage_free[kGemmMaxStages];
    uint64_t raw_full[kGemmMaxRaw], raw_empty[kGemmMaxRaw];
    uint64_t d_full[4], d_free[4];        // two accumulators (PRECISE: two for the leading product, two for the others)
    uint32_t tmem_base, abort_flag, epi_prev, epi_prev1;   // epi_prev, epi_prev1: arrival counts of alternate segments
};

// One decode warp: raw blocks -> bf16 rows in tensor memory.  The 64-weight parts of the groups are dealt to the decode
// warp groups: of two, group grp takes parts grp and grp + 2 (Q6_K, whose halves share their bytes: 2 grp and 2 grp + 1);
// of three (Q3_K) whoever's turn it is.  GRP = grp where a group has code of its own.
template <uint32_t SCHEME, bool PRECISE, uint32_t GRP>
__device__ __forceinline__ void gemm_decode_role(const GemmParams& P, GemmBars* bars, const uint8_t* raw_stage, uint32_t tmem_a,
                                                 uint32_t xtiles, uint32_t warp, uint32_t lane) {
    constexpr uint32_t RAW_ROW = GemmRaw<SCHEME>::ROW, GROUPS = GemmRaw<SCHEME>::GROUPS;
    constexpr uint32_t RAW_STRIDE = (kGemmTileW * RAW_ROW + 127) / 128 * 128, A_COLS = gemm_a_cols(SCHEME, PRECISE);
    constexpr bool LATE = PRECISE && gemm_late_scale(SCHEME);
    volatile uint32_t* abort_flag = &bars->abort_flag;
    auto give_up = [&](int code) {
        atomicExch(P.err, code);
        *abort_flag = 1u;
    };
    const uint32_t quarter = warp & 3u, grp = (warp - 4) >> 2, NS = P.nstages, NR = P.nraw;
    const uint32_t row = quarter * 32 + lane;                       // weight row of the tile == tensor-memory lane
    const uint32_t lane_addr = (quarter * 32) << 16;
    uint32_t r = 0, rph = 0, turn = 0;   // turn (three groups): whose part comes next
    uint32_t s = 0, fph = 1;             // operand stage of the next part, and the parity that says it is free
    // A part's tensor-memory store is announced when the next one is ready to be stored: its few hundred cycles pass
    // under the next part's arithmetic.
    uint32_t pending = 0;                // the barrier to announce it on (0: nothing stored since)
    auto announce = [&]() {
        if (!pending) return;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pending);
        pending = 0;
    };
    uint32_t cur, lim;
    gemm_seg_init(P, xtiles, cur, lim);
    GemmSeg sg;
    uint32_t raw_ready = 0;              // whether the next raw box had arrived when this group's last part was decoded
    while (!*abort_flag && gemm_seg_next(P, cur, lim, sg)) {
        for (uint32_t g = sg.g0; g < sg.g1; ++g) {
            if (!__all_sync(0xFFFFFFFFu, raw_ready)) {
                announce();
                if (*abort_flag || !mbar_wait(smem_u32(&bars->raw_full[r]), rph)) { give_up(15); return; }
            }
            const uint8_t* rp = raw_stage + r * RAW_STRIDE + row * RAW_ROW;
            // Decoded into registers first: only the store needs the stage's tensor-memory columns, so the arithmetic stays
            // off the free -> store -> MMA chain.
            const uint32_t s0 = s, ph0 = fph;
            s += 4;
            if (s >= NS) { s -= NS; fph ^= 1u; }
            if (PRECISE && s >= NS) { s -= NS; fph ^= 1u; }          // (three stages)
            auto stage_of = [&](uint32_t sub, uint32_t& st, uint32_t& sph) {
                st = s0 + sub;
                sph = ph0;
                if (st >= NS) { st -= NS; sph ^= 1u; }
            };
            using Out = std::conditional_t<LATE, GemmOutTwo[2], GemmOut<PRECISE>>;
            auto store = [&](uint32_t st, uint32_t sph, uint32_t ready, Out& v) -> bool {
                announce();
                if (!__all_sync(0xFFFFFFFFu, ready) && (*abort_flag || !mbar_wait(smem_u32(&bars->stage_free[st]), sph))) { give_up(16); return false; }
                tc_fence_after();
                if constexpr (LATE) {
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {
                        tmem_st16(tmem_a + lane_addr + A_COLS * st + 16 * h, v[h].hi);
                        tmem_st16(tmem_a + lane_addr + A_COLS * st + 32 + 16 * h, v[h].lo);
                    }
                } else if constexpr (PRECISE) {
#pragma unroll
                    for (uint32_t q = 0; q < gemm_weight_parts(SCHEME); ++q) {
                        uint32_t p[32];
                        v.part(p);
                        tmem_st32(tmem_a + lane_addr + A_COLS * st + 32 * q, p);
                    }
                } else {
                    tmem_st32(tmem_a + lane_addr + A_COLS * st, v.hi);
                }
                pending = smem_u32(PRECISE && !LATE ? &bars->a_full[st] : &bars->full[st]);
                return true;
            };
            uint32_t st, sph;
            if constexpr (gemm_part_loop(SCHEME)) {
                Q6Half hf;
                if constexpr (SCHEME == RLXQ_Q6_K) hf.load(rp, (210u * g) & 15u, grp);
#pragma unroll 1
                for (uint32_t p = 0; p < 2; ++p) {
                    const uint32_t sub = SCHEME == RLXQ_Q6_K ? 2 * grp + p : grp + 2 * p;
                    stage_of(sub, st, sph);
                    const uint32_t ready = mbar_test(smem_u32(&bars->stage_free[st]), sph);    // answered while decoding
                    Out v;
                    if constexpr (LATE) { decode_q6_wide(rp, sub, 0, v[0]); decode_q6_wide(rp, sub, 1, v[1]); }
                    else if constexpr (SCHEME == RLXQ_Q6_K) hf.decode(p, v);
                    else if constexpr (SCHEME == RLXQ_Q4_K || SCHEME == RLXQ_Q5_K) decode_k45<SCHEME>(rp, sub, v);
                    else decode_blocks32<SCHEME, GRP>(rp, p, v);
                    if (!store(st, sph, ready, v)) return;
                }
            } else {
#pragma unroll
                for (uint32_t sub = 0; sub < 4; ++sub) {
                    if constexpr (GROUPS == 2) {
                        if (sub % 2 != GRP) continue;
                    } else {
                        const bool mine = turn == grp;
                        if (++turn == GROUPS) turn = 0;
                        if (!mine) continue;
                    }
                    stage_of(sub, st, sph);
                    const uint32_t ready = mbar_test(smem_u32(&bars->stage_free[st]), sph);
                    GemmOut<PRECISE> v;
                    if (sub == 0) decode64<SCHEME, 0>(rp, g, v);
                    else if (sub == 1) decode64<SCHEME, 1>(rp, g, v);
                    else if (sub == 2) decode64<SCHEME, 2>(rp, g, v);
                    else decode64<SCHEME, 3>(rp, g, v);
                    if (!store(st, sph, ready, v)) return;
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->raw_empty[r]));
            if (++r == NR) { r = 0; rph ^= 1u; }
            raw_ready = mbar_test(smem_u32(&bars->raw_full[r]), rph);
        }
    }
    announce();
}

// PRECISE: the weight operand is the f32 weight, as three bf16 parts in three sets of tensor-memory columns, and f32
// activations come as three parts as well (GemmOut; split_hi_lo_kernel).  It serves the shapes whose other kernel multiplies
// f32 weights and activations: three products for bf16 activations, six for f32 ones, where the formats' own path takes one
// and two.
//
// The tensor core truncates where f32 arithmetic rounds, every time it adds to an accumulator, so a long accumulation loses
// a multiple of f32's error (6.8e-6 of a result after 1024 columns of six products in one accumulator, 5.7e-5 after 8192; the
// general kernel, which multiplied these shapes before, 3.3e-7 over 11008).  Hence two accumulators of P.tx columns.  The main
// one takes the leading parts' product of main_run k blocks; the epilogue warps add it, rounding, to sums in registers, while
// the other products run.  Those are 2^-8 of the whole and smaller: they pile up in the second accumulator.  Every sum_run
// blocks it joins the sums, and these move on to totals in shared memory, so that no chain of additions is long.  Error
// against 64 bits, general kernel and this one, f32 activations: k = 256 8.1e-8 and 8.0e-8, 2304 1.6e-7 and 9.8e-8, 11008
// 3.3e-7 and 1.4e-7, 16128 4.0e-7 and 1.5e-7.
// Re-laid Q6_K rows (gemm_late_scale) are multiplied without their super-blocks' scale, as two parts instead of three: five
// products for f32 activations and two for bf16 ones, a decoder of four packed instructions a pair of weights on aligned words,
// and the scale applied by the epilogue warps, eight of them, as they add a super-block's sums.  Two threads issue MMAs, for the
// leading product and for the others: beside the products a round of hand-overs takes one thread 0.4 us, whatever else is left
// out (loads, decoding, adding).  Second accumulators of either kind are worth 5 to 9 %.  300 x 11008 x 4096 f32, calls in a graph,
// copy and split included: 223 us with three parts, 172 with two, 187 with aligned rows from a slow first pass, 173 with barriers looked
// at before a round's last MMAs, 148 with two issuers and a faster first pass (167 us a call by itself, its rows in no cache); bf16
// activations and f32 results 188 and 116; 587 x 1280 x 5568 bf16 82 and 50 us, 31 x 13056 x 17990 f32 273 and 210 us.
// Error against 64 bits at k = 11008 1.5e-7 and 1.2e-7.
// Activation rows of a PRECISE tile: what the epilogue threads have registers for (Q3_K's block is larger: 96 a thread) and
// shared memory has room for totals beside three operand stages and two raw boxes (Q8_K's are the largest).
constexpr uint32_t gemm_precise_rows(uint32_t scheme) { return scheme == RLXQ_Q3_K || scheme == RLXQ_Q8_K ? 64u : 96u; }

// Blocks between two emptyings of the main accumulator, and of the sums.  A block costs 1.4e-8 of a result for each of its four
// truncated additions (5.6e-8, 1.0e-7 and 1.9e-7 for runs of 1, 2 and 4), always towards zero, so that the layers of a SwiGLU
// chain add up: held against the general kernel are chains, 2.24e-7 at widths 1024 -> 3328 (here 2.17e-7; 2.22e-7 with f32
// activations), 3.0e-7 at 2304 -> 5888 (2.7e-7), 5.1e-7 at 6912 -> 22272 (4.4e-7).  Shorter runs cost time: 300 x 11040 x 4096 Q8_0
// bf16 takes 220, 236 and 243 us with main runs of 4, 2 and 1, 236, 261 and 300 us with sums of 16, 8 and 4 blocks.
// A result that is stored as bf16 has the error of that rounding, 1.655e-3, the same to six digits with the general kernel and
// with runs of 16 blocks (9e-7 before it is rounded); 300 x 11040 x 4096 Q8_0 bf16 204 us.
static uint32_t gemm_main_run(uint32_t scheme, uint32_t k, bool ybf) {
    const uint32_t most = gemm_late_scale(scheme) ? 4u : 16u;           // (a group's blocks share a scale)
    return std::min(most, ybf ? 16u : k >= 20480 ? 4u : k >= 5632 ? 2u : 1u);
}
static uint32_t gemm_sum_run(uint32_t k, bool ybf) { return ybf || k >= 5632 ? 16u : k >= 2048 ? 8u : 4u; }

// A super-block whose scale is infinite makes infinities of its weights, and NaN of those that are zero.  A sum of weights without
// the scale knows neither the zeros nor the signs, so such a row is multiplied once more, weight by weight: `count` activation rows
// from mi on by row wrow of the stack over the k groups [g0, g1), in f32.  Out of the way of the main loop.
__device__ __noinline__ void gemm_late_infinite(const GemmParams& P, float* total, uint32_t mi, uint32_t rows, uint32_t wrow, uint32_t g0, uint32_t blocks) {
    const uint32_t g1 = g0 + blocks / 4;
    bool infinite = false;
#pragma unroll 1
    for (uint32_t g = g0; g < g1; ++g) infinite |= isinf(P.late[g * P.late_rows + wrow]);
    if (!infinite) return;
#pragma unroll 1
    for (uint32_t i = 0; i < rows; ++i) {
        float sum = 0.f;
#pragma unroll 1
        for (uint32_t g = g0; g < g1; ++g) {
            const float d = P.late[g * P.late_rows + wrow];
            const uint8_t* row = P.w + ((size_t)wrow * P.kgroups + g) * GemmRaw<kQ6Wide>::ROW;
#pragma unroll 1
            for (uint32_t j = 0; j < 256; ++j) {
                const float w = d * (float)(int8_t)row[256 + j / 16] * (float)((int)row[j] - 32) * 0x1p-12f;
                float x = 0.f;                               // the parts' sum: exact
#pragma unroll 1
                for (uint32_t q = 0; q < P.xparts; ++q) x += bf16_bits_to_f32(P.x[((size_t)q * P.lo_row + mi + i) * P.kgroups * 256 + g * 256 + j]);
                sum = fmaf(w, x, sum);
            }
        }
        total[i * kGemmTileW] = sum;
    }
}

// TX = P.tx: no branch between the additions of a block, which are on the chain from one block's product to the next.
template <uint32_t SCHEME, uint32_t TX>
__device__ __forceinline__ void gemm_precise_epilogue(const GemmParams& P, GemmBars* bars, float* total, uint32_t tmem_d,
                                                      uint32_t xtiles, uint32_t warp, uint32_t lane) {
    constexpr bool LATE = gemm_late_scale(SCHEME);
    constexpr uint32_t EW = gemm_epilogue_warps(SCHEME, true), CHUNKS = (TX / 16 + EW / 4 - 1) / (EW / 4);    // chunks of 16 columns of a warp
    const uint32_t quarter = warp & 3u, row = quarter * 32 + lane, epi_tid = (warp - (4 + 4 * GemmRaw<SCHEME>::GROUPS)) * 32 + lane;
    const uint32_t main_d = tmem_d + ((quarter * 32) << 16), cross_d = main_d + TX * (LATE ? P.nmain : 1u), chunk0 = EW == 8 && epi_tid >= 128 ? CHUNKS : 0u;
    uint32_t mph = 0, cph = 0, mb = 0, cb = 0;
    uint32_t cur, lim;
    gemm_seg_init(P, xtiles, cur, lim);
    GemmSeg sg;
    while (gemm_seg_next(P, cur, lim, sg)) {
        GemmTileRows tr = gemm_tile_rows(P, xtiles, sg.tile);
        uint32_t rows = tr.xlim - tr.xrow0;
        const uint32_t blocks = 4 * (sg.g1 - sg.g0);
        auto wait_for = [&](uint32_t d, uint32_t ph) -> bool {
            if (!mbar_wait(smem_u32(&bars->d_full[d]), ph)) {
                atomicExch(P.err, 17);
                *reinterpret_cast<volatile uint32_t*>(&bars->abort_flag) = 1u;
                return false;
            }
            tc_fence_after();
            return true;
        };
        auto release = [&](uint32_t d) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->d_free[d]));
        };
        bool ok = true;
#pragma unroll 1
        for (uint32_t k0 = 0; ok && k0 < blocks; k0 += P.sum_run) {
            uint64_t sum[8 * CHUNKS];                        // pairs of activation rows
#pragma unroll
            for (uint32_t j = 0; j < 8 * CHUNKS; ++j) sum[j] = 0ull;
            uint64_t scale = 0ull;                           // LATE: of the group (2^12 d), twice
            auto add_accumulator = [&](uint32_t acc, bool cross) {
#pragma unroll
                for (uint32_t c = 0; c < CHUNKS; ++c) {
                    if (CHUNKS * (EW / 4) > TX / 16 && chunk0 + c >= TX / 16) break;
                    uint32_t v[16];
                    tmem_ld16(acc + 16 * (chunk0 + c), v);
                    tmem_ld_wait();
                    // An infinite activation times a lower weight part that is zero is a NaN in there.  The main accumulator then
                    // has the infinity (or the NaN) that the product is: its weight part is zero only where the weight is.
                    if (LATE && cross) {
#pragma unroll
                        for (uint32_t j = 0; j < 8; ++j) {
                            const uint64_t p = mul_f32x2(f32x2(v[2 * j], v[2 * j + 1]), scale);
                            asm("mov.b64 {%0, %1}, %2;" : "=r"(v[2 * j]), "=r"(v[2 * j + 1]) : "l"(p));
                        }
                    }
                    if (cross) {
#pragma unroll
                        for (uint32_t j = 0; j < 16; ++j) {
                            float f = fmaxf(__uint_as_float(v[j]), -3.402823466e38f);
                            if (LATE) f = fminf(f, 3.402823466e38f);             // (a rounded weight's second part may have the other sign)
                            v[j] = __float_as_uint(f);
                        }
                    }
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) {
                        if (LATE && !cross) sum[8 * c + j] = fma_f32x2(f32x2(v[2 * j], v[2 * j + 1]), scale, sum[8 * c + j]);
                        else sum[8 * c + j] = add_f32x2(sum[8 * c + j], f32x2(v[2 * j], v[2 * j + 1]));
                    }
                }
            };
            const uint32_t k1 = min(blocks, k0 + P.sum_run);
            // the leading product's runs, then what the other products piled up meanwhile
            // (LATE or not apart: one loop for both kept values alive that cost the others as many spills again)
            if constexpr (LATE) {
#pragma unroll 1
                for (uint32_t kc = k0; ok && kc < k1; kc += P.cross_run) {
                    const uint32_t k2 = min(k1, kc + P.cross_run);
                    scale = f32x2_splat(tr.wt * kGemmTileW + row < P.n ? __ldcg(P.late + (size_t)(sg.g0 + kc / 4) * P.late_rows + tr.wrow0 + row) : 0.f);
#pragma unroll 1
                    for (uint32_t kb = kc; kb < k2; kb += P.main_run) {
                        if (!(ok = wait_for(mb, mph))) break;
                        add_accumulator(main_d + mb * TX, false);
                        release(mb);
                        if (++mb == P.nmain) { mb = 0; mph ^= 1u; }
                    }
                    if (!ok || !(ok = wait_for(2 + cb, cph))) break;
                    add_accumulator(cross_d + cb * TX, true);
                    release(2 + cb);
                    if (++cb == P.ncross) { cb = 0; cph ^= 1u; }
                }
            } else {
#pragma unroll 1
                for (uint32_t kb = k0; kb < k1; kb += P.main_run) {
                    if (!(ok = wait_for(0, mph))) break;
                    mph ^= 1u;
                    add_accumulator(main_d, false);
                    release(0);
                }
                if (!ok || !(ok = wait_for(2, cph))) break;
                cph ^= 1u;
                add_accumulator(cross_d, true);
                release(2);
            }
            if (!ok) break;
            // totals [activation row][weight row]: a thread's own column of them, sixteen loads before the first store
#pragma unroll
            for (uint32_t c = 0; c < CHUNKS; ++c) {
                if (CHUNKS * (EW / 4) > TX / 16 && chunk0 + c >= TX / 16) break;
                float* t = total + 16 * (chunk0 + c) * kGemmTileW + row;
                float old[16];
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) old[j] = k0 ? t[j * kGemmTileW] : 0.f;
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    uint32_t lo, hi;
                    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(sum[8 * c + j]));
                    t[2 * j * kGemmTileW] = old[2 * j] + __uint_as_float(lo);
                    t[(2 * j + 1) * kGemmTileW] = old[2 * j + 1] + __uint_as_float(hi);
                }
            }
        }
        if constexpr (LATE) {                                // worked out again, so that they need no registers up to here
            uint32_t tile = sg.tile;
            asm volatile("" : "+r"(tile));
            tr = gemm_tile_rows(P, xtiles, tile);
            rows = tr.xlim - tr.xrow0;
            // an infinite scale leaves nothing finite in its row
            float* t = total + 16 * chunk0 * kGemmTileW + row;
            if (ok && tr.wt * kGemmTileW + row < P.n && 16 * chunk0 < rows && __builtin_expect(!isfinite(*t), 0))
                gemm_late_infinite(P, t, tr.xrow0 + 16 * chunk0, min(rows - 16 * chunk0, 16 * CHUNKS), tr.wrow0 + row, sg.g0, blocks);
        }
        // the warps leave together: they share the barriers
        if (epilogue_any<32 * EW>(!ok || *reinterpret_cast<volatile uint32_t*>(&bars->abort_flag))) break;
        uint8_t* const out = static_cast<uint8_t*>(P.y) + sg.slice * P.slice_elems * 4;
        const uint32_t n0 = tr.wt * kGemmTileW;
        const uint32_t ps = !P.y_vec ? 7u : P.y_bf16 ? 4u : 5u;      // a row of the tile is 2^ps pieces of 16 bytes, or values
#pragma unroll 4
        for (uint32_t p = epi_tid; p < rows << ps; p += 32 * EW) {
            const uint32_t j = p >> ps, c = (p & ((1u << ps) - 1u)) << (7u - ps), ni = n0 + c, mi = tr.xrow0 + j;
            if (ni >= P.n) continue;
            const size_t o = (size_t)(P.row_map ? __ldg(&P.row_map[mi]) : mi) * P.n + ni;
            const float* t = total + j * kGemmTileW + c;
            if (!P.y_vec) {
                if (P.y_bf16) reinterpret_cast<uint16_t*>(out)[o] = (uint16_t)bf16x2_of(f32x2(__float_as_uint(*t), 0u));
                else reinterpret_cast<float*>(out)[o] = *t;
            } else if (P.y_bf16) {
                const uint4 a = *reinterpret_cast<const uint4*>(t), b = *reinterpret_cast<const uint4*>(t + 4);
                *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out) + o) =
                    make_uint4(bf16x2_of(f32x2(a.x, a.y)), bf16x2_of(f32x2(a.z, a.w)), bf16x2_of(f32x2(b.x, b.y)), bf16x2_of(f32x2(b.z, b.w)));
            } else {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + o) = *reinterpret_cast<const float4*>(t);
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EW) : "memory");       // the totals have been read: the next tile's may be written
    }
}

template <uint32_t SCHEME, bool PRECISE>
__global__ void __launch_bounds__(gemm_threads(GemmRaw<SCHEME>::GROUPS, gemm_epilogue_warps(SCHEME, PRECISE)), 1) gemm_tcgen05_kernel(const __grid_constant__ GemmParams P) {
    constexpr uint32_t RAW_ROW = GemmRaw<SCHEME>::ROW;
    constexpr uint32_t kGemmDecodeGroups = GemmRaw<SCHEME>::GROUPS;
    constexpr uint32_t RAW_BYTES = kGemmTileW * RAW_ROW;
    constexpr uint32_t RAW_STRIDE = (RAW_BYTES + 127) / 128 * 128;
    constexpr uint32_t A_COLS = gemm_a_cols(SCHEME, PRECISE);         // tensor-memory columns of a weight stage
    constexpr bool LATE = PRECISE && gemm_late_scale(SCHEME);         // two MMA issuers
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t NS = P.nstages, NR = P.nraw, B_BYTES = P.b_bytes;
    uint8_t* b_stage = smem;                                          // NS x B_BYTES, 1024-aligned
    uint8_t* raw_stage = smem + NS * B_BYTES;                         // NR x RAW_BYTES (128-aligned)
    GemmBars* bars = reinterpret_cast<GemmBars*>(raw_stage + NR * RAW_STRIDE);
    uint8_t* epi_stage = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(bars + 1) + 15) & ~(uintptr_t)15);

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    volatile uint32_t* abort_flag = &bars->abort_flag;
    griddep_launch_dependents();

    if (tid == 0) {
        for (uint32_t s = 0; s < NS; ++s) {
            mbar_init(smem_u32(&bars->full[s]), PRECISE && !LATE ? 1 : 1 + 4);
            mbar_init(smem_u32(&bars->a_full[s]), 4);
            mbar_init(smem_u32(&bars->stage_free[s]), LATE ? 2 : 1);
        }
        for (uint32_t r = 0; r < NR; ++r) {
            mbar_init(smem_u32(&bars->raw_full[r]), 1);
            mbar_init(smem_u32(&bars->raw_empty[r]), 4 * kGemmDecodeGroups);
        }
        for (uint32_t b = 0; b < 4; ++b) {
            mbar_init(smem_u32(&bars->d_full[b]), 1);
            mbar_init(smem_u32(&bars->d_free[b]), gemm_epilogue_warps(SCHEME, PRECISE));
        }
        bars->abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {               // the whole warp allocates all 512 columns: 256 (PRECISE: nmain + ncross of tx) of accumulators, then weight stages
        tmem_alloc(smem_u32(&bars->tmem_base), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t tmem_d = tmem_base, tmem_a = tmem_base + (PRECISE ? (P.nmain + P.ncross) * P.tx : 256);
    // up to 128 activation rows there are two accumulators: a tile's epilogue runs under the next tile's MMAs
    const uint32_t nacc = P.tx <= 128 ? 2u : 1u;
    auto give_up = [&](int code) {
        atomicExch(P.err, code);
        *abort_flag = 1u;
    };
    // The weights may be requested while the kernel in front still runs; all else that is read from global memory
    // (or written) comes after the dependency wait.  In grouped mode the tile table does, too.
    if (P.groups) griddep_wait();
    // (A plain load: one through the read-only path may be moved up in front of the wait, and read the table before the kernel in
    // front had written it.  The others' addresses depend on this one.)
    const uint32_t xtiles = P.groups ? P.groups[0].x : P.xtiles;

    if (warp == 0) {
        // ---------------- activation tiles (B operand) ----------------
        if (elect_one()) {
            tma_prefetch_desc(&P.xmap);
            griddep_wait();
            uint32_t s = 0, ph = 1;      // parity to wait for on stage_free (1 passes on a fresh barrier)
            uint32_t cur, lim;
            gemm_seg_init(P, xtiles, cur, lim);
            GemmSeg sg;
            bool ok = true;
            while (ok && !*abort_flag && gemm_seg_next(P, cur, lim, sg)) {
                const GemmTileRows tr = gemm_tile_rows(P, xtiles, sg.tile);
                for (uint32_t kb = 4 * sg.g0; kb < 4 * sg.g1; ++kb) {
                    if (*abort_flag || !mbar_wait(smem_u32(&bars->stage_free[s]), ph)) { give_up(11); ok = false; break; }
                    const uint32_t full = smem_u32(&bars->full[s]), dst = smem_u32(b_stage + s * B_BYTES);
                    mbar_arrive_expect_tx(full, B_BYTES);
                    tma_load_2d(dst, &P.xmap, (int32_t)(kb * kGemmBK), (int32_t)tr.xrow0, full);
                    for (uint32_t q = 1; q < P.xparts; ++q)
                        tma_load_2d(dst + q * P.tx * 128u, &P.xmap, (int32_t)(kb * kGemmBK), (int32_t)(q * P.lo_row + tr.xrow0), full);
                    if (++s == NS) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 2) {
        // ---------------- raw weight groups ----------------
        if (elect_one()) {
            tma_prefetch_desc(&P.wmap);
            if (P.w_late) griddep_wait();
            uint32_t r = 0, ph = 1;
            uint32_t cur, lim;
            gemm_seg_init(P, xtiles, cur, lim);
            GemmSeg sg;
            bool ok = true;
            while (ok && !*abort_flag && gemm_seg_next(P, cur, lim, sg)) {
                const GemmTileRows tr = gemm_tile_rows(P, xtiles, sg.tile);
                for (uint32_t g = sg.g0; g < sg.g1; ++g) {
                    if (*abort_flag || !mbar_wait(smem_u32(&bars->raw_empty[r]), ph)) { give_up(12); ok = false; break; }
                    const uint32_t full = smem_u32(&bars->raw_full[r]);
                    mbar_arrive_expect_tx(full, RAW_BYTES);
                    tma_load_2d(smem_u32(raw_stage + r * RAW_STRIDE), &P.wmap, (int32_t)gemm_raw_x<SCHEME>(g), (int32_t)tr.wrow0, full);
                    if (++r == NR) { r = 0; ph ^= 1u; }
                }
            }
        }
    } else if (LATE && (warp == 1 || warp == 3)) {
        // ---------------- MMA issuers: the leading product, and the others ----------------
        // Two threads, because issue is what the rounds are made of: beside the products a round takes 0.4 us of one, whatever
        // else is left out.  They use different accumulators, so neither waits for the other.  (Where a decoder paces the rounds one
        // issuer is faster: with two, Q4_0 300 x 544 x 4096 bf16 takes 33.8 us instead of 28, Q8_0 587 x 2080 x 1024 bf16 48 instead of 42.)
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((P.tx >> 3) << 17) | ((kGemmTileW >> 4) << 24);
            const bool lead = warp == 1;
            const uint32_t run = lead ? P.main_run : P.cross_run, count = lead ? P.nmain : P.ncross, bar0 = lead ? 0u : 2u;
            const uint32_t acc0 = tmem_d + (lead ? 0u : P.nmain * P.tx);
            uint32_t s = 0, ph = 0, d = 0, dph = 1, acc = acc0;        // dph: parity to wait for on d_free (1 passes the first time)
            uint32_t cur, lim;
            gemm_seg_init(P, xtiles, cur, lim);
            GemmSeg sg;
            bool ok = true;
            while (ok && !*abort_flag && gemm_seg_next(P, cur, lim, sg)) {
                const uint32_t blocks = 4 * (sg.g1 - sg.g0);
                // what a round waits for is looked at before the last MMAs of the round in front: an answer takes 118 cycles
                uint32_t ready = mbar_test(smem_u32(&bars->full[s]), ph), free = mbar_test(smem_u32(&bars->d_free[bar0 + d]), dph);
                for (uint32_t kb = 0; kb < blocks; ++kb) {    // the first MMA of a run overwrites the accumulator
                    if (!ready && (*abort_flag || !mbar_wait(smem_u32(&bars->full[s]), ph))) { give_up(14); ok = false; break; }
                    const uint32_t in_run = kb & (run - 1u);
                    if (in_run == 0) {
                        if (!free && (*abort_flag || !mbar_wait(smem_u32(&bars->d_free[bar0 + d]), dph))) { give_up(13); ok = false; break; }
                        acc = acc0 + d * P.tx;
                    }
                    tc_fence_after();
                    const uint32_t sn = s + 1 == NS ? 0u : s + 1, phn = s + 1 == NS ? ph ^ 1u : ph;
                    const bool last = in_run == run - 1u || kb == blocks - 1;
                    const uint32_t dn = !last ? d : d + 1 == count ? 0u : d + 1, dphn = last && d + 1 == count ? dph ^ 1u : dph;
                    const uint64_t bdesc = kmajor_sw128_desc(smem_u32(b_stage + s * B_BYTES));
                    const uint32_t a = tmem_a + A_COLS * s;
                    auto look_ahead = [&] {
                        ready = mbar_test(smem_u32(&bars->full[sn]), phn);
                        if (last) free = mbar_test(smem_u32(&bars->d_free[bar0 + dn]), dphn);
                    };
                    if (lead) {          // weight part 0 by activation part 0
                        look_ahead();
#pragma unroll
                        for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(acc, a + 8 * j, bdesc + 2 * j, idesc, in_run | j ? 1u : 0u);
                    } else {             // parts 1, 2 by part 0, 0..1 by part 1, 0 by part 2; the products left out are below 2^-24 of the whole
                        for (uint32_t q = 1; q < P.xparts; ++q) {
                            const uint64_t ldesc = kmajor_sw128_desc(smem_u32(b_stage + s * B_BYTES + q * P.tx * 128u));
#pragma unroll
                            for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(acc, a + 8 * j, ldesc + 2 * j, idesc, in_run | (q - 1u) | j ? 1u : 0u);
                            if (q == 1) {
#pragma unroll
                                for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(acc, a + 32 + 8 * j, ldesc + 2 * j, idesc, 1u);
                            }
                        }
                        look_ahead();
#pragma unroll
                        for (uint32_t j = 0; j < (gemm_weight_parts(SCHEME) - 1) * (kGemmBK / 16); ++j)
                            tc_mma_ts(acc, a + 32 + 8 * j, bdesc + 2 * (j & 3u), idesc, in_run | (P.xparts - 1u) | j ? 1u : 0u);
                    }
                    if (last) tc_commit(smem_u32(&bars->d_full[bar0 + d]));
                    tc_commit(smem_u32(&bars->stage_free[s]));     // frees the B stage and the A columns when both issuers' MMAs retire
                    d = dn;
                    dph = dphn;
                    s = sn;
                    ph = phn;
                }
            }
        }
    } else if (!LATE && warp == 1) {
        // ---------------- MMA issuer ----------------
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((P.tx >> 3) << 17) | ((kGemmTileW >> 4) << 24);
            uint32_t s = 0, ph = 0, d = 0, dph = 1, cph = 1;   // dph, cph: parities to wait for on d_free (1 passes the first time)
            uint32_t cur, lim;
            gemm_seg_init(P, xtiles, cur, lim);
            GemmSeg sg;
            bool ok = true;
            while (ok && !*abort_flag && gemm_seg_next(P, cur, lim, sg)) {
                const uint32_t blocks = 4 * (sg.g1 - sg.g0);
                if (!PRECISE) {
                    if (!mbar_wait(smem_u32(&bars->d_free[d]), dph)) { give_up(13); break; }
                    tc_fence_after();
                }
                const uint32_t acc = tmem_d + (PRECISE ? 0u : 128u * d);
                uint32_t ready = mbar_test(smem_u32(&bars->full[s]), ph), ra = PRECISE ? mbar_test(smem_u32(&bars->a_full[s]), ph) : 1u;
                for (uint32_t kb = 0; kb < blocks; ++kb) {    // the first MMA of a segment overwrites the accumulator
                    if ((!ready && (*abort_flag || !mbar_wait(smem_u32(&bars->full[s]), ph))) || (PRECISE && !ra && (*abort_flag || !mbar_wait(smem_u32(&bars->a_full[s]), ph)))) { give_up(14); ok = false; break; }
                    tc_fence_after();
                    const uint32_t sn = s + 1 == NS ? 0u : s + 1, phn = s + 1 == NS ? ph ^ 1u : ph;
                    const uint64_t bdesc = kmajor_sw128_desc(smem_u32(b_stage + s * B_BYTES));
                    const uint32_t a = tmem_a + A_COLS * s;
                    if constexpr (PRECISE) {
                        // look at the next stage now: the answer arrives while this stage's MMAs are issued
                        ready = mbar_test(smem_u32(&bars->full[sn]), phn);
                        ra = mbar_test(smem_u32(&bars->a_full[sn]), phn);
                        // weight part 0 by activation part 0, main_run blocks of them in the main accumulator
                        const uint32_t in_run = kb & (P.main_run - 1u);
                        if (in_run == 0) {
                            if (*abort_flag || !mbar_wait(smem_u32(&bars->d_free[0]), dph)) { give_up(13); ok = false; break; }
                            dph ^= 1u;
                            tc_fence_after();
                        }
#pragma unroll
                        for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(acc, a + 8 * j, bdesc + 2 * j, idesc, in_run | j ? 1u : 0u);
                        if (in_run == P.main_run - 1u || kb == blocks - 1) tc_commit(smem_u32(&bars->d_full[0]));
                        // parts 1, 2 by part 0, 0..1 by part 1, 0 by part 2; the products left out are below 2^-24 of the whole
                        const uint32_t cross = acc + P.tx;
                        const bool fresh = (kb & (P.sum_run - 1u)) == 0;
                        if (fresh) {
                            if (*abort_flag || !mbar_wait(smem_u32(&bars->d_free[2]), cph)) { give_up(13); ok = false; break; }
                            cph ^= 1u;
                            tc_fence_after();
                        }
#pragma unroll
                        for (uint32_t j = 0; j < (gemm_weight_parts(SCHEME) - 1) * (kGemmBK / 16); ++j)
                            tc_mma_ts(cross, a + 32 + 8 * j, bdesc + 2 * (j & 3u), idesc, fresh && j == 0 ? 0u : 1u);
                        for (uint32_t q = 1; q < P.xparts; ++q) {
                            const uint64_t ldesc = kmajor_sw128_desc(smem_u32(b_stage + s * B_BYTES + q * P.tx * 128u));
#pragma unroll
                            for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(cross, a + 8 * j, ldesc + 2 * j, idesc, 1u);
                            if (q == 1) {
#pragma unroll
                                for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(cross, a + 32 + 8 * j, ldesc + 2 * j, idesc, 1u);
                            }
                        }
                        if ((kb & (P.sum_run - 1u)) == P.sum_run - 1u || kb == blocks - 1) tc_commit(smem_u32(&bars->d_full[2]));
                    } else {
                        // Upper part of the activations first, as in the paired kernel.  The next stage is looked at before the round's last MMAs
                        // are issued: the answer takes 118 cycles, and arrives meanwhile.
                        if (P.xparts == 1u) ready = mbar_test(smem_u32(&bars->full[sn]), phn);
#pragma unroll
                        for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(acc, a + 8 * j, bdesc + 2 * j, idesc, kb | j ? 1u : 0u);
                        if (P.xparts == 2u) {
                            const uint64_t ldesc = kmajor_sw128_desc(smem_u32(b_stage + s * B_BYTES + P.tx * 128u));
                            ready = mbar_test(smem_u32(&bars->full[sn]), phn);
#pragma unroll
                            for (uint32_t j = 0; j < kGemmBK / 16; ++j) tc_mma_ts(acc, a + 8 * j, ldesc + 2 * j, idesc, 1u);
                        }
                    }
                    tc_commit(smem_u32(&bars->stage_free[s]));     // frees the B stage and the A columns when the MMAs retire
                    s = sn;
                    ph = phn;
                }
                if (!ok) break;
                if (!PRECISE) {
                    tc_commit(smem_u32(&bars->d_full[d]));
                    if (++d == nacc) { d = 0; dph ^= 1u; }
                }
            }
        }
    } else if (warp >= 4 && warp < 4 + 4 * kGemmDecodeGroups) {
        // ---------------- decode ----------------
        constexpr bool ONE = kGemmDecodeGroups != 2 || SCHEME == RLXQ_Q4_K || SCHEME == RLXQ_Q5_K || SCHEME == RLXQ_Q6_K || SCHEME == kQ6Wide;
        if (ONE || warp < 8) gemm_decode_role<SCHEME, PRECISE, 0>(P, bars, raw_stage, tmem_a, xtiles, warp, lane);
        else gemm_decode_role<SCHEME, PRECISE, 1>(P, bars, raw_stage, tmem_a, xtiles, warp, lane);
        tmem_st_wait();                      // (after a timeout a store may still be on its way)
    } else if (PRECISE && warp >= 4 + 4 * kGemmDecodeGroups) {
        // ---------------- epilogue: accumulators -> sums in registers -> totals in shared memory -> y ----------------
        griddep_wait();
        if constexpr (PRECISE) {
            float* total = reinterpret_cast<float*>(epi_stage);
            if (P.tx == 32) gemm_precise_epilogue<SCHEME, 32>(P, bars, total, tmem_d, xtiles, warp, lane);
            else if (P.tx == 64) gemm_precise_epilogue<SCHEME, 64>(P, bars, total, tmem_d, xtiles, warp, lane);
            else if constexpr (gemm_precise_rows(SCHEME) == 96) {
                if (gemm_late_scale(SCHEME) && P.tx == 80) gemm_precise_epilogue<SCHEME, 80>(P, bars, total, tmem_d, xtiles, warp, lane);
                else gemm_precise_epilogue<SCHEME, 96>(P, bars, total, tmem_d, xtiles, warp, lane);
            }
        }
    } else if (!PRECISE && warp >= 4 + 4 * kGemmDecodeGroups) {
        // ---------------- epilogue: accumulator -> y (or -> a partial tile, completed by the last contributor) ----------------
        const uint32_t quarter = warp & 3u;
        const uint32_t lane_addr = (quarter * 32) << 16;
        const uint32_t row = quarter * 32 + lane;
        const uint32_t epi_tid = (warp - (4 + 4 * kGemmDecodeGroups)) * 32 + lane;
        uint32_t d = 0, dph = 0, nseg = 0;
        uint32_t cur, lim;
        gemm_seg_init(P, xtiles, cur, lim);
        GemmSeg sg;
        griddep_wait();                      // y and the workspace may still be in use by the kernel in front
        bool stop = false;                   // the four warps leave together: they share a named barrier
        while (!stop && gemm_seg_next(P, cur, lim, sg)) {
            const GemmTileRows tr = gemm_tile_rows(P, xtiles, sg.tile);
            if (!mbar_wait(smem_u32(&bars->d_full[d]), dph)) { give_up(17); break; }
            tc_fence_after();
            const uint32_t n0 = tr.wt * kGemmTileW, n_idx = n0 + row;
            const bool whole = !P.streamk || (sg.g0 == 0 && sg.g1 == P.kgroups);
            uint8_t* const out = static_cast<uint8_t*>(P.y) + sg.slice * P.slice_elems * 4;
            const uint32_t ncols = (tr.xlim - tr.xrow0 + 31u) / 32u;       // groups of 32 accumulator columns in use
            // a cut tile: this CTA's part goes to its head slot when its range begins inside the tile
            // (only a first segment can), to its tail slot otherwise; layout [activation row][weight row]
            const uint32_t u0 = sg.tile * P.kgroups;
            uint32_t c_first = 0, c_last = 0;
            float* slot = nullptr;
            const float* other = nullptr;     // two contributors and the other one has already published
            if (!whole) {
                slot = P.partial + (size_t)(2 * blockIdx.x + ((nseg == 0 && sg.g0 != 0) ? 0u : 1u)) * (kGemmTileW * P.tx);
                c_first = gemm_owner(P, u0);
                c_last = gemm_owner(P, u0 + P.kgroups - 1);
                if (c_last - c_first == 1u) {
                    // a + b == b + a: with two parts the sum does not depend on who adds, so the second one
                    // to arrive adds the published part to its own registers and never publishes
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (epi_tid == 0) {
                        const unsigned long long word = *reinterpret_cast<volatile unsigned long long*>(&P.counters[sg.tile]);
                        (&bars->epi_prev)[nseg & 1u] = arrival_count(word, P.tag);
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (reinterpret_cast<volatile uint32_t*>(&bars->epi_prev)[nseg & 1u] == 1u) {
                        __threadfence();
                        const uint32_t oc = blockIdx.x == c_first ? c_last : c_first;
                        const uint32_t sid = 2 * oc + (gemm_range_start(P, oc) > u0 ? 0u : 1u);
                        other = P.partial + (size_t)sid * (kGemmTileW * P.tx);
                    }
                }
            }
#pragma unroll 1
            for (uint32_t c = 0; c < ncols; ++c) {
                uint32_t v[32];
                tmem_ld32(tmem_d + 128u * d + lane_addr + 32 * c, v);
                tmem_ld_wait();
                if (c == ncols - 1) {      // everything is in registers: the accumulator may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bars->d_free[d]));
                }
                if (other) {
                    gemm_add_store(epi_stage, epi_tid, row, v, reinterpret_cast<const uint4*>(other + (size_t)(32 * c) * kGemmTileW),
                                   P, tr.xrow0 + 32 * c, n0);
                } else if (!whole) {
                    const GemmDst dst{reinterpret_cast<uint8_t*>(slot), kGemmTileW, 0u, 32u * ncols, 0u, kGemmTileW, nullptr};
                    gemm_store_vec<true>(epi_stage, epi_tid, row, v, dst, c);
                } else if (P.y_vec) {
                    const GemmDst dst{out, P.n, tr.xrow0, tr.xlim, n0, P.n, P.row_map};
                    if (P.y_bf16) gemm_store_vec<false>(epi_stage, epi_tid, row, v, dst, c);
                    else gemm_store_vec<true>(epi_stage, epi_tid, row, v, dst, c);
                } else if (n_idx < P.n) {
#pragma unroll
                    for (uint32_t j = 0; j < 32; ++j) {
                        const uint32_t m_idx = tr.xrow0 + 32 * c + j;
                        if (m_idx < tr.xlim) {
                            const size_t o = (size_t)(P.row_map ? __ldg(&P.row_map[m_idx]) : m_idx) * P.n + n_idx;
                            if (P.y_bf16) reinterpret_cast<uint16_t*>(out)[o] = (uint16_t)bf16x2_of(f32x2(v[j], 0u));
                            else reinterpret_cast<float*>(out)[o] = __uint_as_float(v[j]);
                        }
                    }
                }
            }
            if (other) {
                if (epi_tid == 0) P.counters[sg.tile] = 0ull;          // both contributors are through with the word
            } else if (!whole) {
                // publish, count, and let the last contributor add all parts in contributor order (its own
                // included, re-read from memory: the sum then never depends on who came last)
                __threadfence();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (epi_tid == 0) (&bars->epi_prev)[nseg & 1u] = gemm_arrive(&P.counters[sg.tile], P.tag);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                const uint32_t prev = reinterpret_cast<volatile uint32_t*>(&bars->epi_prev)[nseg & 1u];
                if (prev == c_last - c_first) {
                    __threadfence();
                    if (epi_tid == 0) P.counters[sg.tile] = 0ull;
                    gemm_reduce_parts(P, P.tx, c_first, c_last, u0, tr.xrow0, n0, epi_tid);
                }
            }
            stop = epilogue_any(*abort_flag != 0u);    // and the next segment starts on the first transposition buffer again
            ++nseg;
            if (++d == nacc) { d = 0; dph ^= 1u; }
        }
    }
    // everybody meets here, also after a timeout, so the tensor memory is always returned
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// ---- the same GEMM, two CTAs per MMA (cta_group::2) --------------------------------------------
// A pair of CTAs (a cluster of two, on neighbouring SMs) works on 256 weight rows x 256 activation rows: each CTA
// decodes its own 128 weight rows into its own tensor memory and owns their accumulators, exactly as above, but
// loads only HALF of the activation tile (128 rows) into its shared memory; one tcgen05.mma.cta_group::2, issued by
// the first CTA of the pair, reads both halves.  A CTA therefore takes 16 KB of activations per k block from L2
// instead of 32 KB, so a stage of the same size holds a k block of 128 instead of 64: eight MMAs per round of
// barrier hand-overs instead of four.  That is what the pair buys here: the hand-overs of one round (stage freed ->
// refill and decode -> full -> issue -> commit) cost about 0.42 us whatever the ring depth and whatever else runs
// (measured with everything but the barriers switched off), against 0.35 us of tensor time for four MMAs.
//   barriers: the first CTA's b_full[s] collects its own TMA and the other CTA's (forwarded by a warp that waits
//   on that CTA's own barrier), its a_full[s] the decode warps of both CTAs, its d_free the epilogue warps of
//   both; one tcgen05.commit with a CTA mask signals stage_free[s] / d_full in both CTAs.
// Whole tiles only, n a multiple of 256, no expert groups; everything else runs the single-CTA kernel.
constexpr uint32_t kPairRound = 2;                        // 64-wide k blocks per stage (per round of hand-overs); 4 with two stages measured the same
constexpr uint32_t kPairStages = 8 / kPairRound;          // 8 x 32 tensor-memory columns of A, 8 x 16 KB of B, whatever the round
constexpr uint32_t kPairHalf = 128;                       // activation rows a CTA loads
constexpr uint32_t kPairSubBytes = kPairHalf * kGemmBK * 2;   // one 64-wide swizzled box: 16 KB
constexpr uint32_t kPairBBytes = kPairRound * kPairSubBytes;  // a stage: kPairRound boxes
constexpr uint32_t kPairIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);

struct PairBars {
    uint64_t b_full[kPairStages], b_own[kPairStages], a_full[kPairStages], stage_free[kPairStages];
    uint64_t raw_full[kGemmRawStages], raw_empty[kGemmRawStages];
    uint64_t d_full, d_free;
    uint32_t tmem_base, abort_flag;
};

// How a decode warp waits.  Where the decoders keep pace with the MMA they spend their time waiting, and one polling
// lane per warp keeps the barrier word free (every lane polling serialises on it).  Q6_K's decoders are the pacing
// part (Q3_K's too) and hardly ever find a barrier closed: there the single instruction of an all-lane poll is the
// cheaper form.
template <uint32_t SCHEME>
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t parity, uint32_t lane) {
    if constexpr (SCHEME == RLXQ_Q6_K || SCHEME == RLXQ_Q3_K) return mbar_wait(bar, parity);
    else return mbar_wait_warp(bar, parity, lane);
}

template <uint32_t SCHEME>
__global__ void __launch_bounds__(gemm_threads(GemmRaw<SCHEME>::GROUPS), 1) gemm_pair_kernel(const __grid_constant__ GemmParams P) {
    constexpr uint32_t RAW_ROW = GemmRaw<SCHEME>::ROW;
    constexpr uint32_t kGemmDecodeGroups = GemmRaw<SCHEME>::GROUPS;
    constexpr uint32_t RAW_BYTES = kGemmTileW * RAW_ROW;
    constexpr uint32_t RAW_STRIDE = (RAW_BYTES + 127) / 128 * 128;
    constexpr uint32_t TX = 256;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* b_stage = smem;                                          // kPairStages x 32 KB, 1024-aligned
    uint8_t* raw_stage = smem + kPairStages * kPairBBytes;
    PairBars* bars = reinterpret_cast<PairBars*>(raw_stage + kGemmRawStages * RAW_STRIDE);
    uint8_t* epi_stage = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(bars + 1) + 15) & ~(uintptr_t)15);

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t rank = cluster_cta_rank();            // 0 issues the MMAs
    volatile uint32_t* abort_flag = &bars->abort_flag;
    const bool dual = P.lo_row != 0;     // a round is 128 wide in k, or, for f32 activations, 64 wide with a hi and a lo box
    griddep_launch_dependents();

    if (tid == 0) {
        for (uint32_t s = 0; s < kPairStages; ++s) {
            mbar_init(smem_u32(&bars->b_full[s]), 2);        // own TMA (with its bytes) + the other CTA's, forwarded
            mbar_init(smem_u32(&bars->b_own[s]), 1);
            mbar_init(smem_u32(&bars->a_full[s]), dual ? 8 : 8 * kPairRound);   // per 64-wide block four decode warps, of each CTA
            mbar_init(smem_u32(&bars->stage_free[s]), 1);
        }
        for (uint32_t r = 0; r < kGemmRawStages; ++r) {
            mbar_init(smem_u32(&bars->raw_full[r]), 1);
            mbar_init(smem_u32(&bars->raw_empty[r]), 4 * kGemmDecodeGroups);
        }
        mbar_init(smem_u32(&bars->d_full), 1);
        mbar_init(smem_u32(&bars->d_free), 8);               // four epilogue warps of each CTA
        bars->abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {               // the same warp of both CTAs: all 512 columns in each
        tmem_alloc_pair(smem_u32(&bars->tmem_base), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();            // the other CTA's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t tmem_d = tmem_base, tmem_a = tmem_base + 256;
    auto give_up = [&](int code) {
        atomicExch(P.err, code);
        *abort_flag = 1u;
    };
    // the pair's tiles: 256 weight rows (pair index wp) x 256 activation rows (xt), xt fastest
    const uint32_t pt0 = blockIdx.x >> 1, pstep = gridDim.x >> 1, plim = (P.wtiles >> 1) * P.xtiles;
    const uint32_t rounds = dual ? 4 * P.kgroups : 4 * P.kgroups / kPairRound;  // rounds of a tile

    if (warp == 0) {
        // ---------------- this CTA's half of the activation tile ----------------
        if (elect_one()) {
            tma_prefetch_desc(&P.xmap);
            griddep_wait();
            uint32_t s = 0, ph = 1;
            bool ok = true;
            for (uint32_t pt = pt0; ok && pt < plim && !*abort_flag; pt += pstep) {
                const uint32_t xrow = (pt % P.xtiles) * TX + rank * kPairHalf;
                for (uint32_t kb = 0; kb < rounds; ++kb) {
                    if (*abort_flag || !mbar_wait(smem_u32(&bars->stage_free[s]), ph)) { give_up(21); ok = false; break; }
                    const uint32_t full = smem_u32(rank == 0 ? &bars->b_full[s] : &bars->b_own[s]);
                    mbar_arrive_expect_tx(full, kPairBBytes);
#pragma unroll
                    for (uint32_t q = 0; q < kPairRound; ++q)
                        tma_load_2d(smem_u32(b_stage + s * kPairBBytes + q * kPairSubBytes), &P.xmap,
                                    (int32_t)((dual ? kb : kb * kPairRound + q) * kGemmBK),
                                    (int32_t)(dual && q ? P.lo_row + xrow : xrow), full);
                    if (++s == kPairStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 3) {
        // ---------------- second CTA: tell the first that this half has landed ----------------
        if (lane == 0 && rank == 1) {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (uint32_t pt = pt0; ok && pt < plim && !*abort_flag; pt += pstep) {
                for (uint32_t kb = 0; kb < rounds; ++kb) {
                    if (*abort_flag || !mbar_wait(smem_u32(&bars->b_own[s]), ph)) { give_up(22); ok = false; break; }
                    mbar_arrive_cluster(cluster_map(smem_u32(&bars->b_full[s]), 0));
                    if (++s == kPairStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 2) {
        // ---------------- raw weight groups of this CTA's 128 rows ----------------
        if (elect_one()) {
            tma_prefetch_desc(&P.wmap);
            uint32_t r = 0, ph = 1;
            bool ok = true;
            for (uint32_t pt = pt0; ok && pt < plim && !*abort_flag; pt += pstep) {
                const uint32_t wrow0 = (2 * (pt / P.xtiles) + rank) * kGemmTileW;
                for (uint32_t g = 0; g < P.kgroups; ++g) {
                    if (*abort_flag || !mbar_wait(smem_u32(&bars->raw_empty[r]), ph)) { give_up(23); ok = false; break; }
                    const uint32_t full = smem_u32(&bars->raw_full[r]);
                    mbar_arrive_expect_tx(full, RAW_BYTES);
                    tma_load_2d(smem_u32(raw_stage + r * RAW_STRIDE), &P.wmap, (int32_t)gemm_raw_x<SCHEME>(g), (int32_t)wrow0, full);
                    if (++r == kGemmRawStages) { r = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: the first CTA, for both ----------------
        if (rank == 0 && elect_one()) {
            uint32_t s = 0, ph = 0, dph = 1;
            bool ok = true;
            for (uint32_t pt = pt0; ok && pt < plim && !*abort_flag; pt += pstep) {
                if (!mbar_wait(smem_u32(&bars->d_free), dph)) { give_up(24); break; }
                dph ^= 1u;
                tc_fence_after();
                uint32_t rb = mbar_test(smem_u32(&bars->b_full[s]), ph), ra = mbar_test(smem_u32(&bars->a_full[s]), ph);
                for (uint32_t kb = 0; kb < rounds; ++kb) {
                    if ((!rb && (*abort_flag || !mbar_wait(smem_u32(&bars->b_full[s]), ph))) ||
                        (!ra && (*abort_flag || !mbar_wait(smem_u32(&bars->a_full[s]), ph)))) { give_up(25); ok = false; break; }
                    tc_fence_after();
                    const uint32_t sn = s + 1 == kPairStages ? 0u : s + 1, phn = s + 1 == kPairStages ? ph ^ 1u : ph;
                    rb = mbar_test(smem_u32(&bars->b_full[sn]), phn);
                    ra = mbar_test(smem_u32(&bars->a_full[sn]), phn);
#pragma unroll
                    for (uint32_t j = 0; j < kPairRound * kGemmBK / 16; ++j) {
                        const uint64_t bdesc = kmajor_sw128_desc(smem_u32(b_stage + s * kPairBBytes + (j >> 2) * kPairSubBytes));
                        tc_mma_ts_pair(tmem_d, tmem_a + 32 * kPairRound * s + 8 * (dual ? j & 3u : j), bdesc + 2 * (j & 3u), kPairIdesc, (kb | j) ? 1u : 0u);
                    }
                    tc_commit_pair_both(smem_u32(&bars->stage_free[s]), 3);     // frees the stage in both CTAs
                    s = sn;
                    ph = phn;
                }
                if (!ok) break;
                tc_commit_pair_both(smem_u32(&bars->d_full), 3);
            }
        }
    } else if (warp >= 4 && warp < 4 + 4 * kGemmDecodeGroups) {
        // ---------------- decode: raw blocks -> bf16 rows in this CTA's tensor memory ----------------
        const uint32_t quarter = warp & 3u, grp = (warp - 4) >> 2;
        const uint32_t row = quarter * 32 + lane;
        const uint32_t lane_addr = (quarter * 32) << 16;
        uint32_t r = 0, rph = 0, kbg0 = 0;
        bool ok = true;
        uint32_t raw_ready = 0;
        for (uint32_t pt = pt0; ok && pt < plim && !*abort_flag; pt += pstep) {
            for (uint32_t g = 0; g < P.kgroups && ok; ++g, kbg0 += 4) {
                if (!__all_sync(0xFFFFFFFFu, raw_ready) &&
                    (*abort_flag || !pair_wait<SCHEME>(smem_u32(&bars->raw_full[r]), rph, lane))) { give_up(26); ok = false; break; }
                const uint8_t* rp = raw_stage + r * RAW_STRIDE + row * RAW_ROW;
                // 64-wide block kbg is part kbg % kPairRound of round kbg / kPairRound
                auto stage_of = [&](uint32_t sub, uint32_t& st, uint32_t& sph, uint32_t& col) {
                    const uint32_t kbg = kbg0 + sub, rd = dual ? kbg : kbg / kPairRound;
                    st = rd % kPairStages;
                    sph = ((rd / kPairStages) & 1u) ^ 1u;
                    col = 32 * (kPairRound * st + (dual ? 0u : kbg % kPairRound));
                };
                auto store = [&](uint32_t st, uint32_t sph, uint32_t col, uint32_t ready, const GemmOut<false>& v) -> bool {
                    if (!__all_sync(0xFFFFFFFFu, ready) &&
                        (*abort_flag || !pair_wait<SCHEME>(smem_u32(&bars->stage_free[st]), sph, lane))) { give_up(27); return false; }
                    tc_fence_after();
                    tmem_st32(tmem_a + lane_addr + col, v.hi);
                    // announced at once (the single-CTA kernel's delay costs 4 % here: a round waits for sixteen of these)
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (rank == 0) mbar_arrive(smem_u32(&bars->a_full[st]));
                        else mbar_arrive_cluster(cluster_map(smem_u32(&bars->a_full[st]), 0));
                    }
                    return true;
                };
                uint32_t st, sph, col;
                if constexpr (gemm_part_loop(SCHEME)) {
                    Q6Half hf;
                    if constexpr (SCHEME == RLXQ_Q6_K) hf.load(rp, (210u * g) & 15u, grp);
#pragma unroll 1
                    for (uint32_t p = 0; p < 2 && ok; ++p) {
                        const uint32_t sub = SCHEME == RLXQ_Q6_K ? 2 * grp + p : grp + 2 * p;
                        stage_of(sub, st, sph, col);
                        const uint32_t ready = mbar_test(smem_u32(&bars->stage_free[st]), sph);     // answered while decoding
                        GemmOut<false> v;
                        if constexpr (SCHEME == RLXQ_Q6_K) hf.decode(p, v);
                        else if constexpr (SCHEME == RLXQ_Q4_K || SCHEME == RLXQ_Q5_K) decode_k45<SCHEME>(rp, sub, v);
                        else if (grp == 0) decode_blocks32<SCHEME, 0>(rp, p, v);
                        else decode_blocks32<SCHEME, 1>(rp, p, v);
                        ok = store(st, sph, col, ready, v);
                    }
                } else {
#pragma unroll
                    for (uint32_t sub = 0; sub < 4; ++sub) {
                        if (!ok || (kbg0 + sub) % kGemmDecodeGroups != grp) continue;
                        stage_of(sub, st, sph, col);
                        const uint32_t ready = mbar_test(smem_u32(&bars->stage_free[st]), sph);
                        GemmOut<false> v;
                        if (sub == 0) decode64<SCHEME, 0>(rp, g, v);
                        else if (sub == 1) decode64<SCHEME, 1>(rp, g, v);
                        else if (sub == 2) decode64<SCHEME, 2>(rp, g, v);
                        else decode64<SCHEME, 3>(rp, g, v);
                        ok = store(st, sph, col, ready, v);
                    }
                }
                if (!ok) break;
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->raw_empty[r]));
                if (++r == kGemmRawStages) { r = 0; rph ^= 1u; }
                raw_ready = mbar_test(smem_u32(&bars->raw_full[r]), rph);
            }
        }
    } else if (warp >= 4 + 4 * kGemmDecodeGroups) {
        // ---------------- epilogue: this CTA's 128 weight rows x 256 activation rows -> y ----------------
        const uint32_t quarter = warp & 3u;
        const uint32_t lane_addr = (quarter * 32) << 16;
        const uint32_t row = quarter * 32 + lane;
        const uint32_t epi_tid = (warp - (4 + 4 * kGemmDecodeGroups)) * 32 + lane;
        uint32_t dph = 0;
        griddep_wait();                      // y may still be in use by the kernel in front
        for (uint32_t pt = pt0; pt < plim && !*abort_flag; pt += pstep) {
            const uint32_t wt = 2 * (pt / P.xtiles) + rank, xrow0 = (pt % P.xtiles) * TX;
            if (!mbar_wait_warp(smem_u32(&bars->d_full), dph, lane)) { give_up(28); break; }
            dph ^= 1u;
            tc_fence_after();
            const uint32_t n_idx = wt * kGemmTileW + row;
#pragma unroll 1
            for (uint32_t c = 0; c < TX / 32; ++c) {
                uint32_t v[32];
                tmem_ld32(tmem_d + lane_addr + 32 * c, v);
                tmem_ld_wait();
                if (c == TX / 32 - 1) {          // everything is in registers: the accumulator may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (rank == 0) mbar_arrive(smem_u32(&bars->d_free));
                        else mbar_arrive_cluster(cluster_map(smem_u32(&bars->d_free), 0));
                    }
                }
                if (P.y_vec) {
                    const GemmDst d{reinterpret_cast<uint8_t*>(P.y), P.n, xrow0, P.m, wt * kGemmTileW, P.n, nullptr};
                    if (P.y_bf16) gemm_store_vec<false>(epi_stage, epi_tid, row, v, d, c);
                    else gemm_store_vec<true>(epi_stage, epi_tid, row, v, d, c);
                } else if (n_idx < P.n) {
#pragma unroll
                    for (uint32_t j = 0; j < 32; ++j) {
                        const uint32_t m_idx = xrow0 + 32 * c + j;
                        if (m_idx < P.m) {
                            const size_t o = (size_t)m_idx * P.n + n_idx;
                            if (P.y_bf16) reinterpret_cast<uint16_t*>(P.y)[o] = (uint16_t)bf16x2_of(f32x2(v[j], 0u));
                            else reinterpret_cast<float*>(P.y)[o] = __uint_as_float(v[j]);
                        }
                    }
                }
            }
        }
    }
    // both CTAs meet here, also after a timeout: neither returns its tensor memory while the other may still use it
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---- host side --------------------------------------------------------------------------------
static bool gemm_tc_format(uint32_t scheme) {
    switch (scheme) {
        case RLXQ_Q4_0: case RLXQ_Q8_0: case RLXQ_Q4_K: case RLXQ_Q6_K: case RLXQ_Q5_K: case RLXQ_Q2_K: case RLXQ_Q3_K:
        case RLXQ_Q8_K: case RLXQ_Q4_1: case RLXQ_Q5_0: case RLXQ_Q5_1: return true;
        default: return false;
    }
}
// The GEMM on the weights where they lie: rows of whole 256-weight groups that start on 16-byte boundaries.
bool gemm_tc_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* w, const void* x) {
    if (m == 0 || n == 0 || k == 0 || k % 256 || !gemm_tc_format(scheme)) return false;
    if ((scheme == RLXQ_Q6_K || scheme == RLXQ_Q3_K) && k % 2048) return false;   // rows must stay 16-byte aligned
    if ((scheme == RLXQ_Q2_K || scheme == RLXQ_Q8_K) && k % 1024) return false;
    if (((uintptr_t)w & 15u) || ((uintptr_t)x & 15u)) return false;
    return true;
}
// Every other row length (and alignment of the weights): rows re-laid on a pitch TMA can tile, then the PRECISE form.
bool gemm_relaid_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* x) {
    return m != 0 && n != 0 && k != 0 && k % 32 == 0 && gemm_tc_format(scheme) && !((uintptr_t)x & 15u);
}
// Bytes from one re-laid row to the next: whole 256-weight groups (zero blocks past k), a multiple of 16; and bytes of `rows`
// re-laid rows, with the scales that widened ones keep behind them.
uint64_t gemm_relaid_pitch(uint32_t layout, uint32_t k) {
    if (layout == kQ6Wide) return (uint64_t)(k / 256) * GemmRaw<kQ6Wide>::ROW;
    Geometry g;
    geometry(layout, &g);
    return ((uint64_t)((k + 255) / 256) * (256 / g.elems) * g.bytes + 15) / 16 * 16;
}

uint64_t gemm_relaid_bytes(uint32_t layout, uint32_t k, uint64_t rows) {
    return gemm_relaid_pitch(layout, k) * rows + (layout == kQ6Wide ? (uint64_t)(k / 256) * rows * 4 : 0);
}

int launch_relay(cudaStream_t stream, uint32_t layout, const uint8_t* w, uint32_t k, uint64_t n, uint8_t* out, const uint32_t* used,
                 uint32_t slab_rows) {
    if (layout == kQ6Wide) return launch_widen_q6(stream, w, k, n, out, used, slab_rows);
    Geometry g;
    geometry(layout, &g);
    return launch_relay_rows(stream, w, (uint64_t)k / g.elems * g.bytes, n, out, gemm_relaid_pitch(layout, k), used, slab_rows);
}

// Parts of an activation value: bf16 ones are one, f32 ones hi and lo, or all 24 bits beside PRECISE weights.
uint32_t gemm_x_parts(bool f32, bool precise) { return !f32 ? 1u : precise ? 3u : 2u; }
// The most activation rows of a tile: four operand stages (PRECISE: three) and two raw boxes have to fit in shared memory,
// accumulators and weight stages in tensor memory.
uint32_t gemm_most_rows(uint32_t scheme, bool f32, bool precise) {
    if (!precise) return f32 ? 128u : 256u;
    return gemm_precise_rows(scheme);
}

struct GemmShape { uint32_t tx, xtiles, slices; bool streamk, pair; };

// Activation rows per tile, work split and kernel for a shape, by estimated time in cycles.  A 64-wide k block of a tile
// costs the larger of its MMAs (2 cycles per activation row and product plus the hand-over; `products`: bf16 activations
// 1, f32 2, three times that with PRECISE weights) and its decode, whatever part of the tile's rows is padding; so few rows get a
// narrow tile, and rows are split evenly over the fewest tiles that leave no SM idle.  The constants are fits to 45 shapes
// (five formats, 16 to 1526 rows, k 2048 to 14336), each timed at every tile width, split and kernel: the choice made here
// takes 1 % longer than the best one in the geometric mean, up to 10 % at worst.
// PRECISE: the decoders of three parts and the emptying of the accumulators, measured with one tile on every SM; re-laid Q6_K is
// bound by MMA issue and, above 64 rows of f32 activations, by its three stages (cycles a block at 32, 64, 80, 96 rows: f32 960,
// 1365, 1463, 1800, bf16 850, 885, 900, 920).
static uint32_t gemm_block_cycles(uint32_t scheme, uint32_t tx, uint32_t products, bool precise, bool pair) {
    if (gemm_late_scale(scheme)) return products > 3 ? (tx <= 64 ? 560 + 12 * tx : 20 * tx - 140) : 820 + tx;
    if (precise) {
        const uint32_t base = scheme == RLXQ_Q4_0 ? 1150 : scheme == RLXQ_Q8_0 ? 1900 : scheme == RLXQ_Q3_K ? 3000 : scheme == RLXQ_Q6_K ? 1580 :
                              scheme == RLXQ_Q4_K || scheme == RLXQ_Q5_K ? 1700 : 2750;
        return base + (products > 3 ? 7 : 4) * tx;
    }
    const bool heavy = scheme == RLXQ_Q6_K || scheme == RLXQ_Q3_K;
    if (pair) return heavy && products == 1 ? 925 : 750 * products;        // 256 activation rows, both CTAs at once
    uint32_t mma = 2 * tx * products + 265 + (products > 1 ? 65 : 0);
    if (products == 2 && tx >= 96 && mma < 800) mma = 800;
    if (heavy) mma += 90;
    uint32_t dec = scheme == RLXQ_Q3_K ? 1130 : heavy ? 740 : scheme == RLXQ_Q8_0 || scheme == RLXQ_Q4_0 || scheme == RLXQ_Q4_K ? 570 : 620;
    return mma > dec ? mma : dec;
}
// Two CTAs per MMA; PRECISE weights are not built in that form.
static bool gemm_pair_fits(uint32_t n, bool precise) { return n % 256 == 0 && !precise; }
static GemmShape gemm_choose(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, bool f32, bool precise, bool can_split) {
    const uint64_t sms = (uint64_t)sm_count(), wt = (n + kGemmTileW - 1) / kGemmTileW, groups = (k + 255) / 256, blocks = 4 * groups;
    const uint32_t products = !precise ? (f32 ? 2 : 1) : gemm_weight_parts(scheme) + (f32 ? 3 : 0);
    const uint32_t most = gemm_most_rows(scheme, f32, precise);
    const int64_t fx = options().gemm_tile_x.load(), fs = can_split ? options().gemm_streamk.load() : 1, fp = options().gemm_pair.load();
    const GemmShape pair{256, (m + 255) / 256, 1, false, true};
    if (fp == 2 && gemm_pair_fits(n, precise)) return pair;
    GemmShape best{};
    uint64_t best_cost = ~0ull;
    auto take = [&](uint64_t cost, const GemmShape& sh) { if (cost < best_cost) { best_cost = cost; best = sh; } };
    if (fp != 1 && !fx && fs != 2 && gemm_pair_fits(n, precise)) {
        const uint64_t ptiles = (uint64_t)(n / 256) * pair.xtiles, pairs = sms / 2;
        take((ptiles + pairs - 1) / pairs * blocks * gemm_block_cycles(scheme, 256, products, precise, true) + 24 * 256, pair);
    }
    const uint32_t least_tiles = (m + most - 1) / most;
    for (uint32_t xt = least_tiles; xt <= least_tiles + 8; ++xt) {
        uint32_t tx = ((m + xt - 1) / xt + 31) / 32 * 32;
        if (gemm_late_scale(scheme) && tx == 96 && (m + xt - 1) / xt <= 80) tx = 80;
        if (fx) tx = (uint32_t)fx < most ? (uint32_t)fx : most;
        const uint32_t tiles_x = (m + tx - 1) / tx;
        if (tiles_x != xt && !fx) continue;              // the same width as one tile fewer
        const uint64_t ntiles = wt * tiles_x, cyc = gemm_block_cycles(scheme, tx, products, precise, false);
        const uint64_t epi = (precise ? 100 : 24) * tx;  // the last tile's epilogue, and with one accumulator every tile's
        if (fs != 2 || precise) take((ntiles + sms - 1) / sms * (blocks * cyc + (tx > 128 || precise ? epi : 0)) + epi, GemmShape{tx, tiles_x, 1, false, false});
        // k split over the SMs (stream-K): every SM gets the same blocks, and exchanges up to two parts of 128 x tx values
        // (PRECISE sums are in registers by then, with no code to exchange them: whole tiles and slices only)
        if (!precise && fs != 1 && (fs == 2 || ntiles % sms))
            take((ntiles * blocks + sms - 1) / sms * cyc + epi + 6000 + 200 * tx, GemmShape{tx, tiles_x, 1, true, false});
        // PRECISE: as many slices as make the last wave a full one, where they are no more than 192 MiB
        for (uint64_t sl = 2; precise && fs == 0 && sl <= 8 && 4 * sl <= groups && sl * m * n <= (192ull << 20) / 4; ++sl)
            take((ntiles * sl + sms - 1) / sms * ((groups + sl - 1) / sl * 4 * cyc + epi) + 3200 + sl * m * n / 600, GemmShape{tx, tiles_x, (uint32_t)sl, false, false});
        // few tiles: every SM takes a slice of some tile's k, and a kernel behind this one adds the slices
        if (fs == 0 && 2 * ntiles <= sms) {
            const uint64_t fit = sms / ntiles, sl = groups < fit ? groups : fit;
            if (sl > 1) take((groups + sl - 1) / sl * 4 * cyc + epi + 3200 + sl * m * n / 600, GemmShape{tx, tiles_x, (uint32_t)sl, false, false});
        }
        if (fx) break;
    }
    return best;
}
static size_t gemm_streamk_bytes(uint64_t ntiles, uint32_t tx, size_t* off_partial) {
    const size_t counters = ((size_t)ntiles * 8 + 255) / 256 * 256;
    if (off_partial) *off_partial = counters;
    return counters + 2 * (size_t)sm_count() * kGemmTileW * tx * 4;     // two partial tiles per CTA
}
static size_t gemm_slice_elems(uint32_t m, uint32_t n) { return ((size_t)m * n + 3) / 4 * 4; }
static size_t gemm_shape_bytes(const GemmShape& sh, uint32_t m, uint32_t n) {
    if (sh.slices > 1) return sh.slices * gemm_slice_elems(m, n) * 4;
    return sh.streamk ? gemm_streamk_bytes((uint64_t)((n + kGemmTileW - 1) / kGemmTileW) * sh.xtiles, sh.tx, nullptr) : 0;
}

// Scratch the GEMM would use for this shape (0 when whole tiles fill the SMs well enough).
size_t gemm_tc_workspace_bytes(uint32_t layout, uint32_t m, uint32_t k, uint32_t n, bool f32, bool precise) {
    if (m == 0 || k == 0 || n == 0) return 0;
    return gemm_shape_bytes(gemm_choose(layout, m, k, n, f32, precise, true), m, n);
}

// A different tag for each of the calls that may be in flight together; where they start differs from process to process.
static unsigned long long next_gemm_tag() {
    static std::atomic<unsigned long long> calls{(unsigned long long)std::chrono::steady_clock::now().time_since_epoch().count() * 0x9E3779B97F4A7C15ull};
    return arrival_tag(calls.fetch_add(1));
}

template <uint32_t SCHEME, bool PRECISE>
static int launch_gemm_t(cudaStream_t stream, const GemmCall& c, const GemmShape& sh, void* ws) {
    constexpr uint32_t RAW_ROW = GemmRaw<SCHEME>::ROW;
    constexpr uint32_t RAW_STRIDE = (kGemmTileW * RAW_ROW + 127) / 128 * 128;
    Geometry g;
    geometry(SCHEME & 0xFFu, &g);
    GemmParams P{};
    P.tx = sh.tx;
    P.lo_row = c.f32 ? c.x_rows : 0u;
    P.xparts = gemm_x_parts(c.f32, PRECISE);
    P.main_run = gemm_main_run(SCHEME, c.k, c.ybf);
    P.sum_run = gemm_sum_run(c.k, c.ybf);
    P.cross_run = gemm_late_scale(SCHEME) ? 4u : P.sum_run;
    P.late_rows = (size_t)c.n * c.num_slabs;
    P.late = reinterpret_cast<const float*>(c.w + c.w_pitch * P.late_rows);
    P.x = static_cast<const uint16_t*>(c.x);
    P.w = c.w;
    int rc = encode_bf16_kmajor_map(&P.xmap, c.x, (uint64_t)c.x_rows * P.xparts, c.k, P.tx);
    if (rc) return rc;
    rc = encode_weight_map(&P.wmap, c.w, (uint64_t)c.n * c.num_slabs, c.w_pitch ? c.w_pitch : (uint64_t)c.k / g.elems * g.bytes,
                           RAW_ROW / 8, kGemmTileW);
    if (rc) return rc;
    P.y = c.y; P.m = c.x_rows; P.n = c.n; P.k = c.k; P.y_bf16 = c.ybf;
    P.slices = sh.slices;
    if (sh.slices > 1) {
        P.y = ws; P.y_bf16 = 0;
        P.slice_elems = gemm_slice_elems(c.x_rows, c.n);
    }
    P.groups = static_cast<const uint4*>(c.groups);
    P.row_map = c.row_map;
    P.w_late = c.w_pitch ? 1u : 0u;
    P.y_vec = (((uintptr_t)P.y & 15u) == 0 && c.n % (P.y_bf16 ? 8u : 4u) == 0) ? 1u : 0u;
    P.wtiles = (c.n + kGemmTileW - 1) / kGemmTileW;
    P.xtiles = sh.xtiles;
    P.kgroups = (c.k + 255) / 256;
    P.err = device_error_word();
    if (!P.err) return fail(RLXQ_E_CUDA, "device error word unavailable");
    // as many operand stages as tensor memory and shared memory hold beside two raw boxes, then raw boxes
    P.b_bytes = P.tx * kGemmBK * 2 * P.xparts;
    const uint32_t smem = 227 * 1024;   // all of it: one CTA per SM, so that none waits for another's tensor memory
    const uint32_t budget = smem - (1024 + sizeof(GemmBars) + 64 + (PRECISE ? P.tx * kGemmTileW * 4 : kGemmEpiStage));
    P.nstages = std::min<uint32_t>(PRECISE ? 4u : kGemmMaxStages, (budget - kGemmRawStages * RAW_STRIDE) / P.b_bytes);
    if (PRECISE) {
        // tensor memory: weight stages first, then a second accumulator of either kind
        constexpr uint32_t A_COLS = gemm_a_cols(SCHEME, true);
        P.nstages = std::min(P.nstages, (512u - 2u * P.tx) / A_COLS);
        const uint32_t spare = gemm_late_scale(SCHEME) ? (512u - 2u * P.tx - P.nstages * A_COLS) / P.tx : 0u;
        P.nmain = spare >= 1 ? 2u : 1u;
        P.ncross = spare >= 2 ? 2u : 1u;
    }
    // (a decode group's parts may lie up to three stages apart, gemm_decode_role: no ring below that)
    if (P.nstages < (PRECISE ? 3u : 4u)) return fail(RLXQ_E_LIMIT, "GEMM tile of %u activation rows too large", P.tx);
    P.nraw = std::min<uint32_t>(kGemmMaxRaw, (budget - P.nstages * P.b_bytes) / RAW_STRIDE);
    static std::atomic<uint32_t> attr_set[64];
    int dev = 0;
    RLXQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && attr_set[dev].load() == 0) {
        RLXQ_CUDA_TRY(cudaFuncSetAttribute(gemm_tcgen05_kernel<SCHEME, PRECISE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[dev].store(1);
    }
    uint32_t grid = (uint32_t)sm_count();
    const uint64_t ntiles = (uint64_t)P.wtiles * P.xtiles * P.slices;
    if (ntiles * P.kgroups > 0xFFFFFFFFull) return fail(RLXQ_E_LIMIT, "GEMM too large");
    if (sh.streamk) {
        const uint64_t units = ntiles * P.kgroups;
        if (grid > units) grid = (uint32_t)units;
        size_t off_partial = 0;
        gemm_streamk_bytes(ntiles, P.tx, &off_partial);
        P.streamk = 1;
        P.units_q = (uint32_t)(units / grid);
        P.units_r = (uint32_t)(units % grid);
        P.counters = static_cast<unsigned long long*>(ws);
        P.partial = reinterpret_cast<float*>(static_cast<uint8_t*>(ws) + off_partial);
        P.tag = next_gemm_tag();
    } else if (grid > ntiles && !c.groups) {
        grid = (uint32_t)ntiles;
    }
    rc = launch_pdl(gemm_tcgen05_kernel<SCHEME, PRECISE>, dim3(grid), dim3(gemm_threads(GemmRaw<SCHEME>::GROUPS, gemm_epilogue_warps(SCHEME, PRECISE))), smem,
                    stream, P);
    if (rc) return rc;
    count_launch();
    if (P.slices > 1) return launch_add_slices(stream, static_cast<const float*>(ws), P.slices, P.slice_elems, c.y, c.ybf, (uint64_t)c.x_rows * c.n);
    return check_launch("gemm_tcgen05_kernel");
}
template <uint32_t SCHEME>
static int launch_gemm_t_any(cudaStream_t stream, const GemmCall& c, const GemmShape& sh, void* ws) {
    if constexpr (SCHEME == kQ6Wide) return launch_gemm_t<SCHEME, true>(stream, c, sh, ws);
    else return c.precise ? launch_gemm_t<SCHEME, true>(stream, c, sh, ws) : launch_gemm_t<SCHEME, false>(stream, c, sh, ws);
}

// The two-CTA form: whole 256 x 256 tile pairs dealt round-robin to as many clusters as are resident at once.
template <uint32_t SCHEME>
static int launch_gemm_pair_t(cudaStream_t stream, const GemmCall& c) {
    constexpr uint32_t RAW_ROW = GemmRaw<SCHEME>::ROW;
    constexpr uint32_t RAW_STRIDE = (kGemmTileW * RAW_ROW + 127) / 128 * 128;
    Geometry g;
    geometry(SCHEME, &g);
    GemmParams P{};
    P.lo_row = c.f32 ? c.x_rows : 0u;
    int rc = encode_bf16_kmajor_map(&P.xmap, c.x, (uint64_t)c.x_rows * (c.f32 ? 2 : 1), c.k, kPairHalf);
    if (rc) return rc;
    rc = encode_weight_map(&P.wmap, c.w, c.n, (uint64_t)c.k / g.elems * g.bytes, RAW_ROW / 8, kGemmTileW);
    if (rc) return rc;
    P.y = c.y; P.m = c.x_rows; P.n = c.n; P.k = c.k; P.y_bf16 = c.ybf;
    P.y_vec = (((uintptr_t)c.y & 15u) == 0 && c.n % (c.ybf ? 8u : 4u) == 0) ? 1u : 0u;
    P.wtiles = c.n / kGemmTileW;
    P.xtiles = (c.x_rows + 255) / 256;
    P.kgroups = c.k / 256;
    P.err = device_error_word();
    if (!P.err) return fail(RLXQ_E_CUDA, "device error word unavailable");
    const size_t smem = 1024 + (size_t)kPairStages * kPairBBytes + (size_t)kGemmRawStages * RAW_STRIDE + sizeof(PairBars) + 64 +
                        kGemmEpiStage;
    const uint32_t threads = gemm_threads(GemmRaw<SCHEME>::GROUPS);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = options().pdl.load() ? 1 : 0;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    static std::atomic<int> clusters_of[64];        // resident clusters per device, found once (0 = not yet)
    int dev = 0;
    RLXQ_CUDA_TRY(cudaGetDevice(&dev));
    int clusters = (dev >= 0 && dev < 64) ? clusters_of[dev].load() : 0;
    if (clusters == 0) {
        RLXQ_CUDA_TRY(cudaFuncSetAttribute(gemm_pair_kernel<SCHEME>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        cfg.gridDim = dim3((unsigned)sm_count() & ~1u);
        RLXQ_CUDA_TRY(cudaOccupancyMaxActiveClusters(&clusters, gemm_pair_kernel<SCHEME>, &cfg));
        if (clusters < 1) return fail(RLXQ_E_CUDA, "no cluster of two CTAs of the paired GEMM fits this device");
        if (dev >= 0 && dev < 64) clusters_of[dev].store(clusters);
        options().gemm_pair_clusters = clusters;
    }
    const uint32_t ptiles = (P.wtiles / 2) * P.xtiles;
    uint32_t pairs = (uint32_t)clusters;
    if (pairs > (uint32_t)sm_count() / 2) pairs = (uint32_t)sm_count() / 2;
    if (pairs > ptiles) pairs = ptiles;
    cfg.gridDim = dim3(2 * pairs);
    cfg.numAttrs = 2;
    RLXQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_pair_kernel<SCHEME>, P));
    count_launch();
    return check_launch("gemm_pair_kernel");
}

template <uint32_t SCHEME>
static int launch_gemm_s(cudaStream_t stream, const GemmCall& c, void* ws, size_t ws_bytes) {
    if (c.groups) return launch_gemm_t_any<SCHEME>(stream, c, GemmShape{c.tile_rows, c.group_tiles, 1, false, false}, nullptr);
    GemmShape sh = gemm_choose(SCHEME, c.x_rows, c.k, c.n, c.f32, c.precise, true);
    if ((sh.streamk || sh.slices > 1) && (!ws || ((uintptr_t)ws & 15u) || ws_bytes < gemm_shape_bytes(sh, c.x_rows, c.n)))
        sh = gemm_choose(SCHEME, c.x_rows, c.k, c.n, c.f32, c.precise, false);
    if constexpr (SCHEME != kQ6Wide)
        if (sh.pair) return launch_gemm_pair_t<SCHEME>(stream, c);
    return launch_gemm_t_any<SCHEME>(stream, c, sh, ws);
}

int launch_gemm(cudaStream_t stream, uint32_t layout, const GemmCall& c, void* ws, size_t ws_bytes) {
    if ((uint64_t)c.n * c.num_slabs > 0x7FFFFFFFull) return fail(RLXQ_E_LIMIT, "weights too tall for a tensor map");
    switch (layout) {
        case RLXQ_Q4_0: return launch_gemm_s<RLXQ_Q4_0>(stream, c, ws, ws_bytes);
        case RLXQ_Q8_0: return launch_gemm_s<RLXQ_Q8_0>(stream, c, ws, ws_bytes);
        case RLXQ_Q4_K: return launch_gemm_s<RLXQ_Q4_K>(stream, c, ws, ws_bytes);
        case RLXQ_Q5_K: return launch_gemm_s<RLXQ_Q5_K>(stream, c, ws, ws_bytes);
        case RLXQ_Q2_K: return launch_gemm_s<RLXQ_Q2_K>(stream, c, ws, ws_bytes);
        case RLXQ_Q8_K: return launch_gemm_s<RLXQ_Q8_K>(stream, c, ws, ws_bytes);
        case RLXQ_Q4_1: return launch_gemm_s<RLXQ_Q4_1>(stream, c, ws, ws_bytes);
        case RLXQ_Q5_0: return launch_gemm_s<RLXQ_Q5_0>(stream, c, ws, ws_bytes);
        case RLXQ_Q5_1: return launch_gemm_s<RLXQ_Q5_1>(stream, c, ws, ws_bytes);
        case RLXQ_Q3_K: return launch_gemm_s<RLXQ_Q3_K>(stream, c, ws, ws_bytes);
        case RLXQ_Q6_K: return launch_gemm_s<RLXQ_Q6_K>(stream, c, ws, ws_bytes);
        case kQ6Wide: return launch_gemm_s<kQ6Wide>(stream, c, ws, ws_bytes);
        default: return fail(RLXQ_E_SCHEME, "unknown scheme");
    }
}

}  // namespace rlxq
