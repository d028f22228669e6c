// Streaming decode GEMV with f32 accuracy on the warp-level matrix instruction, for five to eight rows of activations and weight
// rows of any length (Q4_0, Q8_0, Q6_K; gemv_f32.cu has the same rows' batches of one to four).
//
// Quants are small integers, exact in bf16, and an f32 activation is the exact sum of three bf16 parts.  So the products of
// mma.m16n8k16 (sixteen weight rows, eight columns of activations) are exact.  What is rounded are the sums that each of a
// scale's one to six instructions leaves behind, small parts first, and then, in f32, the sum times the scale and the row's
// total: two or four totals a step and four over the warps, added pairwise, because one chain through all scales was up to 1.26
// times as far from 64 bits as the f32 kernel (Q6_K, bf16 activations).  600 calls of batch 5 to 8, k 256 to 16416: error 0.77
// to 0.97 of the f32 kernel's, 0.86 in the mean; the additional sums cost 1 % in the mean, 5 % for long Q6_K rows in bf16.  A weight is
// decoded once for all eight rows, one instruction a 16 x 16 tile of weights for bf16 activations, three for f32 ones.
//
// A CTA's warps form streams: the warps of a stream stand side by side over the columns, 256 each, and take tiles of sixteen
// weight rows, every stream its own.  The activations lie in shared memory in the instruction's operand order, for all
// streams.  Each warp fetches its own pieces of the rows into a ring of its own, in 16-byte asynchronous copies from the
// boundary below the piece, so a row may start on any even byte and no warp waits for another; per tile the sums of a stream's
// warps meet once in shared memory.  Rows of more columns than fit are taken in passes, all of the CTA's tiles in one pass
// after the other.  The loops are rolled: a call lasts microseconds, and straight-line code for 256 columns cost three of
// them to fetch.
//
// Bound: latency at twelve to sixteen warps an SM.  Q6_K 5888 x 14336, batch 8, f32 activations: issue slots 42 % used (8.2 lane
// instructions a weight, a third of them copies, scales and the meeting of the warps), 7.2 cycles from a warp's instruction to its
// next (fixed latencies 1.3, loads 1.1, the meeting 1.0, shared memory 0.8), DRAM 14 %.  Batch 8, f32 activations, the f32 kernel (four
// rows a pass, so twice) and this one: Q6_K 2304 x 6000 19.2 and 13.3 us, 5888 x 14336 95 and 58, 12544 x 14400 224 and 119;
// Q8_0 1056 x 16000 25.4 and 12.8, 9280 x 3328 41.6 and 36.7; Q4_0 544 x 8000 8.8 and 4.7; bf16 activations, Q6_K 5888 x 14336 94
// and 45.  At batch 3 and 4 the f32 kernel is level or ahead.
#include <algorithm>

#include "common.cuh"
#include "decode.cuh"
#include "kernels.h"
#include "staged_common.cuh"

namespace rlxq {

constexpr uint32_t kPartsMaxWarps = 16;
constexpr uint32_t kPartsTile = 16;       // weight rows per tile
constexpr uint32_t kPartsCols = 256;      // columns per warp
constexpr uint32_t kPartsTotals = 64;     // tiles whose totals are kept between column passes

// PIECE: bytes of a row that one step takes; SLOT: bytes between the rows of a step in shared memory (room for 14 bytes in
// front of the piece, and rows that start on different banks); PER: steps per 256 columns.
template <uint32_t SCHEME> struct PartsGeom;
template <> struct PartsGeom<RLXQ_Q4_0> { static constexpr uint32_t PIECE = 144, SLOT = 176, PER = 1; };
template <> struct PartsGeom<RLXQ_Q8_0> { static constexpr uint32_t PIECE = 136, SLOT = 176, PER = 2; };
template <> struct PartsGeom<RLXQ_Q6_K> { static constexpr uint32_t PIECE = 210, SLOT = 240, PER = 1; };
struct PartsParams {
    const void* x;
    const uint8_t* w;
    void* y;
    uint32_t y_bf16, m, k, n;
    uint64_t row_bytes;
    uint32_t passes, tiles, ctas;         // column passes; tiles of the n rows; CTAs that share them
    uint32_t nw, streams, depth;          // warps of a stream (side by side over the columns), streams, steps in a warp's ring
    uint32_t off_ring, off_red, off_total;  // shared-memory layout: operands, rings, the streams' sums, totals between passes
};

__device__ __forceinline__ void parts_copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void parts_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void parts_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

extern __shared__ __align__(16) uint8_t parts_smem[];
__device__ __forceinline__ uint32_t parts_lds(uint32_t a) { return *reinterpret_cast<const uint32_t*>(parts_smem + a); }
__device__ __forceinline__ uint2 parts_lds2(uint32_t a) { return *reinterpret_cast<const uint2*>(parts_smem + a); }
__device__ __forceinline__ uint4 parts_lds4(uint32_t a) { return *reinterpret_cast<const uint4*>(parts_smem + a); }
__device__ __forceinline__ uint32_t parts_lds16(uint32_t a) { return *reinterpret_cast<const uint16_t*>(parts_smem + a); }
// A row piece in shared memory.  at: the offset of its first byte (even).  Words that lie a multiple of four bytes behind it are read
// from `even` on and moved by `even_sh` bits, words two bytes past such a place from `odd` on, moved by `odd_sh`.
struct PartsRow {
    uint32_t at, even, odd, even_sh, odd_sh;
    __device__ __forceinline__ explicit PartsRow(uint32_t a) : at(a) {
        even = a & ~3u;
        even_sh = (a & 2u) * 8u;
        odd = even + 2u * (a & 2u);
        odd_sh = 16u - even_sh;
    }
    __device__ __forceinline__ void move(uint32_t bytes) { at += bytes; even += bytes; odd += bytes; }     // (a multiple of 4)
};
// The word `off` bytes into a row (off is a constant and even).  W4: rows start on whole words.
template <bool W4> __device__ __forceinline__ uint32_t parts_word(const PartsRow& r, uint32_t lane_off, uint32_t off) {
    if (off % 4 == 0) {
        if (W4) return parts_lds(r.at + lane_off + off);
        const uint32_t a = r.even + lane_off + off;
        return __funnelshift_r(parts_lds(a), parts_lds(a + 4), r.even_sh);
    }
    const uint32_t a = (W4 ? r.at : r.odd) + lane_off + off - 2;
    return __funnelshift_r(parts_lds(a), parts_lds(a + 4), W4 ? 16u : r.odd_sh);
}

// d += a . b, 16 x 8 x 16, bf16 operands and f32 sums
__device__ __forceinline__ void parts_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t parts_sub(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// (v & mask) | bits
__device__ __forceinline__ uint32_t parts_pick(uint32_t v, uint32_t mask, uint32_t bits) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(v), "r"(mask), "r"(bits));
    return d;
}
constexpr uint32_t kBf128 = 0x43004300u;  // 128 | q is 128 + q for q < 128, as a bf16 pair

// The activations of a warp's 256 columns: 16-byte entries {b0, b1 of a 32-column block's first step, b0, b1 of its second},
// [part set][block][lane], from offset `at` on, `set` bytes from one part set to the next.
struct PartsX { uint32_t at, set; };
template <int NP> struct PartsB { uint4 v[NP]; };
template <int NP> __device__ __forceinline__ PartsB<NP> parts_load(const PartsX& X, uint32_t block) {
    PartsB<NP> b;
#pragma unroll
    for (int p = 0; p < NP; ++p) b.v[p] = parts_lds4(X.at + p * X.set + block * 512u);
    return b;
}
// A block's two steps of one scale: small parts first, so that only the last products are added at the sums' full size.
template <int NP>
__device__ __forceinline__ void parts_multiply(const PartsB<NP>& b, const uint32_t (&a)[2][4], float (&acc)[4]) {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll
    for (int p = NP - 1; p >= 0; --p) {
        parts_mma(acc, a[0], b.v[p].x, b.v[p].y);
        parts_mma(acc, a[1], b.v[p].z, b.v[p].w);
    }
}
// One step, S of the block's two.
template <int NP, int S>
__device__ __forceinline__ void parts_multiply1(const PartsB<NP>& b, const uint32_t (&a)[4], float (&acc)[4]) {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll
    for (int p = NP - 1; p >= 0; --p) parts_mma(acc, a, S ? b.v[p].z : b.v[p].x, S ? b.v[p].w : b.v[p].y);
}
__device__ __forceinline__ void parts_scale(float (&tot)[4], const float (&acc)[4], float sa, float sb) {
    tot[0] = fmaf(acc[0], sa, tot[0]); tot[1] = fmaf(acc[1], sa, tot[1]);
    tot[2] = fmaf(acc[2], sb, tot[2]); tot[3] = fmaf(acc[3], sb, tot[3]);
}
// A step's scales are added in N totals, which are then added pairwise: one chain through all of them left a fifth more error.
template <int N> __device__ __forceinline__ void parts_join(float (&tot)[4], float (&sum)[N][4]) {
#pragma unroll
    for (int d = N / 2; d >= 1; d /= 2)
#pragma unroll
        for (int i = 0; i < d; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[i][j] += sum[i + d][j];
#pragma unroll
    for (int j = 0; j < 4; ++j) tot[j] += sum[0][j];
}

// One step of a warp: rows lane / 4 (ra) and lane / 4 + 8 (rb) of the tile; `blocks` of its 32-column blocks exist.
template <uint32_t SCHEME, int NP, bool W4> struct PartsStep;

template <int NP, bool W4> struct PartsStep<RLXQ_Q4_0, NP, W4> {
    __device__ static __forceinline__ void run(PartsRow ra, PartsRow rb, uint32_t lane, const PartsX& X, uint32_t, uint32_t blocks, float (&tot)[4]) {
        const uint32_t t4 = 4 * (lane & 3u);
        float sum[2][4] = {};
#pragma unroll 2
        for (uint32_t b0 = 0; b0 < blocks; b0 += 2) {
#pragma unroll
            for (uint32_t b = 0; b < 2; ++b) {
                if (b && b0 + 1 >= blocks) break;
                const PartsB<NP> x = parts_load<NP>(X, b0 + b);
                uint32_t a[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t q = parts_word<W4>(h ? rb : ra, t4, 18 * b + 2);
                    a[0][h] = parts_sub(parts_pick(q, 0x000F000Fu, kBf128), 0x43084308u);
                    a[0][2 + h] = parts_sub(parts_pick(q >> 8, 0x000F000Fu, kBf128), 0x43084308u);
                    a[1][h] = parts_sub(parts_pick(q >> 4, 0x000F000Fu, kBf128), 0x43084308u);
                    a[1][2 + h] = parts_sub(parts_pick(q >> 12, 0x000F000Fu, kBf128), 0x43084308u);
                }
                const float da = f16_bits_to_f32(parts_lds16(ra.at + 18 * b)), db = f16_bits_to_f32(parts_lds16(rb.at + 18 * b));
                float acc[4];
                parts_multiply<NP>(x, a, acc);
                parts_scale(sum[b], acc, da, db);
            }
            ra.move(36);
            rb.move(36);
        }
        parts_join<2>(tot, sum);
    }
};

template <int NP, bool W4> struct PartsStep<RLXQ_Q8_0, NP, W4> {
    // an int8 is its low seven bits less 128 where the eighth is set: (128 + low) - (128 or 256), both exact in bf16
    __device__ static __forceinline__ uint32_t pair(uint32_t q) {
        return parts_sub(parts_pick(q, 0x007F007Fu, kBf128), parts_pick(q, 0x00800080u, kBf128));
    }
    __device__ static __forceinline__ void run(PartsRow ra, PartsRow rb, uint32_t lane, const PartsX& X, uint32_t part, uint32_t blocks, float (&tot)[4]) {
        const uint32_t t8 = 8 * (lane & 3u), lim = min(blocks, 4 * part + 4);
        float sum[2][4] = {};
#pragma unroll 2
        for (uint32_t b0 = 4 * part; b0 < lim; b0 += 2) {
#pragma unroll
            for (uint32_t b = 0; b < 2; ++b) {
                if (b && b0 + 1 >= blocks) break;
                const PartsB<NP> x = parts_load<NP>(X, b0 + b);
                uint32_t a[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const PartsRow& r = h ? rb : ra;
                    const uint32_t off = 34 * b + 2;
                    uint32_t q[2];
                    if (W4 && off % 4 == 0) {
                        q[0] = parts_lds(r.at + t8 + off);
                        q[1] = parts_lds(r.at + t8 + off + 4);
                    } else {
                        const uint32_t at = off % 4 ? (W4 ? r.at : r.odd) + off - 2 : r.even + off, sh = off % 4 ? (W4 ? 16u : r.odd_sh) : r.even_sh;
                        const uint32_t w0 = parts_lds(at + t8), w1 = parts_lds(at + t8 + 4), w2 = parts_lds(at + t8 + 8);
                        q[0] = __funnelshift_r(w0, w1, sh);
                        q[1] = __funnelshift_r(w1, w2, sh);
                    }
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        a[s][h] = pair(q[s]);
                        a[s][2 + h] = pair(q[s] >> 8);
                    }
                }
                const float da = f16_bits_to_f32(parts_lds16(ra.at + 34 * b)), db = f16_bits_to_f32(parts_lds16(rb.at + 34 * b));
                float acc[4];
                parts_multiply<NP>(x, a, acc);
                parts_scale(sum[b], acc, da, db);
            }
            ra.move(68);
            rb.move(68);
        }
        parts_join<2>(tot, sum);
    }
};

// Q6_K (ql[128] | qh[64] | sc[16] i8 | d f16, order as rlx-gguf/src/lib.rs:1070-1114): weights 128 h + 32 g + 16 i .. of the
// super-block are nibble g >> 1 of ql bytes 64 h + 32 (g & 1) + 16 i .. and bits 2 g, 2 g + 1 of qh bytes 32 h + 16 i .., with
// scale 8 h + 2 g + i.  Lane t unpacks scales 4 t .. 4 t + 3.
template <int NP, bool W4> struct PartsStep<RLXQ_Q6_K, NP, W4> {
    __device__ static __forceinline__ void scales(const PartsRow& r, uint32_t t, float (&s)[4]) {
        const uint32_t u = parts_word<W4>(r, 4 * t, 192) ^ 0x80808080u;
        const float d = f16_bits_to_f32(parts_lds16(r.at + 208));
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = d * (__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7440 + i)) - (8388608.0f + 128.0f));
    }
    __device__ static __forceinline__ void run(PartsRow ra, PartsRow rb, uint32_t lane, const PartsX& X, uint32_t, uint32_t, float (&tot)[4]) {
        const uint32_t t = lane & 3u, t4 = 4 * t;
        float sa[4], sb[4];
        scales(ra, t, sa);
        scales(rb, t, sb);
        PartsRow ha = ra, hb = rb;        // (qh advances by half the bytes)
        ha.move(128);
        hb.move(128);
        float sum[4][4] = {};
#pragma unroll 1
        for (uint32_t h = 0; h < 2; ++h) {
            uint32_t qh[2][2], ql[2][2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    qh[i][r] = parts_word<W4>(r ? hb : ha, t4, 16 * i);
                    ql[i][r][0] = parts_word<W4>(r ? rb : ra, t4, 16 * i);
                    ql[i][r][1] = parts_word<W4>(r ? rb : ra, t4, 32 + 16 * i);
                }
#pragma unroll
            for (uint32_t g = 0; g < 4; ++g) {
                const PartsB<NP> x = parts_load<NP>(X, 4 * h + g);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t a[4];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint32_t l = ql[i][r][g & 1u], u = qh[i][r];
                        uint32_t v0 = parts_pick(l >> (4 * (g >> 1)), 0x000F000Fu, kBf128), v1 = parts_pick(l >> (8 + 4 * (g >> 1)), 0x000F000Fu, kBf128);
                        v0 = parts_pick(g < 2 ? u << (4 - 2 * g) : u >> (2 * g - 4), 0x00300030u, v0);
                        v1 = parts_pick(u >> (2 * g + 4), 0x00300030u, v1);
                        a[r] = parts_sub(v0, 0x43204320u);           // less 128 + 32
                        a[2 + r] = parts_sub(v1, 0x43204320u);
                    }
                    const uint32_t s = 2 * g + i, from = (lane & 28u) | (2 * h + (s >> 2));
                    float acc[4];
                    if (i) parts_multiply1<NP, 1>(x, a, acc);
                    else parts_multiply1<NP, 0>(x, a, acc);
                    parts_scale(sum[s & 3u], acc, __shfl_sync(0xFFFFFFFFu, sa[s & 3u], from), __shfl_sync(0xFFFFFFFFu, sb[s & 3u], from));
                }
            }
            ra.move(64); rb.move(64);
            ha.move(32); hb.move(32);
        }
        parts_join<4>(tot, sum);
    }
};

// f = hi + mid + lo, the upper eight bits of the significand, the next and the last: exact.  Infinities and NaN are hi alone.
struct Parts3 { float hi, mid, lo; };
__device__ __forceinline__ Parts3 parts_split(float f) {
    Parts3 p;
    const uint32_t u = __float_as_uint(f);
    p.hi = __uint_as_float(u & 0xFFFF0000u);
    float r = f - p.hi;
    if ((u & 0x7F800000u) == 0x7F800000u) {
        if (f != f) p.hi = __uint_as_float(0x7FC00000u);
        r = 0.f;
    }
    p.mid = __uint_as_float(__float_as_uint(r) & 0xFFFF0000u);
    p.lo = r - p.mid;
    return p;
}
// upper halves of two floats as a bf16 pair, the first low
__device__ __forceinline__ uint32_t parts_pack(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }

// The B operand pairs of two activations, one for each part (NP = 1: bf16 activations, which are their own first part).
template <int NP> __device__ __forceinline__ void parts_operands(float a, float b, uint32_t (&o)[NP]) {
    if constexpr (NP == 1) {
        o[0] = parts_pack(a, b);
    } else {
        const Parts3 p = parts_split(a), q = parts_split(b);
        o[0] = parts_pack(p.hi, q.hi);
        o[1] = parts_pack(p.mid, q.mid);
        o[2] = parts_pack(p.lo, q.lo);
    }
}

template <uint32_t SCHEME, int NP, bool W4>
__global__ void __launch_bounds__(kPartsMaxWarps * 32, 1) gemv_parts_kernel(const __grid_constant__ PartsParams P) {
    using G = PartsGeom<SCHEME>;
    constexpr uint32_t STEP = kPartsTile * G::SLOT;
    constexpr int COPIES = (int)((G::PIECE + 14 + 15) / 16 + 1) / 2;           // of sixteen bytes: two lanes copy a row
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nw = P.nw, D = P.depth;
    const uint32_t stream = warp / nw, cw = warp - stream * nw;                    // this warp's stream and place in it
    const uint32_t ring = P.off_ring + warp * (D * STEP), ring_u32 = smem_u32(parts_smem) + ring;
    float* red = reinterpret_cast<float*>(parts_smem + P.off_red) + stream * (2 * nw * 128u);      // [streams][2][nw][16][8]
    float* total = reinterpret_cast<float*>(parts_smem + P.off_total);             // [tiles of a chunk][16][8]
    griddep_launch_dependents();

    const uint32_t cta = blockIdx.x;
    const uint32_t t0 = (uint32_t)((uint64_t)cta * P.tiles / P.ctas), t1 = (uint32_t)((uint64_t)(cta + 1) * P.tiles / P.ctas);
    const uint8_t* const w = P.w;
    // Order of a warp's steps: chunks of tiles, in each the column passes, in each its stream's tiles, in each its pieces.
    const uint32_t chunk_tiles = P.passes > 1 ? kPartsTotals : t1 - t0;
    const uint32_t crow = lane >> 1, chalf = lane & 1u;
    struct Next { uint32_t c0, pass, tile, part; } nx{t0, 0, t0 + stream, 0};
    auto fetch = [&](uint32_t slot) {     // the next step, if there is one
        while (nx.c0 < t1 && nx.tile >= min(t1, nx.c0 + chunk_tiles)) {
            if (++nx.pass == P.passes) { nx.pass = 0; nx.c0 += chunk_tiles; }
            nx.tile = nx.c0 + stream;
        }
        if (nx.c0 < t1) {
            const uint64_t off = (uint64_t)(nx.pass * nw + cw) * (G::PIECE * G::PER) + nx.part * G::PIECE;
            const uint32_t row = nx.tile * kPartsTile + crow;
            if (off < P.row_bytes && row < P.n) {
                const uint8_t* src = w + (uint64_t)row * P.row_bytes + off;
                const uint32_t lead = (uint32_t)((uintptr_t)src & 15u);
                const uint32_t chunks = (lead + (uint32_t)min((uint64_t)G::PIECE, P.row_bytes - off) + 15u) / 16u;
                const uint8_t* from = src - lead + 16 * chalf;
                const uint32_t to = ring_u32 + slot * STEP + crow * G::SLOT + 16 * chalf;
#pragma unroll
                for (int c = 0; c < COPIES; ++c)
                    if (2 * c + chalf < chunks) parts_copy16(to + 32 * c, from + 32 * c);
            }
            if (++nx.part == G::PER) { nx.part = 0; nx.tile += P.streams; }
        }
        parts_commit();
    };
    uint32_t slot_in = 0, slot = 0;
#pragma unroll 1
    for (uint32_t s = 0; s + 1 < D; ++s) {
        fetch(slot_in);
        if (++slot_in == D) slot_in = 0;
    }
    griddep_wait();                       // the weights are on their way; x and y belong to the kernel in front until here

    const uint32_t col = lane >> 2, t = lane & 3u;
    const bool have_row = col < P.m;      // (columns past the last row are zero)
    PartsX X;
    X.set = nw * (8u * 512u);
    X.at = cw * (8u * 512u) + lane * 16u;
    for (uint32_t c0 = t0; c0 < t1; c0 += chunk_tiles) {
        const uint32_t c1 = min(t1, c0 + chunk_tiles);
        for (uint32_t pass = 0; pass < P.passes; ++pass) {
            const uint32_t first = (pass * nw + cw) * kPartsCols;
            const uint32_t blocks = first < P.k ? min(kPartsCols, P.k - first) / 32 : 0u;
            // ---- the activations of this pass, a 32-column block at a time ----
            if (pass || c0 != t0) __syncthreads();            // (everybody has multiplied by the last pass's)
            if (c0 == t0 || P.passes > 1) {
                const uint32_t nwarps = nw * P.streams;
                constexpr uint32_t STEP_COLS = SCHEME == RLXQ_Q4_0 || SCHEME == RLXQ_Q6_K ? 16 : 4, LANE_COLS = SCHEME == RLXQ_Q4_0 || SCHEME == RLXQ_Q6_K ? 4 : 8;
                constexpr uint32_t BATCH = 4;                 // blocks whose loads are in flight together
                for (uint32_t b0 = warp; b0 < 8 * nw; b0 += BATCH * nwarps) {
                    uint4 raw[BATCH][2];
#pragma unroll
                    for (uint32_t q = 0; q < BATCH; ++q) {
                        const uint32_t c = (pass * nw * 8 + b0 + q * nwarps) * 32 + LANE_COLS * t;
                        const bool in = have_row && c < P.k && b0 + q * nwarps < 8 * nw;
                        raw[q][0] = raw[q][1] = make_uint4(0u, 0u, 0u, 0u);
                        if constexpr (NP == 1) {
                            const uint16_t* src = reinterpret_cast<const uint16_t*>(P.x) + (size_t)col * P.k + c;
                            if (in) {
                                const uint2 u = *reinterpret_cast<const uint2*>(src), v = *reinterpret_cast<const uint2*>(src + STEP_COLS);
                                raw[q][0] = make_uint4(u.x, u.y, v.x, v.y);
                            }
                        } else {
                            const float* src = reinterpret_cast<const float*>(P.x) + (size_t)col * P.k + c;
                            if (in) { raw[q][0] = *reinterpret_cast<const uint4*>(src); raw[q][1] = *reinterpret_cast<const uint4*>(src + STEP_COLS); }
                        }
                    }
#pragma unroll
                    for (uint32_t q = 0; q < BATCH; ++q) {
                        const uint32_t b = b0 + q * nwarps;
                        if (b >= 8 * nw) break;
                        float f[8];
                        if constexpr (NP == 1) {
                            const uint32_t r[4] = {raw[q][0].x, raw[q][0].y, raw[q][0].z, raw[q][0].w};
#pragma unroll
                            for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(r[i] << 16); f[2 * i + 1] = __uint_as_float(r[i] & 0xFFFF0000u); }
                        } else {
                            const uint32_t r[8] = {raw[q][0].x, raw[q][0].y, raw[q][0].z, raw[q][0].w, raw[q][1].x, raw[q][1].y, raw[q][1].z, raw[q][1].w};
#pragma unroll
                            for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(r[i]);
                        }
                        uint32_t o[4][NP];
                        parts_operands<NP>(f[0], f[2], o[0]);
                        parts_operands<NP>(f[1], f[3], o[1]);
                        parts_operands<NP>(f[4], f[6], o[2]);
                        parts_operands<NP>(f[5], f[7], o[3]);
#pragma unroll
                        for (int p = 0; p < NP; ++p) *reinterpret_cast<uint4*>(parts_smem + p * X.set + b * 512u + lane * 16u) = make_uint4(o[0][p], o[1][p], o[2][p], o[3][p]);
                    }
                }
                __syncthreads();
            }
            // where the warp's pieces of rows lane / 4 and lane / 4 + 8 begin behind the copies' boundary: the same in every tile
            const uint64_t at = (uint64_t)(uintptr_t)w + (uint64_t)(c0 * kPartsTile) * P.row_bytes + (uint64_t)(pass * nw + cw) * (G::PIECE * G::PER);
            const uint32_t row_a = (uint32_t)at + col * (uint32_t)P.row_bytes, row_b = row_a + 8 * (uint32_t)P.row_bytes;
            uint32_t turn = 0;
#pragma unroll 1
            for (uint32_t tile = c0 + stream; tile < c1; tile += P.streams, turn ^= 1u) {
                float tot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
                for (uint32_t part = 0; part < G::PER; ++part) {
                    if (D == 2) parts_wait<0>();
                    else if (D == 3) parts_wait<1>();
                    else parts_wait<2>();
                    __syncwarp();         // every lane's copies of this step have landed, and the slot refilled below is read
                    const uint32_t base = ring + slot * STEP + col * G::SLOT;
                    if (blocks) {
                        const PartsRow ra(base + ((row_a + part * G::PIECE) & 15u)), rb(base + 8 * G::SLOT + ((row_b + part * G::PIECE) & 15u));
                        PartsStep<SCHEME, NP, W4>::run(ra, rb, lane, X, part, blocks, tot);
                    }
                    fetch(slot_in);
                    if (++slot_in == D) slot_in = 0;
                    if (++slot == D) slot = 0;
                }
                float* mine = red + (turn * nw + cw) * 128u + col * 8u + 2u * t;
                *reinterpret_cast<float2*>(mine) = make_float2(tot[0], tot[1]);
                *reinterpret_cast<float2*>(mine + 64) = make_float2(tot[2], tot[3]);
                // the stream's warps meet (the buffers alternate: the next tile writes the other one)
                asm volatile("bar.sync %0, %1;" ::"r"(1u + stream), "r"(nw * 32u) : "memory");
                // four rows a warp: lane = (row, column)
                for (uint32_t i0 = 4 * cw; i0 < kPartsTile; i0 += 4 * nw) {
                    const uint32_t i = i0 + (lane >> 3), c = lane & 7u;
                    const float* src = red + turn * nw * 128u + i * 8u + c;
                    float part[4] = {0.f, 0.f, 0.f, 0.f};
                    for (uint32_t q = 0; q < nw; q += 4)
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j)
                            if (q + j < nw) part[j] += src[(q + j) * 128u];
                    float v = (part[0] + part[2]) + (part[1] + part[3]);
                    if (c >= P.m) continue;
                    if (P.passes > 1) {
                        float* sum = total + ((tile - c0) * kPartsTile + i) * 8u + c;
                        if (pass) v += *sum;
                        if (pass + 1 < P.passes) { *sum = v; continue; }
                    }
                    const uint32_t orow = tile * kPartsTile + i;
                    if (orow >= P.n) continue;
                    const size_t out = (size_t)c * P.n + orow;
                    if (P.y_bf16) reinterpret_cast<uint16_t*>(P.y)[out] = (uint16_t)f32_to_bf16_bits(v);
                    else reinterpret_cast<float*>(P.y)[out] = v;
                }
            }
        }
    }
}

// The split of k x n weights: sets P's work split and shared-memory layout, returns the bytes of shared memory.  As few passes as
// leave every warp a ring of two steps at least, with as many streams as sixteen warps make.
template <uint32_t SCHEME> static uint32_t plan_parts(PartsParams& P, uint32_t np) {
    const uint32_t pieces = (P.k + kPartsCols - 1) / kPartsCols;
    P.tiles = (P.n + kPartsTile - 1) / kPartsTile;
    const uint32_t sms = (uint32_t)sm_count();                // one CTA per SM
    P.ctas = sms < P.tiles ? sms : P.tiles;
    const uint32_t most = (P.tiles + P.ctas - 1) / P.ctas;    // tiles of a CTA
    for (P.passes = (pieces + kPartsMaxWarps - 1) / kPartsMaxWarps;; ++P.passes) {
        P.nw = (pieces + P.passes - 1) / P.passes;
        P.streams = std::min({kPartsMaxWarps / P.nw, most, 15u});      // (a named barrier each, of fifteen)
        const uint32_t warps = P.nw * P.streams, step = warps * kPartsTile * PartsGeom<SCHEME>::SLOT;
        P.off_ring = np * P.nw * (8u * 512u);
        const uint32_t red = warps * (2u * 512u), totals = P.passes > 1 ? std::min(most, kPartsTotals) * kPartsTile * 8u * 4u : 0u;
        if (P.off_ring + red + totals + 2 * step <= 227u * 1024u) {
            P.depth = std::min(4u, (227u * 1024u - P.off_ring - red - totals) / step);
            P.off_red = P.off_ring + P.depth * step;
            P.off_total = P.off_red + red;
            return P.off_total + totals;
        }
    }
}

template <uint32_t SCHEME, int NP, bool W4>
static int launch_parts_t(cudaStream_t stream, PartsParams P) {
    const uint32_t smem = plan_parts<SCHEME>(P, NP), warps = P.nw * P.streams;
    static std::atomic<uint32_t> attr_set[64];
    int dev = 0;
    RLXQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && attr_set[dev].load() == 0) {
        RLXQ_CUDA_TRY(cudaFuncSetAttribute(gemv_parts_kernel<SCHEME, NP, W4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        attr_set[dev].store(1);
    }
    int rc = launch_pdl(gemv_parts_kernel<SCHEME, NP, W4>, dim3(P.ctas), dim3(warps * 32), smem, stream, P);
    if (rc) return rc;
    count_launch();
    return check_launch("gemv_parts_kernel");
}
template <uint32_t SCHEME>
static int launch_parts_s(cudaStream_t stream, const PartsParams& P, bool xbf) {
    if constexpr (SCHEME != RLXQ_Q6_K)    // (210 bytes: every other super-block is two bytes off a word)
        if ((uintptr_t)P.w % 4 == 0 && P.row_bytes % 4 == 0) return xbf ? launch_parts_t<SCHEME, 1, true>(stream, P) : launch_parts_t<SCHEME, 3, true>(stream, P);
    return xbf ? launch_parts_t<SCHEME, 1, false>(stream, P) : launch_parts_t<SCHEME, 3, false>(stream, P);
}

// Microseconds, this kernel (a call, a column pass, a pass of one stream, a tile of a stream and pass, and for each of a CTA's warps)
// and the f32 kernel (a call, a row of a CTA and pass, and for sixteen warps of them): fits to 1900 calls of batch 5 to 8, both timed.
struct PartsCost { float call, pass, alone, tile, warp, f32_call, f32_row, f32_warps; };
template <uint32_t SCHEME> static bool parts_is_faster(uint32_t k, uint32_t n, bool xbf) {
    const PartsCost c = SCHEME == RLXQ_Q4_0   ? (xbf ? PartsCost{0.46f, 1.20f, -0.06f, 1.13f, 0.11f, 1.74f, 0.18f, 0.31f} : PartsCost{0.62f, 0.66f, 2.52f, 0.35f, 0.19f, 2.51f, 0.18f, 0.33f})
                        : SCHEME == RLXQ_Q8_0 ? (xbf ? PartsCost{-0.26f, 2.20f, -0.61f, 1.49f, 0.16f, 1.64f, 0.18f, 0.35f} : PartsCost{0.72f, 0.34f, 2.80f, 0.30f, 0.29f, 2.34f, 0.17f, 0.37f})
                                              : (xbf ? PartsCost{-0.03f, 2.30f, -0.52f, 0.98f, 0.18f, 1.66f, 0.23f, 0.37f} : PartsCost{0.90f, 1.04f, 2.22f, 0.34f, 0.25f, 2.51f, 0.20f, 0.42f});
    PartsParams P{};
    P.k = k; P.n = n;
    plan_parts<SCHEME>(P, xbf ? 1 : 3);
    const uint32_t most = (P.tiles + P.ctas - 1) / P.ctas;
    const float passes = (float)P.passes, rounds = passes * (float)((most + P.streams - 1) / P.streams);
    const float parts = c.call + passes * (c.pass + c.alone / (float)P.streams) + rounds * (c.tile + c.warp * (float)(P.nw * P.streams));
    // gemv_f32.cu with four activation rows: 512 columns a warp, sixteen warps an SM, half of the CTAs for either four rows, two
    // weight rows a step
    const uint32_t pieces = (k + 511) / 512, f32_passes = (pieces + 15) / 16, warps = (pieces + f32_passes - 1) / f32_passes;
    const uint32_t per_sm = 16 / warps, tiles = std::max(1u, (uint32_t)sm_count() * per_sm / 2), rows = ((n + tiles - 1) / tiles + 1) / 2 * 2;
    const float f32 = c.f32_call + (float)f32_passes * (float)rows * (c.f32_row + c.f32_warps * (float)(warps * per_sm) / 16.0f);
    return parts < f32;
}

// Five to eight rows where this kernel is the faster one.  Rows of up to 1024 weights: from 2 M weights on, where the two are level
// (2.3 M: Q8_0 1.04 to 1.11 of the f32 kernel's time with f32 activations; 2.9 M: 0.74 to 0.91).  Longer rows: by the estimate,
// because what a column pass or a second tile of a few CTAs costs depends on the split; with the weight count alone one call in
// 27 was slower than the f32 kernel, up to 1.30 times (Q6_K 3840 x 2410 f32, 13.2 and 16.4 us), now one in 160, 1.11 at worst, of 2934.
bool gemv_parts_pays(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, bool xbf, const void* x) {
    const bool known = scheme == RLXQ_Q4_0 || scheme == RLXQ_Q8_0 || scheme == RLXQ_Q6_K;
    if (!known || m < 5 || m > 8 || ((uintptr_t)x & 15u) || k % 32 || k == 0) return false;
    const uint64_t cols = xbf ? 4096 : 2048, passes = (k + cols - 1) / cols;
    if ((uint64_t)k * n <= 2000000ull + 5500000ull * (passes - 1)) return false;      // (too few to be asked about)
    if (k <= 1024) return true;
    switch (scheme) {
        case RLXQ_Q4_0: return parts_is_faster<RLXQ_Q4_0>(k, n, xbf);
        case RLXQ_Q8_0: return parts_is_faster<RLXQ_Q8_0>(k, n, xbf);
        default: return parts_is_faster<RLXQ_Q6_K>(k, n, xbf);
    }
}

int launch_gemv_parts(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y, bool ybf, uint32_t m,
                      uint32_t k, uint32_t n) {
    Geometry g;
    if (!geometry(scheme, &g)) return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    PartsParams P{};
    P.x = x; P.w = w; P.y = y; P.y_bf16 = ybf; P.m = m; P.k = k; P.n = n;
    P.row_bytes = (uint64_t)k / g.elems * g.bytes;
    switch (scheme) {
        case RLXQ_Q4_0: return launch_parts_s<RLXQ_Q4_0>(stream, P, xbf);
        case RLXQ_Q8_0: return launch_parts_s<RLXQ_Q8_0>(stream, P, xbf);
        case RLXQ_Q6_K: return launch_parts_s<RLXQ_Q6_K>(stream, P, xbf);
        default: return fail(RLXQ_E_SCHEME, "no streaming GEMV in parts for scheme %u", scheme);
    }
}

}  // namespace rlxq
