// The SwiGLU gate: out = up * silu(gate), silu(x) = x / (1 + exp(-x))
// (rlx-cpu/src/naive.rs:54-56; composition rlx-cuda/src/unfuse.rs:254-293).
#include "common.cuh"
#include "decode.cuh"
#include "host/session.hpp"
#include "kernels.h"
#include "staged_common.cuh"

namespace rlxq {

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }

__global__ void __launch_bounds__(256) swiglu_mul_kernel(const float* __restrict__ gate,
                                                         const float* __restrict__ up,
                                                         float* __restrict__ out, uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = up[i] * silu_f(gate[i]);
}

int launch_swiglu_mul(cudaStream_t stream, const float* gate, const float* up, float* out, uint64_t n) {
    if (n == 0) return RLXQ_OK;
    uint64_t blocks = (n + 255) / 256;
    const uint64_t cap = (uint64_t)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    swiglu_mul_kernel<<<(unsigned)blocks, 256, 0, stream>>>(gate, up, out, n);
    count_launch();
    return check_launch("swiglu_mul_kernel");
}

// Byte copy between a pinned host staging buffer and device memory (either direction), both 16-byte
// aligned.  A session in graph mode uses it for activations and outputs of a few KB: a kernel node
// starts sooner than a copy-engine node, and the bytes cross PCIe as plain loads / posted stores.
// Launched with programmatic stream serialization: the kernel behind an input copy becomes resident and
// requests its first weights while the input crosses PCIe, and an output copy is resident, waiting, when
// the kernel in front of it completes.
__global__ void __launch_bounds__(256) copy_bytes_kernel(uint8_t* __restrict__ dst, const uint8_t* src,
                                                         uint64_t bytes) {
    griddep_launch_dependents();
    griddep_wait();                // every thread: whoever waits for this kernel has then waited for its predecessors
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t n16 = bytes / 16;
    for (uint64_t i = tid; i < n16; i += stride)
        reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    for (uint64_t i = n16 * 16 + tid; i < bytes; i += stride) dst[i] = src[i];
}

int launch_copy_bytes(cudaStream_t stream, void* dst, const void* src, uint64_t bytes) {
    if (bytes == 0) return RLXQ_OK;
    if (((uintptr_t)dst | (uintptr_t)src) & 15u) return fail(RLXQ_E_ALIGN, "copy_bytes: buffers must be 16-byte aligned");
    uint64_t blocks = (bytes / 16 + 255) / 256;
    if (blocks == 0) blocks = 1;
    if (blocks > 64) blocks = 64;
    int rc = launch_pdl(copy_bytes_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, (uint8_t*)dst, (const uint8_t*)src, bytes);
    if (rc) return rc;
    count_launch();
    return check_launch("copy_bytes_kernel");
}

// f32 activations for the tensor-core GEMM, whose operands are bf16 (split_bf16x4): x = hi + lo, which leaves 2^-17 of x behind,
// or (parts = 3) x = hi + mid + lo, which leaves nothing.  Rows [0, rows) of x become rows [0, rows) (hi), [rows, 2 rows) and, if
// asked for, [2 rows, 3 rows) of `out`; the GEMM multiplies all of them by the same decoded weights.  One pass of 8 bytes a
// value, a few microseconds; the GEMM behind it is resident meanwhile and fetches its first weights.
__global__ void __launch_bounds__(256) split_hi_lo_kernel(const float* x, uint16_t* __restrict__ out,
                                                          uint64_t rows, uint64_t k, uint32_t parts) {
    const uint64_t total = rows * k / 4, stride = (uint64_t)gridDim.x * blockDim.x;     // k % 4 == 0
    griddep_launch_dependents();
    griddep_wait();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const float4 v = reinterpret_cast<const float4*>(x)[i];
        const float f[4] = {v.x, v.y, v.z, v.w};
        uint32_t h[4], l[4], e[4];
        split_bf16x4(f, h, l, e);
        reinterpret_cast<uint2*>(out)[i] = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
        reinterpret_cast<uint2*>(out + rows * k)[i] = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
        if (parts == 3) reinterpret_cast<uint2*>(out + 2 * rows * k)[i] = make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
    }
}

int launch_split_hi_lo(cudaStream_t stream, const float* x, void* out, uint64_t rows, uint64_t k, uint32_t parts) {
    if (rows == 0 || k == 0) return RLXQ_OK;
    uint64_t blocks = (rows * k / 4 + 255) / 256;
    const uint64_t cap = (uint64_t)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    int rc = launch_pdl(split_hi_lo_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, x, reinterpret_cast<uint16_t*>(out), rows, k, parts);
    if (rc) return rc;
    count_launch();
    return check_launch("split_hi_lo_kernel");
}

// y[i] = the sum over s, in order, of part[s * stride + i]: the k slices of a GEMM with few tiles, or (two "slices") the
// hi and lo results of f32 activations.  Every slice's value is loaded before the first is added; out of L2.
template <bool VEC>
__global__ void __launch_bounds__(256) add_slices_kernel(const float* part, uint32_t slices, uint64_t stride,
                                                         void* __restrict__ y, uint32_t y_bf16, uint64_t total) {
    constexpr uint32_t W = VEC ? 4 : 1, kAtOnce = 8;
    griddep_launch_dependents();
    griddep_wait();
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total / W; i += step) {
        float acc[W];
#pragma unroll
        for (uint32_t q = 0; q < W; ++q) acc[q] = 0.f;
        for (uint32_t s0 = 0; s0 < slices; s0 += kAtOnce) {
            float v[kAtOnce][W];
#pragma unroll
            for (uint32_t s = 0; s < kAtOnce; ++s) {
                if (s0 + s >= slices) continue;
                const float* p = part + (s0 + s) * stride + i * W;
                if constexpr (VEC) {
                    const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
                    v[s][0] = t.x; v[s][1] = t.y; v[s][2] = t.z; v[s][3] = t.w;
                } else {
                    v[s][0] = __ldcg(p);
                }
            }
#pragma unroll
            for (uint32_t s = 0; s < kAtOnce; ++s)
                if (s0 + s < slices)
#pragma unroll
                    for (uint32_t q = 0; q < W; ++q) acc[q] = s0 + s == 0 ? v[s][q] : acc[q] + v[s][q];
        }
        if (y_bf16) {
            uint32_t b[W];
#pragma unroll
            for (uint32_t q = 0; q < W; ++q) b[q] = f32_to_bf16_bits(acc[q]) & 0xFFFFu;
            if constexpr (VEC) reinterpret_cast<uint2*>(y)[i] = make_uint2(b[0] | (b[1] << 16), b[2] | (b[3] << 16));
            else reinterpret_cast<uint16_t*>(y)[i] = (uint16_t)b[0];
        } else {
            if constexpr (VEC) reinterpret_cast<float4*>(y)[i] = make_float4(acc[0], acc[1], acc[2], acc[3]);
            else reinterpret_cast<float*>(y)[i] = acc[0];
        }
    }
}

int launch_add_slices(cudaStream_t stream, const float* part, uint32_t slices, uint64_t stride, void* y, bool ybf, uint64_t total) {
    if (total == 0) return RLXQ_OK;
    const bool vec = total % 4 == 0 && stride % 4 == 0 && !(((uintptr_t)y | (uintptr_t)part) & 15u);
    uint64_t blocks = (total / (vec ? 4 : 1) + 255) / 256;
    const uint64_t cap = (uint64_t)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    int rc = launch_pdl(vec ? add_slices_kernel<true> : add_slices_kernel<false>, dim3((unsigned)blocks), dim3(256), 0, stream, part, slices,
                        stride, y, ybf ? 1u : 0u, total);
    if (rc) return rc;
    count_launch();
    return check_launch("add_slices_kernel");
}

// Packed weight rows of any (even) length on a pitch that TMA can tile: row r moves from byte r * row_bytes to byte
// r * pitch, zeros behind it (a zero block decodes to zeros).  Rows start on any even byte, so a 4-byte word of the
// result is two halves of neighbouring source words; a warp reads its 1 KB piece of a row in eight coalesced loads,
// all in flight together, and takes the neighbour's word by shuffle.  HBM-bound: one read and one write of the weights
// (the write mostly stays in L2 for the GEMM behind it).
// used (expert stacks; may be null): slab s of slab_rows rows is skipped when used[s + 1] == used[s].
__global__ void __launch_bounds__(256) relay_rows_kernel(const uint8_t* __restrict__ w, uint64_t row_bytes, uint64_t n,
                                                         uint8_t* __restrict__ out, uint64_t pitch,
                                                         const uint32_t* used, uint32_t slab_rows) {
    constexpr uint32_t kSeg = 1024;
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t segs = (uint32_t)((pitch + kSeg - 1) / kSeg);
    const uint64_t items = (uint64_t)segs * n, total = row_bytes * n;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    const uintptr_t base = reinterpret_cast<uintptr_t>(w), end = base + total;
    // the 32-bit word at aligned address a: halves outside the weights read as zero
    auto word = [&](uintptr_t a) -> uint32_t {
        if (a >= base && a + 4 <= end) return __ldg(reinterpret_cast<const uint32_t*>(a));
        uint32_t v = 0u;
        if (a >= base && a + 2 <= end) v = __ldg(reinterpret_cast<const uint16_t*>(a));
        if (a + 2 >= base && a + 4 <= end) v |= (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(a + 2)) << 16;
        return v;
    };
    for (uint64_t it = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < items; it += warps) {
        const uint64_t r = items <= 0xFFFFFFFFull ? (uint32_t)it / segs : it / segs;
        const uint64_t o0 = (it - r * segs) * kSeg;                        // byte offset of the piece inside its row
        if (used) {
            const uint32_t slab = (uint32_t)(r / slab_rows);
            if (used[slab + 1] == used[slab]) continue;
        }
        const uintptr_t src = base + r * row_bytes + o0, a_first = src & ~(uintptr_t)3, a0 = a_first + 4 * lane;
        const uint32_t sh = (uint32_t)(src & 2u) * 8u;
        uint32_t v[9];
        if (a_first >= base && a_first + kSeg + 4 <= end) {                // (what lies behind the row is masked below)
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) v[i] = __ldg(reinterpret_cast<const uint32_t*>(a0 + 128 * i));
            v[8] = lane == 0 ? __ldg(reinterpret_cast<const uint32_t*>(a0 + kSeg)) : 0u;
        } else {
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) v[i] = word(a0 + 128 * i);
            v[8] = lane == 0 ? word(a0 + kSeg) : 0u;
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t up = __shfl_down_sync(0xFFFFFFFFu, v[i], 1), wrap = __shfl_sync(0xFFFFFFFFu, v[i + 1], 0);
            uint32_t q = __funnelshift_r(v[i], lane == 31u ? wrap : up, sh);
            const uint64_t o = o0 + 128 * i + 4 * lane;
            if (o + 4 > row_bytes) q = o + 2 <= row_bytes ? q & 0xFFFFu : 0u;
            if (o < pitch) *reinterpret_cast<uint32_t*>(out + r * pitch + o) = q;
        }
    }
}

int launch_relay_rows(cudaStream_t stream, const uint8_t* w, uint64_t row_bytes, uint64_t n, uint8_t* out, uint64_t pitch,
                      const uint32_t* used, uint32_t slab_rows) {
    if (n == 0 || pitch == 0) return RLXQ_OK;
    if (((uintptr_t)w & 1u) || ((uintptr_t)out & 15u) || pitch % 16 || row_bytes % 2 || row_bytes > pitch)
        return fail(RLXQ_E_ALIGN, "relay_rows: bad alignment");
    uint64_t blocks = ((pitch + 1023) / 1024 * n + 7) / 8;
    const uint64_t cap = (uint64_t)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    int rc = launch_pdl(relay_rows_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, w, row_bytes, n, out, pitch, used, slab_rows);
    if (rc) return rc;
    count_launch();
    return check_launch("relay_rows_kernel");
}

// Q6_K rows for the GEMM on f32 weights: a super-block (ql[128] | qh[64] | sc[16] | d, 210 bytes that start on any even byte)
// becomes 272 bytes, its quants 0 .. 63 one a byte in the order of the weights, then its scale bytes, and 2^12 d goes to
// d_out[group][row].  The decoders, which read a row once per tile of activations, then find whole aligned words.  A warp takes
// four super-blocks at a time, which lie one after the other whatever rows they belong to, in 16-byte loads, and picks them
// apart in shared memory, eight weights a lane.  Bound by instruction issue (78 % of the slots, 0.36 warp instructions a weight; 37 MB in
// 23 us with cold caches, where the copy above is HBM-bound).
__global__ void __launch_bounds__(256) widen_q6_kernel(const uint8_t* __restrict__ w, uint32_t groups, uint64_t n, uint8_t* __restrict__ out,
                                                       float* __restrict__ d_out, const uint32_t* used, uint32_t slab_rows) {
    constexpr uint32_t kAtOnce = 4, kChunks = (kAtOnce * 210 + 14 + 15) / 16;
    __shared__ __align__(16) uint8_t buf[8][kChunks * 16 + 16];       // (a word past the last d)
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t lane = threadIdx.x & 31u;
    uint8_t* const mine = buf[threadIdx.x >> 5];
    const uint64_t items = groups * n, step = (uint64_t)gridDim.x * (blockDim.x >> 5) * kAtOnce;
    const uintptr_t base = reinterpret_cast<uintptr_t>(w), end = base + items * 210u;
    // lane: weights 8 lane .. of the super-block = half h, group g of 32, bytes l .. l + 7 of it
    const uint32_t h = lane >> 4, g = (lane >> 2) & 3u, l = 8 * (lane & 3u);
    const uint32_t ql = 64 * h + 32 * (g & 1u) + l, qh = 128 + 32 * h + l, nib = 4 * (g >> 1);
    auto skip = [&](uint64_t it, uint32_t count) {             // nobody is routed to the slab (or to either of two)
        return used && used[(uint32_t)((it + count - 1) / groups / slab_rows) + 1] == used[(uint32_t)(it / groups / slab_rows)];
    };
    auto fetch = [&](uint64_t it, uint4 (&v)[2]) {             // a lane's two chunks of the super-blocks from `it` on
        if (it >= items) return;
        const uint32_t count = (uint32_t)min((uint64_t)kAtOnce, items - it);
        if (skip(it, count)) return;
        const uintptr_t src = base + it * 210u, a0 = src & ~(uintptr_t)15;
        const uint32_t chunks = ((uint32_t)(src - a0) + count * 210u + 15u) / 16u;
#pragma unroll
        for (uint32_t t = 0; t < 2; ++t) {
            const uintptr_t a = a0 + 16 * (lane + 32 * t);
            if (lane + 32 * t >= chunks) continue;
            if (a >= base && a + 16 <= end) {
                v[t] = __ldg(reinterpret_cast<const uint4*>(a));
            } else {                                           // the ends of the weights: what lies inside
                uint32_t q[8];
                for (uint32_t i = 0; i < 8; ++i) q[i] = a + 2 * i >= base && a + 2 * i + 2 <= end ? __ldg(reinterpret_cast<const uint16_t*>(a + 2 * i)) : 0u;
                v[t] = make_uint4(q[0] | (q[1] << 16), q[2] | (q[3] << 16), q[4] | (q[5] << 16), q[6] | (q[7] << 16));
            }
        }
    };
    uint64_t it = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kAtOnce;
    uint4 ahead[2] = {};
    fetch(it, ahead);
    for (; it < items; it += step) {
        const uint32_t count = (uint32_t)min((uint64_t)kAtOnce, items - it), lead = (uint32_t)((base + it * 210u) & 15u);
        __syncwarp();
#pragma unroll
        for (uint32_t t = 0; t < 2; ++t)
            if (lane + 32 * t < kChunks) *reinterpret_cast<uint4*>(mine + 16 * (lane + 32 * t)) = ahead[t];
        __syncwarp();
        fetch(it + step, ahead);                               // on its way while these are picked apart
        if (skip(it, count)) continue;
        uint64_t r = items <= 0xFFFFFFFFull ? (uint32_t)it / groups : it / groups;
        uint32_t gi = (uint32_t)(it - r * groups);
#pragma unroll
        for (uint32_t i = 0; i < kAtOnce; ++i) {
            if (i >= count) break;
            // (every offset below is a multiple of four: one shift for the whole super-block)
            const uint32_t at = lead + 210u * i, sh = (at & 2u) * 8u;
            const uint32_t* p = reinterpret_cast<const uint32_t*>(mine + (at & ~3u));
            const uint32_t a0 = p[ql / 4], a1 = p[ql / 4 + 1], a2 = p[ql / 4 + 2], b0 = p[qh / 4], b1 = p[qh / 4 + 1], b2 = p[qh / 4 + 2];
            const uint32_t v0 = ((__funnelshift_r(a0, a1, sh) >> nib) & 0x0F0F0F0Fu) | (((__funnelshift_r(b0, b1, sh) >> (2 * g)) & 0x03030303u) << 4);
            const uint32_t v1 = ((__funnelshift_r(a1, a2, sh) >> nib) & 0x0F0F0F0Fu) | (((__funnelshift_r(b1, b2, sh) >> (2 * g)) & 0x03030303u) << 4);
            uint8_t* dst = out + (it + i) * 272u;
            reinterpret_cast<uint2*>(dst)[lane] = make_uint2(v0, v1);
            if (lane < 5) {                                    // four words of scales, d
                const uint32_t u = __funnelshift_r(p[48 + lane], p[49 + lane], sh);
                if (lane < 4) reinterpret_cast<uint32_t*>(dst + 256)[lane] = u;
                else d_out[(uint64_t)gi * n + r] = f16_bits_to_f32(u & 0xFFFFu) * 0x1p12f;
            }
            if (++gi == groups) { gi = 0; ++r; }
        }
    }
}

int launch_widen_q6(cudaStream_t stream, const uint8_t* w, uint32_t k, uint64_t n, uint8_t* out, const uint32_t* used, uint32_t slab_rows) {
    if (n == 0 || k == 0) return RLXQ_OK;
    if (((uintptr_t)w & 1u) || ((uintptr_t)out & 15u) || k % 256) return fail(RLXQ_E_ALIGN, "widen_q6: bad alignment");
    const uint32_t groups = k / 256;
    uint64_t blocks = (groups * n + 31) / 32;
    const uint64_t cap = (uint64_t)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    int rc = launch_pdl(widen_q6_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, w, groups, n, out,
                        reinterpret_cast<float*>(out + (uint64_t)groups * 272u * n), used, slab_rows);
    if (rc) return rc;
    count_launch();
    return check_launch("widen_q6_kernel");
}

}  // namespace rlxq
