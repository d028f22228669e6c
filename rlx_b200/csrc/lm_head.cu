// Greedy / top-k selection over a GGUF-packed tied LM head.
//
// Replaces gguf_tied_lm_argmax (rlx-cpu/src/lm_head.rs:223-251) and gguf_tied_lm_topk (:172-199).
// logits = hidden . W^T is one batch-1 call of the streaming GEMV (the vocabulary is the output
// dimension: 128 k rows x 4096 columns of Q4_K is 295 MB, i.e. pure HBM streaming).  Selection:
//   lm_peaks_kernel  a warp per slice of 256 logits writes its largest (value, then the smaller token id)
//   lm_rank_kernel   C CTAs.  The C best logits lie in the C slices with the largest peaks, and none is below the smallest of
//                    these, so each CTA finds that peak (a search over the keys' bits), collects what reaches it from the
//                    C slices, takes the candidate of its own rank and (RLXQ_LM_EXACT) recomputes that logit exactly as the
//                    reference does: f32 products in column order, multiply and add rounded separately (row_dot_gguf,
//                    lm_head.rs:46-76), decoders bit-exact; the CTA that finishes last ranks the C candidates by the
//                    (exact) values and writes the first `cap`
// Bound: latency, most of it the serial chain of k additions, 4 cycles each at best.  Selecting one candidate after the other
// (C rounds per slice, C more to merge, in two kernels), a chain that waited for each load and a kernel for the final
// ranking took 40 us behind the GEMV at 128256 x 4096 Q4_K and cap 1 and 72 us at cap 40; now 24 and 30 us.
// C = cap + 8 spare candidates, so the exact re-ranking can repair any reordering the GEMV's
// rounding (15-bit activations, different summation order) causes among near-equal logits.
#include <math_constants.h>

#include "common.cuh"
#include "decode.cuh"
#include "kernels.h"
#include "rlxq_lm.h"
#include "staged_common.cuh"

namespace rlxq {

constexpr uint32_t kLmMaxSlices = 2048;   // slices: of 256 logits, or the multiple of 256 that gives no more than this
constexpr uint32_t kLmMaxVocab = 4u << 20;
constexpr uint32_t kLmThreads = 256;
constexpr uint32_t kLmSpare = 8;          // candidates beyond cap
constexpr uint32_t kLmNone = 0xFFFFFFFFu; // "no token"
constexpr uint32_t kLmChunk = 4096;       // products staged per pass of the exact sum
constexpr uint32_t kLmCollect = 1024;     // entries ranked by counting

// Order-preserving map of f32 onto u32 (larger float <-> larger integer); NaN maps to 0, below -inf.
__device__ __forceinline__ uint32_t ord_of(float v) {
    if (!(v == v)) return 0u;
    const uint32_t u = __float_as_uint(v);
    return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float ord_to_float(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}
// Larger is better (value, then the smaller token id); 0 = cannot be chosen.
__device__ __forceinline__ uint64_t lm_key(float v, uint32_t id) {
    const uint32_t ord = ord_of(v);
    return ord ? (uint64_t)ord << 32 | (uint32_t)~id : 0ull;
}

__global__ void __launch_bounds__(kLmThreads) lm_peaks_kernel(const float* logits, uint32_t n, uint32_t slice,
                                                              uint32_t nslices, uint64_t* __restrict__ peaks,
                                                              uint32_t* __restrict__ done) {
    const uint32_t s = (blockIdx.x * kLmThreads + threadIdx.x) / 32, lane = threadIdx.x & 31u;
    griddep_wait();                   // the logits come from the kernel in front
    // (the ranking kernel is not let in early: its CTAs waiting beside the GEMV cost 9 us at 57651 x 3072 Q8_0)
    if (blockIdx.x == 0 && threadIdx.x == 0) *done = 0u;
    if (s >= nslices) return;
    uint64_t best = 0ull;
    for (uint32_t base = 0; base < slice; base += 256) {
        float v[8];                   // all loads first: NaN cannot be chosen
        const uint32_t j = s * slice + base + lane;
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) v[r] = j + 32 * r < n ? logits[j + 32 * r] : CUDART_NAN_F;
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) {
            const uint64_t key = lm_key(v[r], j + 32 * r);
            best = key > best ? key : best;
        }
    }
    const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best >> 32));
    const uint32_t lo = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best >> 32) == hi ? (uint32_t)best : 0u);
    if (lane == 0) peaks[s] = (uint64_t)hi << 32 | lo;
}


// a before b: larger value, then smaller token id.  NaN is never before anything.
__device__ __forceinline__ bool before(float av, uint32_t ai, float bv, uint32_t bi) {
    return av > bv || (av == bv && ai < bi);
}

// The largest T that at least C keys reach (keys are unique: the search ends where C reach it); 1 when fewer than C keys can
// be chosen at all.  count(T, lane): a lane's part of the keys >= T.  Three bits a step: warp w counts for the trial w + 1.
template <typename F> __device__ __forceinline__ uint64_t lm_threshold(uint32_t C, F&& count, uint32_t (*sh)[8]) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t T = 0ull;
    uint32_t parity = 0;
#pragma unroll 1
    for (int shift = 61; shift >= -2; shift -= 3) {
        const int at = shift < 0 ? 0 : shift;
        const uint32_t trials = shift < 0 ? 1u : 7u;
        if (warp < trials) {
            const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, count(T | (uint64_t)(warp + 1) << at, lane));
            if (lane == 0) sh[parity][warp] = c;
        }
        __syncthreads();
        uint32_t best = 0;
        bool found = false;
#pragma unroll
        for (uint32_t w = 0; w < 7; ++w) {
            if (w < trials && sh[parity][w] >= C) { best = w + 1; found = sh[parity][w] == C; }
        }
        T |= (uint64_t)best << at;
        parity ^= 1u;                     // one barrier a step: the next step writes the other half
        if (found) break;
    }
    return T ? T : 1ull;
}

__device__ __forceinline__ void lm_load32(float4 (&v)[8], uint32_t a) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i].z), "=f"(v[i].w) : "r"(a + 16 * i) : "memory");
}
__device__ __forceinline__ void lm_add32(float& acc, const float4 (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        acc = __fadd_rn(acc, v[i].x);
        acc = __fadd_rn(acc, v[i].y);
        acc = __fadd_rn(acc, v[i].z);
        acc = __fadd_rn(acc, v[i].w);
    }
}

template <uint32_t SCHEME>
__device__ __forceinline__ float lm_exact_logit(const void* __restrict__ hidden, uint32_t h_bf16, const uint8_t* __restrict__ w,
                                                uint32_t k, uint32_t row, float* prod) {
    constexpr uint32_t E = SchemeTraits<SCHEME>::kElems, B = SchemeTraits<SCHEME>::kBytes;
    const uint8_t* wrow = w + (uint64_t)row * (k / E) * B;
    float acc = 0.0f;
    for (uint32_t base = 0; base < k; base += kLmChunk) {
        const uint32_t chunk = min(kLmChunk, k - base);                // a multiple of 32
#pragma unroll 4
        for (uint32_t q = threadIdx.x; q < chunk / 4; q += kLmThreads) {   // independent iterations: loads overlap
            const uint32_t e = base + 4 * q;
            const float4 wv = decode4_exact<SCHEME>(wrow + (uint64_t)(e / E) * B, e % E);
            float h[4];
            if (h_bf16) {
                const uint2 hb = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(hidden) + e);
                h[0] = __uint_as_float(hb.x << 16); h[1] = __uint_as_float(hb.x & 0xFFFF0000u);
                h[2] = __uint_as_float(hb.y << 16); h[3] = __uint_as_float(hb.y & 0xFFFF0000u);
            } else {
                const float4 hv = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(hidden) + e);
                h[0] = hv.x; h[1] = hv.y; h[2] = hv.z; h[3] = hv.w;
            }
            prod[4 * q + 0] = __fmul_rn(h[0], wv.x);
            prod[4 * q + 1] = __fmul_rn(h[1], wv.y);
            prod[4 * q + 2] = __fmul_rn(h[2], wv.z);
            prod[4 * q + 3] = __fmul_rn(h[3], wv.w);
        }
        // zeros up to the next 64: a sum that starts at +0 is never -0, so adding +0 leaves every bit of it
        if (threadIdx.x < 64 && chunk + threadIdx.x < (chunk + 63) / 64 * 64) prod[chunk + threadIdx.x] = 0.0f;
        __syncthreads();
        if (threadIdx.x == 0) {
            // The reference's order: one running f32 sum over the columns, a serial chain of adds.  The next 32 products are
            // on their way from shared memory while 32 are added; two buffers by name, because a rotated one was loaded
            // right before its use (14 cycles an add instead of 4).
            const uint32_t pa = smem_u32(prod);
            float4 a[8], b[8];
            lm_load32(a, pa);
            for (uint32_t p = 0; p < chunk; p += 64) {
                lm_load32(b, pa + 4 * (p + 32));
                lm_add32(acc, a);
                lm_load32(a, pa + 4 * (p + 64));                       // (past the end: not used)
                lm_add32(acc, b);
            }
        }
        __syncthreads();
    }
    return acc;                                                        // thread 0's
}

struct LmRank {
    const float* logits;
    const uint64_t* peaks;
    uint32_t n, slice, nslices, C, cap, exact, argmax_mode, h_bf16, k;
    const void* hidden;
    const uint8_t* w;
    uint32_t *si, *done, *out_i;
    float *ev, *out_v;
};

template <uint32_t SCHEME>
__global__ void __launch_bounds__(kLmThreads) lm_rank_kernel(const __grid_constant__ LmRank P) {
    // one region for the peaks, then the collected entries, then the products: a block that fits beside others starts sooner
    __shared__ __align__(16) float prod[kLmChunk + 64];
    static_assert(sizeof(prod) >= 8 * kLmMaxSlices && kLmMaxSlices >= kLmCollect, "shared region");
    uint64_t *peaks = reinterpret_cast<uint64_t*>(prod), *cand = peaks;
    __shared__ uint64_t mine;
    __shared__ uint32_t sel[RLXQ_LM_MAX_CAP], sums[2][8], nsel, ncand, last;
    __shared__ float fv[RLXQ_LM_MAX_CAP];
    __shared__ uint32_t fi[RLXQ_LM_MAX_CAP];
    const uint32_t t = threadIdx.x;
    griddep_launch_dependents();
    griddep_wait();
    for (uint32_t q = t; q < P.nslices; q += kLmThreads) peaks[q] = P.peaks[q];
    if (t == 0) { nsel = 0; ncand = 0; mine = 0ull; }
    __syncthreads();
    uint64_t T = lm_threshold(P.C, [&](uint64_t at, uint32_t lane) {
        uint32_t c = 0;
#pragma unroll 8
        for (uint32_t q = lane; q < P.nslices; q += 32) c += peaks[q] >= at;
        return c;
    }, sums);
    for (uint32_t q = t; q < P.nslices; q += kLmThreads)
        if (peaks[q] >= T) sel[atomicAdd(&nsel, 1u)] = q;      // C of them at most
    __syncthreads();
    auto collect = [&] {
        for (uint32_t off = t; off < P.slice; off += kLmThreads)
            for (uint32_t q = 0; q < nsel; q += 8) {
                uint32_t id[8];
                float v[8];               // eight loads in flight; NaN cannot be chosen
#pragma unroll
                for (uint32_t r = 0; r < 8; ++r) id[r] = q + r < nsel ? sel[q + r] * P.slice + off : P.n;
#pragma unroll
                for (uint32_t r = 0; r < 8; ++r) v[r] = id[r] < P.n ? __ldcg(P.logits + id[r]) : CUDART_NAN_F;
#pragma unroll
                for (uint32_t r = 0; r < 8; ++r) {
                    const uint64_t key = lm_key(v[r], id[r]);
                    if (key >= T) {
                        const uint32_t at = atomicAdd(&ncand, 1u);
                        if (at < kLmCollect) cand[at] = key;
                    }
                }
            }
        __syncthreads();
    };
    collect();
    if (ncand > kLmCollect) {             // hosts of equal logits: the exact threshold among the slices' entries
        T = lm_threshold(P.C, [&](uint64_t at, uint32_t lane) {
            uint32_t c = 0;
            for (uint32_t q = 0; q < nsel; ++q)
                for (uint32_t off = lane; off < P.slice; off += 32) {
                    const uint32_t id = sel[q] * P.slice + off;
                    if (id < P.n) c += lm_key(__ldcg(P.logits + id), id) >= at;
                }
            return c;
        }, sums);
        if (t == 0) ncand = 0;
        __syncthreads();
        collect();
    }
    const uint32_t count = ncand;
    for (uint32_t q = t; q < count; q += kLmThreads) {
        const uint64_t key = cand[q];
        uint32_t rank = 0;
#pragma unroll 8
        for (uint32_t i = 0; i < count; ++i) rank += cand[i] > key;
        if (rank == blockIdx.x) mine = key;
    }
    __syncthreads();
    const uint32_t row = mine ? ~(uint32_t)mine : kLmNone;
    float v = row != kLmNone ? ord_to_float((uint32_t)(mine >> 32)) : -CUDART_INF_F;
    if (P.exact && row != kLmNone) v = lm_exact_logit<SCHEME>(P.hidden, P.h_bf16, P.w, P.k, row, prod);
    if (t == 0) {
        P.ev[blockIdx.x] = v;
        P.si[blockIdx.x] = row;
        __threadfence();
        last = atomicAdd(P.done, 1u) == P.C - 1 ? 1u : 0u;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    if (t < P.C) { fv[t] = __ldcg(P.ev + t); fi[t] = __ldcg(P.si + t); }
    if (t < P.cap) { P.out_i[t] = kLmNone; P.out_v[t] = -CUDART_INF_F; }
    __syncthreads();
    if (t < P.C) {
        const float mv = fv[t];
        const uint32_t mi = fi[t];
        if (mi != kLmNone && mv == mv) {
            uint32_t rank = 0;
#pragma unroll 8
            for (uint32_t j = 0; j < P.C; ++j)
                if (fi[j] != kLmNone && fv[j] == fv[j] && before(fv[j], fi[j], mv, mi)) ++rank;
            if (rank < P.cap) { P.out_i[rank] = mi; P.out_v[rank] = mv; }
        }
    }
    __syncthreads();
    // the reference's greedy scan starts from (0, -inf) and only moves on a strictly larger logit
    if (P.argmax_mode && t == 0 && !(P.out_v[0] > -CUDART_INF_F)) { P.out_i[0] = 0u; P.out_v[0] = -CUDART_INF_F; }
}

struct LmPlan {
    uint32_t slice, nslices, C;
    size_t off_peaks, off_done, off_si, off_ev, off_mm, mm_bytes, total;
};

static LmPlan plan_lm(uint32_t scheme, uint32_t n_embd, uint32_t n_vocab, uint32_t x_dtype, uint32_t cap) {
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    LmPlan p{};
    p.slice = (n_vocab + 256 * kLmMaxSlices - 1) / (256 * kLmMaxSlices) * 256;
    p.nslices = (n_vocab + p.slice - 1) / p.slice;
    p.C = cap + kLmSpare;
    if (p.C > RLXQ_LM_MAX_CAP) p.C = RLXQ_LM_MAX_CAP;
    size_t off = up((size_t)n_vocab * 4);                       // logits first
    p.off_peaks = off; off += up((size_t)p.nslices * 8);
    p.off_done = off; off += 256;
    p.off_si = off; off += up((size_t)p.C * 4);
    p.off_ev = off; off += up((size_t)p.C * 4);
    p.off_mm = off;
    p.mm_bytes = matmul_workspace_bytes(scheme, 1, n_embd, n_vocab, x_dtype, RLXQ_F32);
    p.total = off + up(p.mm_bytes);
    return p;
}

template <uint32_t SCHEME>
static int launch_rank(cudaStream_t s, const LmRank& P) {
    return launch_pdl(lm_rank_kernel<SCHEME>, dim3(P.C), dim3(kLmThreads), 0, s, P);
}

static int lm_run(cudaStream_t stream, uint32_t scheme, const void* hidden, uint32_t x_dtype, const void* w_blocks,
                  uint32_t n_embd, uint32_t n_vocab, uint32_t cap, uint32_t flags, bool argmax_mode, void* workspace,
                  size_t workspace_bytes, uint32_t* idx_out, float* val_out) {
    Geometry g;
    if (!geometry(scheme, &g)) return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    if (x_dtype != RLXQ_F32 && x_dtype != RLXQ_BF16) return fail(RLXQ_E_DTYPE, "unknown dtype");
    if (n_embd == 0 || n_embd % g.elems) return fail(RLXQ_E_SHAPE, "n_embd=%u is not a positive multiple of the block size %u", n_embd, g.elems);
    if (n_vocab == 0) return fail(RLXQ_E_SHAPE, "n_vocab is zero");
    if (n_vocab > kLmMaxVocab) return fail(RLXQ_E_LIMIT, "n_vocab=%u beyond %u", n_vocab, kLmMaxVocab);
    if (cap == 0 || cap > RLXQ_LM_MAX_CAP || cap > n_vocab)
        return fail(RLXQ_E_ARG, "cap=%u must be in [1, min(%u, n_vocab)]", cap, RLXQ_LM_MAX_CAP);
    if (flags & ~(uint32_t)RLXQ_LM_EXACT) return fail(RLXQ_E_ARG, "unknown flags 0x%x", flags);
    if (!hidden || !w_blocks || !idx_out || !val_out || !workspace) return fail(RLXQ_E_NULL, "null buffer");
    if (((uintptr_t)hidden & 15u) || ((uintptr_t)workspace & 15u)) return fail(RLXQ_E_ALIGN, "hidden and workspace must be 16-byte aligned");
    if ((uintptr_t)w_blocks & 1u) return fail(RLXQ_E_ALIGN, "w_blocks must be 2-byte aligned");
    const LmPlan p = plan_lm(scheme, n_embd, n_vocab, x_dtype, cap);
    if (workspace_bytes < p.total)
        return fail(RLXQ_E_WORKSPACE, "LM head needs %zu workspace bytes, got %zu", p.total, workspace_bytes);
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    float* logits = reinterpret_cast<float*>(ws);
    const bool hbf = x_dtype == RLXQ_BF16;
    const bool exact = (flags & RLXQ_LM_EXACT) != 0;
    const uint32_t C = exact ? p.C : cap;

    int rc = dispatch_matmul(stream, scheme, hidden, hbf, (const uint8_t*)w_blocks, logits, false, 1, n_embd, n_vocab,
                             p.mm_bytes ? ws + p.off_mm : nullptr, p.mm_bytes);
    if (rc) return rc;
    // programmatic dependent launch: each kernel is resident before its predecessor ends and orders itself with
    // griddepcontrol.wait, so a small launch costs a microsecond, not three
    uint64_t* peaks = reinterpret_cast<uint64_t*>(ws + p.off_peaks);
    uint32_t* done = reinterpret_cast<uint32_t*>(ws + p.off_done);
    rc = launch_pdl(lm_peaks_kernel, dim3((p.nslices + kLmThreads / 32 - 1) / (kLmThreads / 32)), dim3(kLmThreads), 0, stream,
                    (const float*)logits, n_vocab, p.slice, p.nslices, peaks, done);
    if (rc) return rc;
    count_launch();
    LmRank P{};
    P.logits = logits; P.peaks = peaks; P.n = n_vocab; P.slice = p.slice; P.nslices = p.nslices; P.C = C; P.cap = cap; P.exact = exact ? 1u : 0u; P.argmax_mode = argmax_mode ? 1u : 0u;
    P.h_bf16 = hbf ? 1u : 0u; P.k = n_embd; P.hidden = hidden; P.w = (const uint8_t*)w_blocks;
    P.si = reinterpret_cast<uint32_t*>(ws + p.off_si); P.done = done; P.out_i = idx_out;
    P.ev = reinterpret_cast<float*>(ws + p.off_ev); P.out_v = val_out;
    switch (scheme) {
        case RLXQ_Q4_K: rc = launch_rank<RLXQ_Q4_K>(stream, P); break;
        case RLXQ_Q5_K: rc = launch_rank<RLXQ_Q5_K>(stream, P); break;
        case RLXQ_Q6_K: rc = launch_rank<RLXQ_Q6_K>(stream, P); break;
        case RLXQ_Q8_K: rc = launch_rank<RLXQ_Q8_K>(stream, P); break;
        case RLXQ_Q2_K: rc = launch_rank<RLXQ_Q2_K>(stream, P); break;
        case RLXQ_Q3_K: rc = launch_rank<RLXQ_Q3_K>(stream, P); break;
        case RLXQ_Q4_1: rc = launch_rank<RLXQ_Q4_1>(stream, P); break;
        case RLXQ_Q5_0: rc = launch_rank<RLXQ_Q5_0>(stream, P); break;
        case RLXQ_Q5_1: rc = launch_rank<RLXQ_Q5_1>(stream, P); break;
        case RLXQ_Q4_0: rc = launch_rank<RLXQ_Q4_0>(stream, P); break;
        case RLXQ_Q8_0: rc = launch_rank<RLXQ_Q8_0>(stream, P); break;
        default: return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    }
    if (rc) return rc;
    count_launch();
    return check_launch("lm_head kernels");
}

}  // namespace rlxq

using namespace rlxq;

extern "C" int rlxq_lm_head_workspace_bytes(uint32_t scheme, uint32_t n_embd, uint32_t n_vocab, uint32_t x_dtype,
                                            uint32_t cap, size_t* bytes) {
    if (!bytes) return fail(RLXQ_E_NULL, "bytes is null");
    Geometry g;
    if (!geometry(scheme, &g)) return fail(RLXQ_E_SCHEME, "unknown scheme %u", scheme);
    if (x_dtype != RLXQ_F32 && x_dtype != RLXQ_BF16) return fail(RLXQ_E_DTYPE, "unknown dtype");
    if (n_embd == 0 || n_embd % g.elems || n_vocab == 0) return fail(RLXQ_E_SHAPE, "bad LM head shape %u x %u", n_vocab, n_embd);
    if (cap == 0 || cap > RLXQ_LM_MAX_CAP) return fail(RLXQ_E_ARG, "cap=%u must be in [1, %u]", cap, RLXQ_LM_MAX_CAP);
    *bytes = plan_lm(scheme, n_embd, n_vocab, x_dtype, cap).total;
    return RLXQ_OK;
}

extern "C" int rlxq_lm_head_topk(rlxq_stream_t stream, uint32_t scheme, const void* hidden, uint32_t x_dtype,
                                 const void* w_blocks, uint32_t n_embd, uint32_t n_vocab, uint32_t cap, uint32_t flags,
                                 void* workspace, size_t workspace_bytes, uint32_t* idx_out, float* val_out) {
    return lm_run((cudaStream_t)stream, scheme, hidden, x_dtype, w_blocks, n_embd, n_vocab, cap, flags, false, workspace,
                  workspace_bytes, idx_out, val_out);
}

extern "C" int rlxq_lm_head_argmax(rlxq_stream_t stream, uint32_t scheme, const void* hidden, uint32_t x_dtype,
                                   const void* w_blocks, uint32_t n_embd, uint32_t n_vocab, uint32_t flags,
                                   void* workspace, size_t workspace_bytes, uint32_t* idx_out, float* val_out) {
    return lm_run((cudaStream_t)stream, scheme, hidden, x_dtype, w_blocks, n_embd, n_vocab, 1, flags, true, workspace,
                  workspace_bytes, idx_out, val_out);
}
