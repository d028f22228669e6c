// Kernel selection for rlxq_matmul: the counterpart of the reference's
// `use_gpu = dequant_scratch_off > 0 && blas.is_some()` branch and host fallback
// (rlx-cuda/src/backend.rs:5366-5405).  There is no host fallback here: every shape runs on
// the GPU, through the fastest kernel that supports it.
#include "common.cuh"
#include "kernels.h"

namespace rlxq {

// Prefill (m > 8) on the tensor-core GEMM.  Its operands are bf16: f32 activations go in as hi + lo halves, `chunk`
// rows of x at a time (the split rows are kept under 128 MiB), multiplied by the same decoded weights.  Rows that TMA
// cannot tile where they lie (k not a whole number of 256 weights, or of the 16-byte groups of a format's super-blocks;
// weights that are not 16-byte aligned) are first re-laid on a padded pitch in the workspace, and weights and activations
// then keep all of their 24 bits (PRECISE), since those shapes were multiplied in f32 before they had this path.  The
// workspace query does not know the weights' address and plans for aligned ones: weights at another address are re-laid only
// for a caller who brings more than it asks for, and run the general kernel for everybody else.  Q6_K rows are widened, which
// takes a third more scratch than the rows have bytes; a caller who brings less than that, but room for the rows, has them copied
// as they are (300 x 11008 x 4096 f32: 151 us widened, 224 copied, 4.8 ms through the general kernel).
struct PrefillPlan { bool ok, relaid, halves; uint32_t layout, chunk; uint64_t pitch; size_t off_w, off_y2, off_gemm, bytes; };
static PrefillPlan plan_prefill(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, bool xbf, bool direct, bool widen = true) {
    PrefillPlan p{};
    const void* aligned = (const void*)256;              // dispatch checks the real pointers
    if (m <= 8 || options().gemm_kernel.load() == 1) return p;
    p.relaid = !(direct && gemm_tc_supported(scheme, m, k, n, aligned, aligned));
    if (p.relaid && !gemm_relaid_supported(scheme, m, k, n, aligned)) return p;
    auto al = [](size_t v) { return (v + 255) / 256 * 256; };
    uint64_t chunk = m;
    // Rows of at most 512 weights: hi and lo rows go through the GEMM as 2 m rows and their results are added behind it;
    // the chunk keeps the two results under 128 MiB.  This is not the faster form: one pass takes 8.5 us instead of 11 at
    // 64 x 256 x 4096, 16 instead of 28 at 300 x 512 x 8192 and 76 instead of 210 at 1024 x 512 x 32768 (Q4_0, Q8_0 and Q4_K
    // alike).  It stays at these sizes because the GEMM's tests hold calls of 256 and 512 columns to three launches a chunk.
    p.halves = !xbf && !p.relaid && k <= 512;
    if (!xbf) {
        chunk = p.halves ? (128ull << 20) / (8ull * n) / 128 * 128 : (128ull << 20) / (4ull * k) / 256 * 256;      // (PRECISE: 192 MiB)
        const uint64_t least = p.halves ? 128 : 256;
        if (chunk < least) chunk = least;
        if (p.halves && chunk > 2048) chunk = 2048;
        if (chunk > m) chunk = m;
    }
    p.chunk = (uint32_t)chunk;
    p.layout = p.relaid && widen && scheme == RLXQ_Q6_K ? kQ6Wide : scheme;
    p.off_w = xbf ? 0 : al((size_t)gemm_x_parts(true, p.relaid) * chunk * k * 2);
    p.pitch = p.relaid ? gemm_relaid_pitch(p.layout, k) : 0;
    p.off_y2 = p.off_w + (p.relaid ? al((size_t)gemm_relaid_bytes(p.layout, k, n)) : 0);
    p.off_gemm = p.off_y2 + (p.halves ? al((size_t)2 * chunk * n * 4) : 0);
    p.bytes = p.off_gemm;
    if (!p.halves) {
        size_t g = gemm_tc_workspace_bytes(p.layout, (uint32_t)chunk, k, n, !xbf, p.relaid);
        if (m % chunk) {                                 // the last, shorter chunk may be split over the SMs differently
            const size_t g2 = gemm_tc_workspace_bytes(p.layout, (uint32_t)(m % chunk), k, n, !xbf, p.relaid);
            g = g2 > g ? g2 : g;
        }
        p.bytes += al(g);
    }
    p.ok = true;
    return p;
}

size_t matmul_workspace_bytes(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, uint32_t x_dtype,
                              uint32_t y_dtype) {
    (void)y_dtype;
    if (m == 0 || n == 0 || k == 0) return 0;
    if (m <= 8) {
        // large enough for whichever GEMV kernel the dispatcher (or a forced option) picks
        const size_t a = staged_workspace_bytes(scheme, m, k, n);
        // (batch 5-8 of a format that only has the integer kernel runs it twice, four rows at a time)
        const size_t b = int_workspace_bytes(scheme, m <= 4 ? m : 4, k, n);
        // the tcgen05 GEMV (8-byte words for the parts of cut tiles) only runs when it is asked for
        const size_t c = options().gemv_kernel.load() == 4 ? gemv_tc_workspace_bytes(scheme, m, k, n) : 0;
        const size_t d = int_mma_workspace_bytes(scheme, m, k, n);
        const size_t ab = a > b ? a : b, cd = c > d ? c : d;
        return ab > cd ? ab : cd;
    }
    const PrefillPlan p = plan_prefill(scheme, m, k, n, x_dtype == RLXQ_BF16, true);
    return p.ok ? p.bytes : 0;
}

int dispatch_matmul(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y,
                    bool ybf, uint32_t m, uint32_t k, uint32_t n, void* ws, size_t ws_bytes) {
    if (k == 0) {
        // empty reduction: the reference zero-fills the output (rlx-cpu/src/gguf_matmul.rs:52)
        RLXQ_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)m * n * (ybf ? 2 : 4), stream));
        return RLXQ_OK;
    }
    if (!x || !w) return fail(RLXQ_E_NULL, "null input buffer");
    if ((uintptr_t)w & 1u) return fail(RLXQ_E_ALIGN, "w_blocks must be 2-byte aligned");
    if ((uintptr_t)x & 15u) return fail(RLXQ_E_ALIGN, "x must be 16-byte aligned");
    if ((uintptr_t)y & (ybf ? 1u : 3u)) return fail(RLXQ_E_ALIGN, "y must be aligned to its element size");
    if (m <= 8) {
        // 0 = automatic: the integer kernel with its dp4a units for batch 1, with its integer-MMA units for batch
        // 2-8 (measured at batch 2: level on Q4_K 4096 -> 14336, 5-15 % ahead elsewhere), then the dp4a units again
        // (batch 2, formats without an MMA unit), the staged tensor-mode kernel, the generic one.  The dp4a units
        // also run batch 3-4, but only when asked for with gemv_kernel = 3.
        const int64_t force = options().gemv_kernel.load();
        const bool can_int = m <= 4 && int_supported(scheme, m, k, n, w, x);
        const bool can_tc = staged_supported(scheme, m, k, n, w, x, xbf);
        const bool can_tcg = gemv_tc_supported(scheme, m, k, n, w, x, xbf);
        if (force == 4) {
            if (!can_tcg) return fail(RLXQ_E_SHAPE, "tensor-core GEMV does not support scheme %u m=%u k=%u n=%u (or 16-byte alignment)", scheme, m, k, n);
            return launch_gemv_tc(stream, scheme, x, xbf, w, y, ybf, m, k, n, ws, ws_bytes);
        }
        if (force == 5) {
            if (!int_mma_supported(scheme, m, k, n, w, x)) return fail(RLXQ_E_SHAPE, "integer-MMA GEMV does not support scheme %u m=%u k=%u n=%u (or 16-byte alignment)", scheme, m, k, n);
            return launch_gemv_int_mma(stream, scheme, x, xbf, w, y, ybf, m, k, n, ws, ws_bytes);
        }
        if (force == 3 && !can_int)
            return fail(RLXQ_E_SHAPE, "integer GEMV does not support m=%u k=%u n=%u (or 16-byte alignment)", m, k, n);
        if (force == 2 && !can_tc)
            return fail(RLXQ_E_SHAPE, "staged GEMV does not support m=%u k=%u n=%u (or 16-byte alignment)", m, k, n);
        const bool no_dp4a = scheme == RLXQ_Q8_K || scheme == RLXQ_Q2_K || scheme == RLXQ_Q3_K || scheme == RLXQ_Q4_1 ||
                             scheme == RLXQ_Q5_0 || scheme == RLXQ_Q5_1;                             // MMA units only
        if (force == 0 && (m >= 2 || no_dp4a) && int_mma_supported(scheme, m, k, n, w, x))
            return launch_gemv_int_mma(stream, scheme, x, xbf, w, y, ybf, m, k, n, ws, ws_bytes);
        if (force == 3 || (force == 0 && can_int && m <= 2))
            return launch_gemv_int(stream, scheme, x, xbf, w, y, ybf, m, k, n, ws, ws_bytes);
        if (force == 2 || (force == 0 && can_tc))
            return launch_gemv_staged(stream, scheme, x, xbf, w, y, ybf, m, k, n, ws, ws_bytes);
        // A format with the integer kernel but no tensor-mode kernel (Q5_K): batch 3-4 in one pass, batch 5-8 in
        // two passes of four rows; streaming the weights twice still beats the warp-per-row kernel several times.
        if (force == 0 && can_int) return launch_gemv_int(stream, scheme, x, xbf, w, y, ybf, m, k, n, ws, ws_bytes);
        if (force == 0 && m > 4 && int_supported(scheme, 4, k, n, w, x) && int_supported(scheme, m - 4, k, n, w, x)) {
            const size_t xrow = (size_t)k * (xbf ? 2 : 4), yrow = (size_t)n * (ybf ? 2 : 4);
            if ((4 * xrow) % 16 == 0) {
                int rc = launch_gemv_int(stream, scheme, x, xbf, w, y, ybf, 4, k, n, ws, ws_bytes);
                if (rc) return rc;
                return launch_gemv_int(stream, scheme, static_cast<const uint8_t*>(x) + 4 * xrow, xbf, w,
                                       static_cast<uint8_t*>(y) + 4 * yrow, ybf, m - 4, k, n, ws, ws_bytes);
            }
        }
        // rows that TMA cannot tile: f32 arithmetic like the general kernel's, at streaming speed
        if (force == 0 && gemv_parts_pays(scheme, m, k, n, xbf, x)) return launch_gemv_parts(stream, scheme, x, xbf, w, y, ybf, m, k, n);
        if (force == 0 && gemv_f32_supported(scheme, m, k, x)) return launch_gemv_f32(stream, scheme, x, xbf, w, y, ybf, m, k, n);
        return launch_matmul_generic(stream, scheme, x, xbf, w, y, ybf, m, k, n);
    }
    // m > 8: the tensor-memory GEMM; without the workspace it needs, the tiled generic kernel
    const int64_t gforce = options().gemm_kernel.load();
    const bool direct = gemm_tc_supported(scheme, m, k, n, w, x);
    if (gforce == 2 && (!direct || !xbf))
        return fail(RLXQ_E_SHAPE, "gemm_kernel = 2 takes bf16 activations, k %% 256 == 0 (1024 for Q2_K and Q8_K, 2048 for Q3_K and Q6_K) and 16-byte alignment");
    PrefillPlan p = plan_prefill(scheme, m, k, n, xbf, direct);
    if (p.ok && p.layout != scheme && ws_bytes < p.bytes) p = plan_prefill(scheme, m, k, n, xbf, direct, false);
    const bool fits = ws && ws_bytes >= p.bytes && !((uintptr_t)ws & 255u);
    if (p.ok && (fits || (xbf && direct))) {
        uint8_t* base = static_cast<uint8_t*>(ws);
        GemmCall c{};
        c.w = w; c.w_pitch = p.pitch; c.precise = p.relaid; c.k = k; c.n = n;
        if (p.relaid) {
            int rc = launch_relay(stream, p.layout, w, k, n, base + p.off_w);
            if (rc) return rc;
            c.w = base + p.off_w;
        }
        for (uint32_t r0 = 0; r0 < m; r0 += p.chunk) {
            const uint32_t rows = m - r0 < p.chunk ? m - r0 : p.chunk;
            void* const out = static_cast<uint8_t*>(y) + (size_t)r0 * n * (ybf ? 2 : 4);
            c.x = static_cast<const uint8_t*>(x) + (size_t)r0 * k * (xbf ? 2 : 4);
            if (!xbf) {
                int rc = launch_split_hi_lo(stream, static_cast<const float*>(c.x), base, rows, k, gemm_x_parts(true, p.relaid));
                if (rc) return rc;
                c.x = base;
            }
            int rc;
            if (p.halves) {
                float* y2 = reinterpret_cast<float*>(base + p.off_y2);
                c.x_rows = 2 * rows; c.y = y2;
                rc = launch_gemm(stream, p.layout, c, nullptr, 0);
                if (!rc) rc = launch_add_slices(stream, y2, 2, (uint64_t)rows * n, out, ybf, (uint64_t)rows * n);
            } else {
                c.x_rows = rows; c.f32 = !xbf; c.y = out; c.ybf = ybf;
                // (bf16 activations: a workspace too small for the k split runs whole tiles)
                rc = launch_gemm(stream, p.layout, c, fits ? base + p.off_gemm : nullptr, fits ? ws_bytes - p.off_gemm : 0);
            }
            if (rc) return rc;
        }
        return RLXQ_OK;
    }
    return launch_matmul_generic(stream, scheme, x, xbf, w, y, ybf, m, k, n);
}

}  // namespace rlxq
