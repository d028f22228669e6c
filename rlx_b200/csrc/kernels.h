// Internal launch entry points shared between the translation units of the library.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace rlxq {

int launch_dequant_f32(cudaStream_t stream, uint32_t scheme, const uint8_t* w, uint64_t n_elems, float* out);

int launch_matmul_generic(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w,
                          void* y, bool ybf, uint32_t m, uint32_t k, uint32_t n);

// Staged tensor-mode GEMV (m <= 8).
bool staged_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* w, const void* x, bool xbf);
size_t staged_workspace_bytes(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n);
int launch_gemv_staged(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w,
                       void* y, bool ybf, uint32_t m, uint32_t k, uint32_t n, void* ws, size_t ws_bytes);
// Integer (dp4a) GEMV (m <= 2).
bool int_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* w, const void* x);
size_t int_workspace_bytes(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n);
int launch_gemv_int(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y,
                    bool ybf, uint32_t m, uint32_t k, uint32_t n, void* ws, size_t ws_bytes);

// tcgen05 / tensor-memory GEMV (m <= 8): weights decoded to fp16 in tensor memory, activations as bf16 high / low rows.
int launch_split_hi_lo(cudaStream_t stream, const float* x, void* out, uint64_t rows, uint64_t k, uint32_t parts);
uint32_t gemm_x_parts(bool f32, bool precise);
uint32_t gemm_most_rows(uint32_t scheme, bool f32, bool precise);
int launch_add_slices(cudaStream_t stream, const float* part, uint32_t slices, uint64_t stride, void* y, bool ybf, uint64_t total);
int launch_swiglu_pair(cudaStream_t stream, const float* gu, void* h, uint32_t m, uint32_t f);
// A chain of dependent batch-1/2 GEMVs in one cooperative launch (gemv_int.cu, gemv_chain_kernel).
struct ChainLayer { const uint8_t* w; uint32_t k, n, swiglu; };
size_t chain_workspace_bytes(uint32_t scheme, const ChainLayer* layers, uint32_t nlayers, uint32_t m);
int launch_gemv_chain(cudaStream_t stream, uint32_t scheme, const ChainLayer* layers, uint32_t nlayers, const void* x, bool xbf,
                      void* y, bool ybf, uint32_t m, void* ws, size_t ws_bytes);
bool int_mma_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* w, const void* x);
// whether the format's down projection also exists as a kernel that pushes its tiles into peers' exchange buffers
bool int_push_supported(uint32_t scheme);
size_t int_mma_workspace_bytes(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n);
int launch_gemv_int_mma(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y,
                        bool ybf, uint32_t m, uint32_t k, uint32_t n, void* ws, size_t ws_bytes);
bool gemv_tc_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* w, const void* x, bool xbf);
size_t gemv_tc_workspace_bytes(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n);
int launch_gemv_tc(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y, bool ybf,
                   uint32_t m, uint32_t k, uint32_t n, void* ws, size_t ws_bytes);

// tcgen05 / tensor-memory GEMM (m > 8).  What it reads its weights from (`layout`) is a format's own id, or Q6_K rows as
// widen_q6_kernel re-lays them: 256 bytes of quants in order, 16 scale bytes; the super-blocks' d apart.  These are PRECISE weights.
constexpr uint32_t kQ6Wide = 0x100u + RLXQ_Q6_K;
struct GemmCall {
    const void* x;             // bf16 [x_rows, k]; with f32 set, bf16(x) followed by bf16(x - bf16(x)), x_rows rows each
    uint32_t x_rows;
    bool f32;
    const uint8_t* w;
    uint64_t w_pitch;          // bytes between weight rows that a kernel in front has re-laid (0: packed, and constant)
    bool precise;              // f32 weights and activations, in bf16 parts, instead of weights rounded to bf16
    void* y;
    bool ybf;
    uint32_t k, n;
    // expert stacks: num_slabs [n, k] slabs, groups = the device-side tile table (GemmParams::groups) of tiles of tile_rows
    // rows, at most group_tiles of them, and the row of y every gathered row of x belongs to
    uint32_t num_slabs = 1;
    const void* groups = nullptr;
    uint32_t group_tiles = 0, tile_rows = 0;
    const uint32_t* row_map = nullptr;
};
bool gemm_tc_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* w, const void* x);
bool gemm_relaid_supported(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, const void* x);
uint64_t gemm_relaid_pitch(uint32_t layout, uint32_t k);
uint64_t gemm_relaid_bytes(uint32_t layout, uint32_t k, uint64_t rows);
size_t gemm_tc_workspace_bytes(uint32_t layout, uint32_t m, uint32_t k, uint32_t n, bool f32, bool precise);
int launch_gemm(cudaStream_t stream, uint32_t layout, const GemmCall& c, void* ws, size_t ws_bytes);
// n rows of row_bytes bytes -> rows of pitch bytes (a multiple of 16), zero behind the row.  With `used` (the exclusive
// scan of an expert stack's row counts) slabs of slab_rows rows that nobody is routed to are left out.
int launch_relay_rows(cudaStream_t stream, const uint8_t* w, uint64_t row_bytes, uint64_t n, uint8_t* out, uint64_t pitch,
                      const uint32_t* used = nullptr, uint32_t slab_rows = 1);
int launch_widen_q6(cudaStream_t stream, const uint8_t* w, uint32_t k, uint64_t n, uint8_t* out, const uint32_t* used = nullptr,
                    uint32_t slab_rows = 1);
// Whichever of the two makes `layout`: gemm_relaid_bytes(layout, k, n) bytes at out.
int launch_relay(cudaStream_t stream, uint32_t layout, const uint8_t* w, uint32_t k, uint64_t n, uint8_t* out, const uint32_t* used = nullptr,
                 uint32_t slab_rows = 1);

// f32 streaming GEMV (m <= 8) for rows of any length; with expert_idx, row i of x by the slab it names, all rows in one launch.
bool gemv_f32_supported(uint32_t scheme, uint32_t m, uint32_t k, const void* x);
int launch_gemv_f32(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y, bool ybf, uint32_t m,
                    uint32_t k, uint32_t n, const float* expert_idx = nullptr, uint32_t num_experts = 0);

// The same accuracy on the matrix instruction, for five to eight rows of the 32-weight formats and Q6_K: whether it is the faster one.
bool gemv_parts_pays(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, bool xbf, const void* x);
int launch_gemv_parts(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y, bool ybf, uint32_t m,
                      uint32_t k, uint32_t n);

// MoE decode rows: the slab of the weight stack is chosen by expert_sel[row] on the device.
bool int_expert_supported(uint32_t scheme, uint32_t k, uint32_t n, uint32_t rows, const void* w, const void* x, size_t* scratch);
int launch_gemv_int_expert(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w_stack, void* y,
                           bool ybf, uint32_t rows, uint32_t k, uint32_t n, uint32_t num_experts, const float* expert_sel, void* ws,
                           size_t ws_bytes);

struct TpPush;   // tp_comm.cuh: the exchange buffers of a tensor-parallel group (null: plain output)
int launch_gemv_int_swiglu(cudaStream_t stream, uint32_t scheme, const float* gu, const uint8_t* w, void* y, bool ybf,
                           uint32_t m, uint32_t k, uint32_t n, void* ws, size_t ws_bytes, const TpPush* tp = nullptr);

int staged_device_error(int* value);   // synchronises the device
int* static_error_word_if_resolved();  // error word inside the library image, once an allocation-free call resolved it
int staged_prepare_device();           // allocates the per-device error word (call outside capture)

// Shape-based selection used by rlxq_matmul / rlxq_workspace_bytes.
size_t matmul_workspace_bytes(uint32_t scheme, uint32_t m, uint32_t k, uint32_t n, uint32_t x_dtype, uint32_t y_dtype);
int dispatch_matmul(cudaStream_t stream, uint32_t scheme, const void* x, bool xbf, const uint8_t* w, void* y,
                    bool ybf, uint32_t m, uint32_t k, uint32_t n, void* ws, size_t ws_bytes);

}  // namespace rlxq
