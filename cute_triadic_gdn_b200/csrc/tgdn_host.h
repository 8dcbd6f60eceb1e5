// Host-side helpers shared by the translation units of libtgdn_b200 (not part of the public ABI).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tgdn.h"
#include "../../include/tgdn_selftest.h"

// -(1000 + e) for a CUDA runtime error, 0 for cudaSuccess.
int tgdn_cuda_error(cudaError_t e);

// Device pointer of the status word of the current device (a __device__ int of this library).
int* tgdn_status_word();

// Tensor map over a (B, T, H, 128) bf16 tensor in token layout: box = [box_cols columns][1 head][box_rows tokens][1 row].
// swizzle = 1 asks for the swizzle as wide as a row of the box (box_cols 64, 32 or 16).  row_tokens: tokens from one batch row to the next
// (0: T), for a token range of longer rows.
int tgdn_make_token_map(CUtensorMap* map, const void* base, int B, int T, int H, int box_cols, int box_rows, int swizzle,
                        int row_tokens = 0);

// The same tensors for boxes that land in shared memory as operand images [column / 8][64 tokens][column % 8]: coordinates
// (0, token, first 8-column block, head, batch row), box_blocks blocks of 1 KB.
int tgdn_make_image_map(CUtensorMap* map, const void* base, int B, int T, int H, int box_blocks, int row_tokens = 0);

// Tensor map over the [A; Pm A] images whose boxes are the A half of one item (8 KB, an image of 64 rows): coordinates (0, 0, 0, 0, item).
int tgdn_make_a_half_map(CUtensorMap* map, const void* base, long long items);

// Tensor map over a (B, T, H, E) f32 gate tensor (k2, q2) in token layout, E a multiple of 4: box = [E][1 head][64 tokens][1 row],
// which lands in shared memory as 64 dense rows of E floats.
int tgdn_make_gate_map(CUtensorMap* map, const float* base, int B, int T, int H, int E, int row_tokens = 0);

// Tensor map over a (B, T, C) bf16 tensor with element strides (stride_b, stride_t, 1): box = [box_cols][box_rows][1], no swizzle.
int tgdn_make_rows_map(CUtensorMap* map, const void* base, int C, int T, int B, int64_t stride_t, int64_t stride_b, int box_cols,
                       int box_rows);

// True when the current device is compute capability 10.x; also binds the device's primary context to the calling thread.
int tgdn_check_device();

// Opts a kernel in to `bytes` of dynamic shared memory on the current device, once per device (configured[64]).
int tgdn_dynamic_smem(const void* kernel, int bytes, bool* configured);

// The core stages on a token range of longer rows: the arguments of the entry points of the same name (include/tgdn.h) plus
// row_tokens >= T, the tokens from one batch row to the next in every token-layout tensor (inputs and outputs; the chunk-layout
// tensors are those of the T tokens alone).  Dense rows; the entry points of the public ABI are these with row_tokens = T.
int tgdn_masks_rows(const void* q, const void* k, const float* k2, const float* q2, const float* g, const float* beta, float scale,
                    const int32_t* chunk_map, int B, int T, int H, int E, int NC, int row_tokens, float* gc, void* AP, void* Pm,
                    void* stream);
int tgdn_fwd_rows(const void* q, const void* k, const void* v, const float* k2, const float* q2, const float* beta, const float* gc,
                  const void* AP, float scale, const int32_t* doc_offsets, const int32_t* chunk_map, int n_docs, int B, int T, int H,
                  int E, int NC, int row_tokens, void* o, void* W, void* U, void* h, const float* state_in, float* state_out,
                  void* stream);
int tgdn_bwd_recurrent_rows(const void* q, const void* k, const void* dO, const float* k2, const float* q2, const float* beta,
                            const float* gc, const void* AP, const void* Pm, const void* U, float scale, const int32_t* doc_offsets,
                            const int32_t* chunk_map, int n_docs, int B, int T, int H, int E, int NC, int row_tokens, void* dV,
                            void* dU, void* ds, void* dkg, float* dr, const float* grad_state_in, float* grad_state_out,
                            void* stream, int* zeroed = nullptr);   // zeroed: a word that the kernel sets to zero, or nullptr
int tgdn_bwd_state_grads_rows(const void* q, const void* k, const void* dO, const void* dV, const void* h, const void* ds,
                              const void* dkg, const float* k2, const float* q2, const float* gc, float scale,
                              const int32_t* chunk_map, int B, int T, int H, int E, int NC, int row_tokens, void* dkq, float* da,
                              float* dc, float* dd, void* stream);
int tgdn_bwd_matrix_rows(const void* q, const void* k, const void* dO, const void* dU, const void* W, const void* U, const void* AP,
                         const float* k2, const float* q2, const float* beta, const float* gc, const void* dkq, const float* da,
                         const float* dc, const float* dd, const float* dr, float scale, const int32_t* chunk_map, int B, int T,
                         int H, int E, int NC, int row_tokens, void* dq, void* dk, float* dk2, float* dq2, float* dg, float* dbeta,
                         void* stream);
// The state gradients and the matrix gradients in one kernel, bitwise the two above one after the other.  next_item: a word of the call's own
// that is zero when the kernel starts (tgdn_bwd_recurrent_rows can zero it).
int tgdn_bwd_grads_rows(const void* q, const void* k, const void* dO, const void* dV, const void* dU, const void* W, const void* U,
                        const void* AP, const void* h, const void* ds, const void* dkg, const float* k2, const float* q2,
                        const float* beta, const float* gc, const float* dr, float scale, const int32_t* chunk_map, int B, int T, int H,
                        int E, int NC, int row_tokens, int* next_item, void* dq, void* dk, float* dk2, float* dq2, float* dg, float* dbeta, void* stream);

// The convolution for any channel count, strides and 2-byte aligned rows (weight: 8-byte aligned); the entry points of the public ABI
// are these for whole 16-byte pieces.  The backward uses as many weight-gradient partials as the scratch holds, up to
// tgdn_conv_bwd_best_scratch.
int tgdn_conv_fwd_any(const void* x, const void* weight, void* y, const int32_t* cu, int n_docs, int B, int T, int C, int64_t stride_b,
                      int64_t stride_t, int act_channels, void* stream);
int tgdn_conv_bwd_any(const void* x, const void* weight, const void* dy, void* dx, void* dw, const int32_t* cu, int n_docs, int B, int T,
                      int C, int64_t stride_b, int64_t stride_t, int64_t dy_stride_b, int64_t dy_stride_t, int act_channels,
                      void* scratch, int64_t scratch_bytes, void* stream);
int64_t tgdn_conv_bwd_best_scratch(int B, int T, int C);

// The whole backward of tgdn_glue_fwd: from the gradients of q, k, v, k2, q2 to dx (B, T, C) and dw (C, 4) without the gradient of the
// convolution's output in between (except for the gate channels: dy_gates, bf16 (B, T, 2 H E)).  scratch as for the convolution.
int tgdn_glue_bwd(const void* x, const void* weight, const int32_t* cu, int n_docs, int B, int T, int C, int64_t stride_b, int64_t stride_t,
                  int H, int E, float eps, const void* dq, const void* dk, const void* dv, const float* dk2, const float* dq2, void* dx,
                  void* dw, void* dy_gates, void* scratch, int64_t scratch_bytes, void* stream);

// Value columns of a block of the reverse recurrence: dkg (rounded per block) and dr have 128 / tgdn_value_block(E) of them.
int tgdn_value_block(int E);
