// Internal launch interface between the C-ABI translation unit and the kernel files.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace oal {

struct PrologueArgs;      // oal_prologue.cuh

// Delivery of a call's status word to pinned host memory by the last block of its last kernel: `counter` (device, zero
// at the start of that kernel) counts finished blocks.  host == null: not delivered.
struct StatusSink {
  int32_t* counter;
  volatile int32_t* host;
};
constexpr int32_t STATUS_DELIVERED = (int32_t)0x80000000;

// Arguments of the token-pair kernels (oal_pairs.cu).
struct PairArgs {
  int B, Hq, Hkv, N, G;
  int io_dt, out_dt;
  float scale, floor;
  const void *q, *k, *v;
  const int32_t *dim_perm, *group_start;
  const float *A, *Bc, *Cc;
  int32_t* status;
  // forward
  void* out;
  float *num, *den;
  StatusSink sink;       // forward
  // backward
  const float* g;        // [B,Hq,N,80] augmented upstream gradient
  void *dq, *dk, *dv;
  float* coef_partial;   // [B][Hq][tiles][split][NCOEF] or null
  float *dk_part, *dv_part;      // [B,Hq,N,64] fp32, where a KV head has several query heads
  // set by the launch: 64-token tiles, CTAs that share a tile, which of q, k, v, num (bits) allow accesses of four elements
  int tiles, split, vec;
};

cudaError_t pairs_forward(const PairArgs& a, cudaStream_t st);
cudaError_t pairs_backward_q(const PairArgs& a, cudaStream_t st);
cudaError_t pairs_backward_kv(const PairArgs& a, cudaStream_t st);
int pairs_tiles(int n);
int pairs_split(int B, int Hq, int N);      // partial sums of the coefficient gradient per tile

cudaError_t norm_vjp(const void* grad_out, int out_dt, const float* grad_num, const float* grad_den,
                     const float* num, const float* den, float floor_v, float* g, size_t rows,
                     int32_t* clear_status, cudaStream_t st);

// extra: [Hq][NCOEF] slots already summed over the batch (cross-chunk term), or null
cudaError_t reduce_coefs(const float* p0, int tiles0, const float* extra, int B, int Hq, int G,
                         float* dA, float* dB, float* dC, cudaStream_t st);

// ---- tensor-core state kernels (oal_state.cu) ---------------------------------------
// rotary embedding fused with the layout move between [B, N, H, 64] and [B, H, N, 64] (bf16)
cudaError_t rope_to_heads(const void* src, void* dst, const float* cosv, const float* sinv, int B, int N, int H,
                          bool rotate, cudaStream_t st);
cudaError_t rope_to_flat(const void* src, void* dst, const float* cosv, const float* sinv, int B, int N, int H,
                         bool rotate, cudaStream_t st);

size_t state_rows();                       // feature rows of the running state (2432)
size_t state_image_bytes_per_chunk();      // bytes of one bf16 state image [19 slabs][10][128][8]
size_t state_slab_image_bytes();           // bytes of one slab image [10][128][8] bf16

cudaError_t build_coef_table(const int32_t* dim_perm, const int32_t* group_start, const float* A,
                             const float* Bc, const float* Cc, int Hq, int G, float scale, float* table,
                             cudaStream_t st);
// increments of the first NC chunks
cudaError_t state_update(const void* k, const void* v, float* ds, int units, int N, int NB, int NC, int32_t* status, cudaStream_t st);
// Operand images of the rows of q and k [B*H, NB, 8, 128, 8] and of [v | 1 | 0] [B*Hkv, NB, 10, 128, 8].
struct RowImages {
  const void *q, *k, *v;
  void *q_image, *k_image, *u_image;
};
// images of k and [v | 1]; `prologue` (optional): its blocks ride in the same launch
cudaError_t rows_prologue(const RowImages& rows, int units, int N, int NB, const PrologueArgs* prologue, int q_heads, cudaStream_t st);
// both images of every chunk (trim: but the first), the running state kept on chip; state_walk_pays: faster than state_update
// and state_scan
bool state_walk_pays(int units, int NB);
cudaError_t state_walk(const RowImages& rows, void* image, void* image_lo, const float* state_in, int units, int NB, bool trim,
                       int32_t* status, cudaStream_t st);
// image_lo: optional second image holding bf16(state - bf16(state)); trim: see state_scan_kernel
cudaError_t state_scan(const float* ds, void* image, void* image_lo, const float* state_in, float* state_total,
                       int units, int NB, int reverse, bool trim, cudaStream_t st);
// chunks [c0, c0 + NC) of every sequence; the other rows of out64 / out1 are not written
cudaError_t cross_read(bool query, const void* x, const void* image, const float* coef_table, float* out64,
                       float* out1, int B, int H, int rep, int N, int NB, int c0, int NC, int32_t* status, cudaStream_t st);


// ---- tensor-core backward kernels (oal_state_bwd.cu): chunks [c0, c0 + NC) of every sequence ----------
// carry_img / carry_lo: the saved state image and its remainder image (both or neither)
cudaError_t dstate_heads(const void* q_image, const void* gimg, const void* carry_img, const void* carry_lo, const float* coef_table,
                         float* dcarry, float* dcoef_partial, int B, int Hq, int Hkv, int NB, int c0, int NC, float scale,
                         int32_t* status, cudaStream_t st);
// query: x_image, a_image = images of q and G; else of k and [v | 1]
cudaError_t feature_grad(bool query, const void* x_image, const void* a_image, const void* image,
                         const float* coef_table, float* dx, int B, int H, int rep, int N, int NB, int c0, int NC,
                         int32_t* status, cudaStream_t st);
cudaError_t dcoef_reduce(const float* partial, int outer, int Hq, int G, const int32_t* dim_perm,
                         const int32_t* group_start, float* dcoef, float* slots, cudaStream_t st);
// writes the images of G and of q
cudaError_t norm_vjp_image(const void* grad_out, int out_dt, const float* grad_num, const float* grad_den,
                           const float* num, const float* den, float floor_v, void* gimg, int heads,
                           int N, int NB, int token_major_heads /* > 0: grad_out is [B, N, Hq, 64] */, const RowImages& rows,
                           int32_t* clear_status, cudaStream_t st);


// ---- factored intra-chunk weight (oal_factor.cu) -----------------------------------------
// Per-head table of the factored quadratic form (c_r, l_r[d], back-transform, sign split).
size_t head_factor_bytes(int Hq);
// Packed lower-triangular factor rows [factor_rows (1 or Hq), (G+1)(G+2)/2] -> A, B, C, and the transpose map.
cudaError_t expand_factor(const float* factor, int factor_rows, int Hq, int G, float eps, float* A, float* B, float* C,
                          cudaStream_t st);
cudaError_t expand_factor_grad(const float* factor, int factor_rows, int Hq, int G, const float* dA, const float* dB,
                               const float* dC, float* dfactor, cudaStream_t st);
cudaError_t build_head_factors(const int32_t* dim_perm, const int32_t* group_start, const float* A, const float* Bc,
                               const float* Cc, int Hq, int G, float scale, void* table, cudaStream_t st);
// dA, dB, dC = sum of the query-side partial sums [B][Hq][tiles][1 + G + G (G + 1) / 2] (dA, dB, upper triangle of dC) +
// extra ([Hq][NCOEF] slots of the cross-chunk term, or null); dfactor (optional): the gradient of `factor`, a row per head.
cudaError_t intra_coef_finish(const float* partial, int tiles, const float* extra, int B, int Hq, int G, float* dA, float* dB,
                              float* dC, const float* factor, float* dfactor, cudaStream_t st);
cudaError_t launch_head_prologue(const PrologueArgs& a, int Hq, cudaStream_t st);
// writes *status | STATUS_DELIVERED to the sink's host word
cudaError_t deliver_status(const int32_t* status, StatusSink sink, cudaStream_t st);

// ---- tensor-core intra-chunk kernels (oal_intra.cu, oal_intra_bwd.cu) ----------------------------
// cross_from: first chunk that has a cross-chunk part in num / den (dq_init)
cudaError_t intra_forward(const void* q, const void* k, const void* v, const void* factors, void* out, float* num,
                          float* den, int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups, int out_dt,
                          float floor_v, bool out_token_major, int cross_from, StatusSink sink, cudaStream_t st);
int intra_row_blocks(int N);     // row blocks per head: partial sums of the coefficient gradient
cudaError_t intra_backward_q(const RowImages& rows, const void* gimg, const void* factors,
                             void* dq, const float* dq_init, float* coef_partial, int32_t* status, int B, int Hq,
                             int Hkv, int N, int NB, int groups, float scale, int cross_from, cudaStream_t st);
int intra_kv_parts(int B, int Hq, int Hkv, int NB);     // CTAs the heads of a KV head are spread over
// dk, dv: null where not requested; *_cross: fp32 cross-chunk parts of the tokens before cross_end; *_part: scratch of
// B * Hq * N * 64 floats
cudaError_t intra_backward_kv(const RowImages& rows, const void* gimg, const void* factors,
                              void* dk, void* dv, const float* dk_cross, const float* dv_cross, int cross_end, float* dk_part,
                              float* dv_part, int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups, cudaStream_t st);

}  // namespace oal
