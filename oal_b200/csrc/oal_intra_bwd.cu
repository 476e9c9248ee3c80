// Intra-chunk term of the chunked scan on the tensor cores (tcgen05 / TMEM), backward.
//
// Query side (rows are query rows, columns are keys).  dW = G [v|1]^T once (G as hi + lo bf16).  The gradient needs the
// scores of each group, s_g = sum over the group's dims of q k, and no term of the factored weight: with s_0 = 1,
//   X_r = dW s_r               registers -> tensor memory, bf16 value + remainder,  r = 0 .. G
//   Z_r = X_r K                one accumulator per r
//   dq  += e_r * Z_r           element-wise in the dimension d of group g: e_0 = scale B_g, e_r = 2 scale^2 C_rg
//   y_r  = sum over rows of q * Z_r, one 64-vector per row block
// s_g is one MMA chain over the rows of q with the other groups' dims set to zero, exact in bf16.  dB_g and dC_rg are
// sums of y_0 and y_r over the dims of g: 64 sums per r instead of G (G + 1) / 2 products per pair.  X_r's remainder
// keeps these strongly cancelling sums (sum_j dW_ij w_ij = 0 for every row) at 16 bits.
//
// Key / value side (rows are keys, columns are the queries of one head): per head and term r of the factored weight
// (oal_intra.cuh; the scaled rows as bf16 value + remainder: the rounding of the scaled keys alone would act like a
// perturbation that is the same for every query)
//   P_r^T = 2 dW^T u_r^T (bf16 value; with its remainder above 8 groups),  Z_r = P_r^T Q,  dk += sgn_r l_r * Z_r,  w += sgn_r u_r^2 in registers,
// and after the last term dU += W^T G (W as value + remainder, as in the forward: a row's weights and its denominator
// then agree to 16 bits).  A CTA walks several query heads of its KV head; dk stays in registers, dU
// in tensor memory, and the next head's operands arrive while the current one is worked on.
//
// The cross-chunk parts computed by the state kernels arrive as fp32 buffers and are added before the final cast.
// Reference stages replaced: oal_attention/hd_block_gemm_backward_wave.py:253-476 (dS, local dphi_q / dphi_k / dU
// GEMMs) and the folds / coefficient partials of oal_attention/hd_block_gemm_feature_backward.py:59-474.
#include "oal_intra.cuh"
#include "oal_kernels.h"

namespace oal {
namespace {

using namespace umma;

struct IntraBwdArgs {
  // operand images: rows of q, k [heads, NB, 8, 128, 8], [v | 1 | 0] and G [heads, NB, 10, 128, 8]
  const unsigned char *q_image, *k_image, *u_image;
  const unsigned char* gimg;        // bf16(G), then (gimg_lo_offset bytes on) the images of G - bf16(G)
  size_t gimg_lo_offset;
  const HeadFactor* factors;
  __nv_bfloat16* dq;                // may be null
  const float* dq_init;             // fp32 cross part, or null
  float* coef_partial;              // [B][Hq][row blocks][1 + G + G (G + 1) / 2] or null: dA, dB, upper triangle of dC
  float scale;
  // key / value side: fp32 partials [B, Hkv * parts, N, 64] when the heads are spread over `parts` CTAs, else the
  // results with the cross parts of the tokens before cross_end added
  float *dk_part, *dv_part;
  const float *dk_cross, *dv_cross;
  __nv_bfloat16 *dk, *dv;
  int cross_end, heads_per_cta, parts;
  int32_t* status;
  int N, NB, Hq, Hkv, rep, rank;    // rank = groups + 1, the same for every head of a call
  int cross_from;                   // first chunk that has a cross-chunk part in dq_init
};

// Warps 0..15 compute, warp 16 issues; 17..19 only fill the issuer's warpgroup, whose registers the compute warps
// take: 640 threads x 96 at launch = 512 x 112 + 128 x 24 and 1024 to spare.
constexpr int BW_COMPUTE = 16, BW_ISSUER = BW_COMPUTE, BW_THREADS = (BW_COMPUTE + 4) * 32;

// dW[128, n] = rows . cols^T over the 80-long augmented value axis; the side given as hi + lo is walked twice.
__device__ __forceinline__ void issue_dw(uint32_t tmem_dw, uint64_t rows_hi, uint64_t rows_lo, uint32_t rows_step, uint64_t cols_hi,
                                         uint64_t cols_lo, uint32_t cols_step, int n) {
  const uint32_t idesc = instr_desc_bf16(128, n, 0, 0);
#pragma unroll
  for (int ks = 0; ks < 2 * (EP / 16); ++ks) {
    const int lo = ks / (EP / 16), kk = ks % (EP / 16);
    mma_bf16_ss(tmem_dw, desc_advance(lo ? rows_lo : rows_hi, kk * rows_step), desc_advance(lo ? cols_lo : cols_hi, kk * cols_step),
                idesc, ks > 0);
  }
}

__device__ __forceinline__ f32x2 f2_shfl_xor(f32x2 v, int o) {
  float lo, hi;
  f2_unpack(v, lo, hi);
  return f2_pack(__shfl_xor_sync(0xffffffffu, lo, o), __shfl_xor_sync(0xffffffffu, hi, o));
}

// ---------------------------------------------------------------------------
// query side
// ---------------------------------------------------------------------------
// What bounds it: the chain score chain -> products -> X -> Z of each r (about 2000 clocks; the MMAs of an r are 1250) and the
// first and last phase of a tile.  Eight compute warps with 64 keys each, one barrier of theirs per r: it says at once that
// the scores have been read, X is written, the next masked rows are in place and the Z before last has been drained.
// 14 / 2 heads, 8 groups, B = 4, N = 4096: 353 -> 204 us against walking the terms of the factored weight (scaled rows as value +
// remainder, twice the MMA steps, 16 warps with 32 keys each and six barriers per term); of a tile's 32000 clocks 20000 are the
// loop.
// Warps 0..7 compute, warp 8 issues; 9..11 only help to load and fill the issuer's warpgroup, whose registers the compute
// warps take: 384 threads x 168 at launch = 256 x 224 + 128 x 40 and 2048 to spare.
constexpr int BQ_COMPUTE = 8, BQ_ISSUER = BQ_COMPUTE, BQ_THREADS = (BQ_COMPUTE + 4) * 32;
// tensor memory: scores (128; first dW) | X hi (64) | X lo (64) | two Z (64) | two slots of masked rows (32)
constexpr uint32_t BQ_S = 0, BQ_X = 128, BQ_XLO = 192, BQ_Z = 256, BQ_ROWS = 384, BQ_ROW_COLS = 32;
static_assert(BQ_ROWS + 2 * BQ_ROW_COLS <= 512, "tensor-memory columns of the query-side kernel");
// shared memory: images of q, k, [v | 1] and G (hi, lo), then of each quadrant's head
constexpr int BQ_K = ROW_IMAGE_BYTES, BQ_U = BQ_K + ROW_IMAGE_BYTES, BQ_G = BQ_U + SLAB_S_BYTES;
constexpr int BQ_E = BQ_G + 2 * SLAB_S_BYTES;                           // e_r[d], [quadrant][r][64] fp32
constexpr int BQ_MASK = BQ_E + 4 * RMAX_ALL * HD * 4;                   // dims of a group, [quadrant][group][32] words of two bf16
constexpr int BQ_ORDER = BQ_MASK + 4 * GMAX * (HD / 2) * 4;
constexpr int BQ_SMEM = BQ_ORDER + 4 * (int)sizeof(HeadOrder);
static_assert(4 * RMAX_ALL * HD * 4 <= 2 * SLAB_S_BYTES, "the y sums take the place of the images of G");

__global__ void __launch_bounds__(BQ_THREADS, 1) intra_bwd_q_kernel(const IntraBwdArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Qimg = smem;
  float* e_s = reinterpret_cast<float*>(smem + BQ_E);
  uint32_t* mask_s = reinterpret_cast<uint32_t*>(smem + BQ_MASK);
  float* ys = reinterpret_cast<float*>(smem + BQ_G);            // [quadrant][r][64], dims sorted by group; G is dead once dW is complete
  __shared__ float sum_s[BQ_COMPUTE], cls_s[4][RMAX_ALL * GMAX];
  __shared__ uint64_t in_full, dw_full, s_full, x_full, z_full;
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const QueryTile tile(a.Hkv, a.N, a.rep);
  if (tile.empty()) return;
  const int qd = warp & 3, row = 32 * qd + lane;
  const int tok0 = tile.c * CT, cols = tile.columns(), G = a.rank - 1;
  const int my_rb = tile.rb(qd), my_head = tile.head(qd);
  if (warp == 0) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    mbar_init(&in_full, 1);
    mbar_init(&dw_full, 1);
    mbar_init(&s_full, 1);
    mbar_init(&x_full, BQ_COMPUTE);
    mbar_init(&z_full, 1);
    mbar_fence_init();
    mbar_arrive_expect_tx(&in_full, ROW_IMAGE_BYTES + SLAB_S_BYTES +
                                        4 * ((8 + 2 * (EP / 8)) * 512 + a.rank * HD * 4 + G * (HD / 2) * 4 + (int)sizeof(HeadOrder)));
    dead = 0;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp >= BQ_ISSUER) {
    // a copy per thread: the key side whole, 32 rows of a plane at a time of each quadrant's rows and G, its head's tables
    constexpr int PER = 8 + 2 * (EP / 8) + 3;
    static_assert(4 * PER + 2 <= 128, "a copy per thread");
    const int x = tid - BQ_ISSUER * 32, quadrant = x & 3, y = x >> 2;
    const size_t unit = ((size_t)tile.b * a.Hkv + tile.kvh) * a.NB + tile.c;
    const size_t head = ((size_t)tile.b * a.Hq + tile.head(quadrant)) * a.NB + tile.c, rows = 32 * tile.rb(quadrant) * 16;
    const HeadFactor* f = a.factors + tile.head(quadrant);
    const int dst = 32 * quadrant * 16;
    if (y < 8) bulk_g2s(smem + y * ROW_PLANE + dst, a.q_image + head * ROW_IMAGE_BYTES + y * ROW_PLANE + rows, 512, &in_full);
    else if (y < 8 + 2 * (EP / 8)) {
      const int lo = y - 8 >= EP / 8, e = y - 8 - lo * (EP / 8);
      bulk_g2s(smem + BQ_G + lo * SLAB_S_BYTES + e * ROW_PLANE + dst, a.gimg + lo * a.gimg_lo_offset + head * SLAB_S_BYTES + e * ROW_PLANE + rows,
               512, &in_full);
    } else if (y == PER - 3) bulk_g2s(e_s + quadrant * RMAX_ALL * HD, &f->e[0][0], a.rank * HD * 4, &in_full);
    else if (y == PER - 2) bulk_g2s(mask_s + quadrant * GMAX * (HD / 2), &f->mask[0][0], G * (HD / 2) * 4, &in_full);
    else if (y == PER - 1) bulk_g2s(smem + BQ_ORDER + quadrant * (int)sizeof(HeadOrder), &f->order, (int)sizeof(HeadOrder), &in_full);
    else if (x == 4 * PER) bulk_g2s(smem + BQ_K, a.k_image + unit * ROW_IMAGE_BYTES, ROW_IMAGE_BYTES, &in_full);
    else if (x == 4 * PER + 1) bulk_g2s(smem + BQ_U, a.u_image + unit * SLAB_S_BYTES, SLAB_S_BYTES, &in_full);
  }
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);
  const uint32_t lane_off = (uint32_t)(32 * qd) << 16;
  const bool want_coef = a.coef_partial != nullptr;
  w.wait(&in_full, 0, 0x20);
  __syncwarp();

  if (warp >= BQ_ISSUER) {
    registers_down_to<40>();
    if (warp == BQ_ISSUER && elect_one()) {
      const uint32_t k_addr = smem_u32(smem + BQ_K), g_addr = smem_u32(smem + BQ_G), u_addr = smem_u32(smem + BQ_U);
      const uint64_t du = smem_desc(u_addr, ROW_PLANE, 128), dk_rows = smem_desc(k_addr, ROW_PLANE, 128), dk_dims = smem_desc(k_addr, 128, ROW_PLANE);
      const uint32_t idesc_s = instr_desc_bf16(128, cols, 0, 0), idesc_z = instr_desc_bf16(128, HD, 0, 1);
      issue_dw(tmem + BQ_S, smem_desc(g_addr, ROW_PLANE, 128), smem_desc(g_addr + SLAB_S_BYTES, ROW_PLANE, 128), 2 * ROW_PLANE, du, du,
               2 * ROW_PLANE, cols);
      mma_commit(&dw_full);
      for (int r = 0; r <= G; ++r) {
        w.wait(&x_full, r & 1, 0x21);
        fence_after_sync();
        if (r < G) {
          const uint32_t slot = tmem + BQ_ROWS + ((r + 1) & 1) * BQ_ROW_COLS;
#pragma unroll
          for (int ks = 0; ks < HD / 16; ++ks)
            mma_bf16_ts(tmem + BQ_S, slot + 8 * ks, desc_advance(dk_rows, ks * 2 * ROW_PLANE), idesc_s, ks > 0);
          mma_commit(&s_full);
        }
        const uint32_t z = tmem + BQ_Z + (r & 1) * HD;
        for (int ks = 0; ks < cols / 16; ++ks) {
          mma_bf16_ts(z, tmem + BQ_X + 8 * ks, desc_advance(dk_dims, ks * 256), idesc_z, ks > 0);
          mma_bf16_ts(z, tmem + BQ_XLO + 8 * ks, desc_advance(dk_dims, ks * 256), idesc_z, 1);
        }
        mma_commit(&z_full);
      }
    }
    __syncwarp();
  } else {
    registers_up_to<224>();
    const int sub = warp >> 2, m = lane & 3, d0 = 32 * sub;
    const int my_key = 32 * my_rb + lane;
    // this warp's keys: half of every 32, in blocks of 16; blocks behind the diagonal stay zero in X
    const auto key_of = [&](int x) { return 32 * x + 16 * sub; };
    const auto on = [&](int x) { return 32 * x < cols && x <= my_rb; };
    // rows of q with only the dims of group r - 1, as the A operand: 32 dims per warp
    const auto build = [&](int r) {
      const uint32_t* mask = mask_s + (qd * GMAX + r - 1) * (HD / 2) + d0 / 2;
      const uint32_t slot = tmem + BQ_ROWS + (r & 1) * BQ_ROW_COLS + lane_off + d0 / 2;
      uint32_t o[16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 x = *reinterpret_cast<const uint4*>(Qimg + (d0 / 8 + c) * ROW_PLANE + row * 16);
        const uint4 k = *reinterpret_cast<const uint4*>(mask + 4 * c);
        o[4 * c] = x.x & k.x; o[4 * c + 1] = x.y & k.y; o[4 * c + 2] = x.z & k.z; o[4 * c + 3] = x.w & k.w;
      }
      tmem_st16(slot, o);
    };
    // eight pairs of products as bf16 value and remainder, into the columns of one block of 16 keys
    const auto store_x = [&](int x, const uint32_t (&hi)[8], const uint32_t (&lo)[8]) {
      tmem_st8(tmem + BQ_X + lane_off + key_of(x) / 2, hi);
      tmem_st8(tmem + BQ_XLO + lane_off + key_of(x) / 2, lo);
    };
    const auto split = [&](const f32x2 (&t)[8], uint32_t (&hi)[8], uint32_t (&lo)[8]) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float t0, t1;
        f2_unpack(t[j], t0, t1);
        hi[j] = pack_bf16(t0, t1);
        lo[j] = pack_bf16(t0 - bf16_lo(hi[j]), t1 - bf16_hi(hi[j]));
      }
    };
    // q rows lane / 4 + 8 t, dims d0 + 8 i + 2 m, + 1: the arrangement in which Z is drained
    uint32_t qp[4][4];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        qp[t][i] = *reinterpret_cast<const uint32_t*>(Qimg + (d0 / 8 + i) * ROW_PLANE + (32 * qd + (lane >> 2) + 8 * t) * 16 + 4 * m);
    // the dimension whose sum this lane ends up with, in group order
    const HeadOrder& order = *reinterpret_cast<const HeadOrder*>(smem + BQ_ORDER + qd * (int)sizeof(HeadOrder));
    float* y_out = ys + qd * RMAX_ALL * HD + order.pos[d0 + 16 * (lane >> 4) + 8 * ((lane >> 3) & 1) + 2 * m + ((lane >> 2) & 1)];
    build(1);
    {
      const uint32_t zero[8] = {};
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (32 * x < cols && !on(x)) store_x(x, zero, zero);
    }
    f32x2 dw[4][8];
    f32x2 sum2 = 0ull;
    w.wait(&dw_full, 0, 0x22);
    __syncwarp();
    fence_after_sync();
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (on(x)) {
        float d[16];
        tmem_ld16(tmem + BQ_S + lane_off + key_of(x), d);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int kj = key_of(x) + 2 * j;
          dw[x][j] = f2_pack(kj <= my_key ? d[2 * j] : 0.f, kj + 1 <= my_key ? d[2 * j + 1] : 0.f);
          sum2 = f2_add(sum2, dw[x][j]);
        }
        uint32_t hi[8], lo[8];
        split(dw[x], hi, lo);
        store_x(x, hi, lo);
      }
    tmem_st_wait();
    fence_before_sync();
    warp_arrive(&x_full, lane);
    f32x2 dq[4][4];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) dq[t][i] = 0ull;
    // Z_r: dq, and the sums over the 32 rows of q * Z (one warp holds all rows of its block)
    const auto drain = [&](int r) {
      float z[2][16];
      const uint32_t at = tmem + BQ_Z + (r & 1) * HD + lane_off + d0;
      tmem_ld_rows16(at, z[0]);
      tmem_ld_rows16(at + (16u << 16), z[1]);
      const float* e = e_s + (qd * RMAX_ALL + r) * HD + d0 + 2 * m;
      f32x2 ev[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) ev[i] = *reinterpret_cast<const f32x2*>(e + 8 * i);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const f32x2 z2 = f2_pack(z[t >> 1][4 * i + 2 * (t & 1)], z[t >> 1][4 * i + 2 * (t & 1) + 1]);
          dq[t][i] = f2_fma(ev[i], z2, dq[t][i]);
          const f32x2 q2 = f2_pack(bf16_lo(qp[t][i]), bf16_hi(qp[t][i]));
          y[i] = t ? f2_fma(q2, z2, y[i]) : f2_mul(q2, z2);
        }
      if (!want_coef) return;
      // over the eight lanes with the same dims, halving what is carried: lane bit 4 picks i / 2, bit 3 i % 2, bit 2 the element
      const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
      const f32x2 u0 = f2_add(b4 ? y[2] : y[0], f2_shfl_xor(b4 ? y[0] : y[2], 16));
      const f32x2 u1 = f2_add(b4 ? y[3] : y[1], f2_shfl_xor(b4 ? y[1] : y[3], 16));
      const f32x2 u = f2_add(b3 ? u1 : u0, f2_shfl_xor(b3 ? u0 : u1, 8));
      float v0, v1;
      f2_unpack(u, v0, v1);
      const float v = (b2 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, b2 ? v0 : v1, 4);
      y_out[r * HD] = v;
    };
    for (int r = 1; r <= G; ++r) {
      // the next rows' slot was last read for the scores of r - 1, which have arrived
      if (r < G) build(r + 1);
      w.wait(&s_full, (r - 1) & 1, 0x23);
      __syncwarp();
      fence_after_sync();
      float sc[2][16];
      uint32_t hi[2][8], lo[2][8];
      const auto products = [&](int x, int k) {
        f32x2 t[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) t[j] = f2_mul(dw[x][j], f2_pack(sc[k][2 * j], sc[k][2 * j + 1]));
        split(t, hi[k], lo[k]);
      };
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (on(x)) tmem_ld16(tmem + BQ_S + lane_off + key_of(x), sc[x]);
      tmem_ld_wait();
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (on(x)) products(x, x);
#pragma unroll
      for (int x = 2; x < 4; ++x)
        if (on(x)) tmem_ld16(tmem + BQ_S + lane_off + key_of(x), sc[x - 2]);
      tmem_ld_wait();
      w.wait(&z_full, (r - 1) & 1, 0x24);            // X of r - 1 has been read
      __syncwarp();
      fence_after_sync();
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (on(x)) store_x(x, hi[x], lo[x]);
#pragma unroll
      for (int x = 2; x < 4; ++x)
        if (on(x)) {
          products(x, x - 2);
          store_x(x, hi[x - 2], lo[x - 2]);
        }
      tmem_st_wait();
      fence_before_sync();
      warp_arrive(&x_full, lane);
      drain(r - 1);
    }
    const int rows = max(tile.nc - 32 * my_rb, 0);            // of the row block that exist
    const size_t out0 = (((size_t)tile.b * a.Hq + my_head) * a.N + tok0 + 32 * my_rb + (lane >> 2)) * HD + d0 + 2 * m;
    float2 cross[4][4];
    const bool add_cross = a.dq && a.dq_init && tile.c >= a.cross_from;
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        cross[t][i] = add_cross && (lane >> 2) + 8 * t < rows ? *reinterpret_cast<const float2*>(a.dq_init + out0 + 8 * t * HD + 8 * i)
                                                               : make_float2(0.f, 0.f);
    w.wait(&z_full, G & 1, 0x25);
    __syncwarp();
    fence_after_sync();
    drain(G);
    if (a.dq && !dead) {
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if ((lane >> 2) + 8 * t < rows) {
            float v0, v1;
            f2_unpack(dq[t][i], v0, v1);
            *reinterpret_cast<uint32_t*>(a.dq + out0 + 8 * t * HD + 8 * i) = pack_bf16(v0 + cross[t][i].x, v1 + cross[t][i].y);
          }
    }
    if (want_coef) {
      float s0, s1;
      f2_unpack(sum2, s0, s1);
      s0 += s1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      if (lane == 0) sum_s[warp] = s0;
      // the quadrant's two warps: sums of y over the dims of each group, then dA, dB and dC (symmetrised: both orders are
      // the same sum)
      asm volatile("bar.sync %0, 64;" ::"r"(1 + qd) : "memory");
      const float* y = ys + qd * RMAX_ALL * HD;
      for (int x = sub * 32 + lane; x < a.rank * G; x += 64) {
        const int r = x / G, g = x % G, end = order.start[g + 1];
        float t = 0.f;
#pragma unroll 4
        for (int p = order.start[g]; p < end; ++p) t += y[r * HD + p];
        cls_s[qd][x] = t;
      }
      asm volatile("bar.sync %0, 64;" ::"r"(1 + qd) : "memory");
      const int slots = 1 + G + G * (G + 1) / 2, blocks = (a.N + 31) / 32;
      float* dst = a.coef_partial + (((size_t)tile.b * a.Hq + my_head) * blocks + tile.c * 4 + my_rb) * slots;
      for (int x = sub * 32 + lane; x < slots && rows > 0; x += 64) {
        float t;
        if (x == 0) {
          t = sum_s[qd] + sum_s[4 + qd];
        } else if (x <= G) {
          t = a.scale * cls_s[qd][x - 1];
        } else {
          int g = 0, rest = x - 1 - G;
          while (rest >= G - g) { rest -= G - g; ++g; }
          t = 0.5f * a.scale * a.scale * (cls_s[qd][(1 + g) * G + g + rest] + cls_s[qd][(1 + g + rest) * G + g]);
        }
        dst[x] = t;
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
}

// ---------------------------------------------------------------------------
// key / value side: one CTA per (chunk, KV head, batch row) and group of query heads; rows are keys
// ---------------------------------------------------------------------------
// tensor memory: U (two halves of 64; first dW^T of a head) | P^T (64), later W^T | their remainders (64) | Z (64) | dU (64) |
// two term slots (64)
constexpr uint32_t BK_U = 0, BK_P = 128, BK_PLO = 192, BK_Z = 256, BK_V = 320, BK_TERM = 384;
static_assert(BK_TERM + 2 * TERM_COLS <= 512, "tensor-memory columns of the key/value-side kernel");
constexpr int BK_HEAD_L = RMAX_ALL * HD * 4;
constexpr int BK_HEAD_BYTES = ROW_IMAGE_BYTES + 2 * SLAB_S_BYTES + BK_HEAD_L;       // Q image, G hi, G lo, l: one head's operands
constexpr int BK_SMEM = ROW_IMAGE_BYTES + SLAB_S_BYTES + 2 * BK_HEAD_BYTES;
static_assert(BK_HEAD_BYTES % 16 == 0 && BK_SMEM <= 227 * 1024, "shared memory of the key/value-side kernel");

// FINE: P^T with its remainders and W^T against both images of G, for heads of more than 8 groups.  Their weights were
// formed and summed in fp32 (oal_pairs.cu) before these kernels took them over, and the bf16 values alone were up to 1.24
// times as far from 64 bits in dv and 1.18 times in dk (14 / 2 heads, N = 347, 16 groups: 2.13e-3 -> 2.64e-3 and 2.14e-3 ->
// 2.52e-3); up to 8 groups the bf16 values are nearer than the tiles that they replaced (dk 3.3e-3 -> 2.8e-3).
template <bool FINE>
__global__ void __launch_bounds__(BW_THREADS, 1) intra_bwd_kv_kernel(const IntraBwdArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Kimg = smem;
  unsigned char* Uimg = Kimg + ROW_IMAGE_BYTES;
  unsigned char* heads = Uimg + SLAB_S_BYTES;                   // two sets of a head's operands
  __shared__ __align__(16) HeadScalars sc[2];
  __shared__ uint64_t u_in, g_full[2], dw_full, dw_free, u_full[2], u_free[2], term_full[2], p_full[2], z_half[2], z_free, w_full, v_full;
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int part = blockIdx.z, c = blockIdx.x, b = blockIdx.y / a.Hkv, kvh = blockIdx.y - b * a.Hkv;
  const int h0 = part * a.heads_per_cta, n_heads = min(a.heads_per_cta, a.rep - h0), rank = a.rank;
  const int qd = warp & 3, sub = (warp >> 2) & 3, row = 32 * qd + lane;     // row: key index inside the chunk
  const int tok0 = c * CT, nc = min(CT, a.N - tok0), cols = (nc + 31) & ~31;
  const size_t koff = ((size_t)b * a.Hkv + kvh) * a.N + tok0;
  const auto head_of = [&](int i) { return kvh * a.rep + h0 + i; };
  if (warp == 0) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&g_full[s], 1);
      mbar_init(&u_full[s], 1);
      mbar_init(&u_free[s], BW_COMPUTE);
      mbar_init(&term_full[s], BW_COMPUTE);
      mbar_init(&p_full[s], BW_COMPUTE);
      mbar_init(&z_half[s], 1);
    }
    mbar_init(&dw_full, 1);
    mbar_init(&dw_free, BW_COMPUTE);
    mbar_init(&z_free, BW_COMPUTE);
    mbar_init(&w_full, BW_COMPUTE);
    mbar_init(&v_full, 1);
    mbar_init(&u_in, 1);
    mbar_fence_init();
    dead = 0;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);
  const uint32_t lane_off = (uint32_t)(32 * qd) << 16;
  const int na = min(cols, 64), nb2 = cols - na;              // columns of the two halves

  if (warp >= BW_ISSUER) {
    registers_down_to<24>();
    if (warp == BW_ISSUER) {
      if (elect_one()) {
        const uint32_t u_addr = smem_u32(Uimg);
        const size_t unit = ((size_t)b * a.Hkv + kvh) * a.NB + c;
        mbar_arrive_expect_tx(&u_in, ROW_IMAGE_BYTES + SLAB_S_BYTES);
        bulk_g2s(Kimg, a.k_image + unit * ROW_IMAGE_BYTES, ROW_IMAGE_BYTES, &u_in);
        bulk_g2s(Uimg, a.u_image + unit * SLAB_S_BYTES, SLAB_S_BYTES, &u_in);
        const auto fetch_head = [&](int i) {                  // rows of q, both images of G, l and scalars of head i
          unsigned char* dst = heads + (i & 1) * BK_HEAD_BYTES;
          const size_t at = ((size_t)b * a.Hq + head_of(i)) * a.NB + c;
          const HeadFactor* f = a.factors + head_of(i);
          uint64_t* bar = &g_full[i & 1];
          mbar_arrive_expect_tx(bar, ROW_IMAGE_BYTES + 2 * SLAB_S_BYTES + rank * HD * 4 + (int)sizeof(HeadScalars));
          bulk_g2s(dst, a.q_image + at * ROW_IMAGE_BYTES, ROW_IMAGE_BYTES, bar);
          bulk_g2s(dst + ROW_IMAGE_BYTES, a.gimg + at * SLAB_S_BYTES, SLAB_S_BYTES, bar);
          bulk_g2s(dst + ROW_IMAGE_BYTES + SLAB_S_BYTES, a.gimg + a.gimg_lo_offset + at * SLAB_S_BYTES, SLAB_S_BYTES, bar);
          bulk_g2s(dst + ROW_IMAGE_BYTES + 2 * SLAB_S_BYTES, &f->l[0][0], rank * HD * 4, bar);
          bulk_g2s(&sc[i & 1], &f->s, (int)sizeof(HeadScalars), bar);
        };
        fetch_head(0);
        w.wait(&u_in, 0, 0x32);
        int T = 0;                                            // terms issued so far, over all heads
        for (int i = 0; i < n_heads; ++i) {
          const uint32_t q_addr = smem_u32(heads + (i & 1) * BK_HEAD_BYTES), g_addr = q_addr + ROW_IMAGE_BYTES;
          if (i + 1 < n_heads) {
            if (i > 0) w.wait(&v_full, (i - 1) & 1, 0x30);    // head i - 1 no longer reads the set that head i + 1 takes
            fetch_head(i + 1);
          }
          w.wait(&g_full[i & 1], (i >> 1) & 1, 0x31);
          if (T > 0) {
            w.wait(&u_free[0], (T - 1) & 1, 0x33);
            w.wait(&u_free[1], (T - 1) & 1, 0x34);
          }
          fence_after_sync();
          // dW^T[j, i] = [v|1]_j . g_i: rows from the U image, columns from the hi and lo images of G
          const uint64_t du = smem_desc(u_addr, ROW_PLANE, 128);
          issue_dw(tmem + BK_U, du, du, 2 * ROW_PLANE, smem_desc(g_addr, CT * 16, 128), smem_desc(g_addr + SLAB_S_BYTES, CT * 16, 128),
                   2 * CT * 16, cols);
          mma_commit(&dw_full);
          const uint64_t dq = smem_desc(q_addr, 128, ROW_PLANE), dg = smem_desc(g_addr, 128, CT * 16);
          const uint64_t dg_lo = smem_desc(g_addr + SLAB_S_BYTES, 128, CT * 16);
          const auto issue_z = [&](int t, int hf) {
            w.wait(&p_full[hf], t & 1, 0x35);
            if (hf == 0 && t > 0) w.wait(&z_free, (t - 1) & 1, 0x36);
            fence_after_sync();
            const int k0 = hf ? 4 : 0, k1 = hf ? 4 + nb2 / 16 : na / 16;
            for (int part = 0; part < (FINE ? 2 : 1); ++part)
              for (int ks = k0; ks < k1; ++ks)
                mma_bf16_ts(tmem + BK_Z, tmem + (part ? BK_PLO : BK_P) + 8 * ks, desc_advance(dq, ks * 256),
                            instr_desc_bf16(128, HD, 0, 1), part + ks > 0);
            mma_commit(&z_half[hf]);
          };
          for (int r = 0; r < rank; ++r, ++T) {
            const uint32_t slot = tmem + BK_TERM + (T & 1) * TERM_COLS;
            w.wait(&term_full[T & 1], (T >> 1) & 1, 0x37);
            if (r > 0) w.wait(&u_free[0], (T - 1) & 1, 0x38);
            else w.wait(&dw_free, i & 1, 0x39);
            fence_after_sync();
            issue_term<ROW_PLANE>(tmem + BK_U, slot, q_addr, na);
            mma_commit(&u_full[0]);
            if (r > 0) {
              issue_z(T - 1, 0);
              w.wait(&u_free[1], (T - 1) & 1, 0x3A);
            }
            if (nb2) {
              fence_after_sync();
              issue_term<ROW_PLANE>(tmem + BK_U + 64, slot, q_addr + 64 * 16, nb2);
            }
            mma_commit(&u_full[1]);            // also: the term's slot has been read
            if (r > 0) issue_z(T - 1, 1);
          }
          issue_z(T - 1, 0);
          issue_z(T - 1, 1);
          w.wait(&w_full, i & 1, 0x3B);
          fence_after_sync();
          // dU (+)= W^T G: the weights' bf16 values, then their remainders, then the values against G's remainders
          for (int part = 0; part < (FINE ? 3 : 2); ++part)
            for (int ks = 0; ks < cols / 16; ++ks)
              mma_bf16_ts(tmem + BK_V, tmem + (part == 1 ? BK_PLO : BK_P) + 8 * ks, desc_advance(part == 2 ? dg_lo : dg, ks * 256),
                          instr_desc_bf16(128, HD, 0, 1), i + part + ks > 0);
          mma_commit(&v_full);
        }
      }
      __syncwarp();
    }
  } else {
    registers_up_to<112>();
    const unsigned char* xrow = Kimg + row * 16;
    const int d0 = 16 * sub;
    // this warp's queries: a quarter of each half, in blocks of 8; blocks before the diagonal stay zero in P^T and W^T
    const auto col_of = [&](int hf, int x) { return 64 * hf + sub * ((hf ? nb2 : na) / 4) + 8 * x; };
    const auto exists = [&](int hf, int x) { return 32 * x < (hf ? nb2 : na); };
    const auto on = [&](int hf, int x) { return exists(hf, x) && col_of(hf, x) + 7 >= 32 * qd; };
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (exists(hf, x) && !on(hf, x)) {
          tmem_st4(tmem + BK_P + lane_off + col_of(hf, x) / 2, 0u, 0u, 0u, 0u);
          tmem_st4(tmem + BK_PLO + lane_off + col_of(hf, x) / 2, 0u, 0u, 0u, 0u);
        }
    w.wait(&u_in, 0, 0x3F);
    f32x2 dk[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) dk[j] = 0ull;
    int T = 0;
    for (int i = 0; i < n_heads; ++i) {
      const float* l = reinterpret_cast<const float*>(heads + (i & 1) * BK_HEAD_BYTES + ROW_IMAGE_BYTES + 2 * SLAB_S_BYTES);
      const HeadScalars& hs = sc[i & 1];
      w.wait(&g_full[i & 1], (i >> 1) & 1, 0x3C);             // l and the scalars are read below
      if (i > 0) w.wait(&v_full, (i - 1) & 1, 0x3D);          // W^T of the previous head has been read
      __syncwarp();
      const int rpos = uniform(hs.rpos);
      const auto build = [&](int r) {
        build_term16<ROW_PLANE>(tmem + BK_TERM + ((T + r) & 1) * TERM_COLS + lane_off, xrow, l + r * HD, d0);
        tmem_st_wait();
        fence_before_sync();
        warp_arrive(&term_full[(T + r) & 1], lane);
      };
      build(0);
      f32x2 dw[2][2][4], wt[2][2][4];
      w.wait(&dw_full, i & 1, 0x3E);
      fence_after_sync();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf)
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (on(hf, x)) {
            float d[8];
            tmem_ld8(tmem + BK_U + lane_off + col_of(hf, x), d);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int i0 = col_of(hf, x) + 2 * j;             // query not earlier than the key
              dw[hf][x][j] = f2_pack(i0 >= row ? 2.f * d[2 * j] : 0.f, i0 + 1 >= row ? 2.f * d[2 * j + 1] : 0.f);
              wt[hf][x][j] = f2_bcast(hs.w0);
            }
          }
      fence_before_sync();
      warp_arrive(&dw_free, lane);
      const auto drain = [&](int r) {
        float z[16];
        tmem_ld16(tmem + BK_Z + lane_off + d0, z);
        tmem_ld_wait();
        fence_before_sync();
        warp_arrive(&z_free, lane);
        const f32x2 sgn = f2_bcast(r < rpos ? 1.f : -1.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const ulonglong2 lv = *reinterpret_cast<const ulonglong2*>(l + r * HD + d0 + 4 * j);
          dk[2 * j] = f2_fma(f2_mul(lv.x, sgn), f2_pack(z[4 * j], z[4 * j + 1]), dk[2 * j]);
          dk[2 * j + 1] = f2_fma(f2_mul(lv.y, sgn), f2_pack(z[4 * j + 2], z[4 * j + 3]), dk[2 * j + 1]);
        }
      };
      for (int r = 0; r < rank; ++r) {
        // the next term is built while the MMAs of this one run; its slot's last reader was term r - 1, complete
        // since u_full[1](r - 1)
        if (r + 1 < rank) build(r + 1);
        const f32x2 c2 = f2_bcast(hs.c[r]), sgn = f2_bcast(r < rpos ? 1.f : -1.f);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          w.wait(&u_full[hf], (T + r) & 1, 0x40 + hf);
          fence_after_sync();
          float u[2][8];
#pragma unroll
          for (int x = 0; x < 2; ++x)
            if (on(hf, x)) tmem_ld8(tmem + BK_U + lane_off + col_of(hf, x), u[x]);
          tmem_ld_wait();
          fence_before_sync();
          warp_arrive(&u_free[hf], lane);
          uint32_t p[2][4], rest[2][4];
#pragma unroll
          for (int x = 0; x < 2; ++x)
            if (on(hf, x)) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const f32x2 u2 = f2_add(f2_pack(u[x][2 * j], u[x][2 * j + 1]), c2);
                float t0, t1;
                f2_unpack(f2_mul(dw[hf][x][j], u2), t0, t1);
                p[x][j] = pack_bf16(t0, t1);
                if (FINE) rest[x][j] = pack_bf16(t0 - bf16_lo(p[x][j]), t1 - bf16_hi(p[x][j]));
                wt[hf][x][j] = f2_fma(rpos == rank ? u2 : f2_mul(u2, sgn), u2, wt[hf][x][j]);
              }
            }
          if (r > 0) {                         // the previous term's P^T has been read
            w.wait(&z_half[hf], (T + r - 1) & 1, 0x42 + hf);
            fence_after_sync();
          }
#pragma unroll
          for (int x = 0; x < 2; ++x)
            if (on(hf, x)) {
              const uint32_t at = lane_off + col_of(hf, x) / 2;
              tmem_st4(tmem + BK_P + at, p[x][0], p[x][1], p[x][2], p[x][3]);
              if (FINE) tmem_st4(tmem + BK_PLO + at, rest[x][0], rest[x][1], rest[x][2], rest[x][3]);
            }
          tmem_st_wait();
          fence_before_sync();
          // the whole Z of the previous term is complete: out of the way before the next one starts
          if (hf == 1 && r > 0) drain(r - 1);
          warp_arrive(&p_full[hf], lane);
        }
      }
      w.wait(&z_half[0], (T + rank - 1) & 1, 0x44);
      w.wait(&z_half[1], (T + rank - 1) & 1, 0x45);
      fence_after_sync();
      drain(rank - 1);
      // W^T and its remainders in the place of P^T and its, whose last readers are complete
#pragma unroll
      for (int hf = 0; hf < 2; ++hf)
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (on(hf, x)) {
            uint32_t o[4], rest[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float w_a, w_b;
              f2_unpack(wt[hf][x][j], w_a, w_b);
              const int i0 = col_of(hf, x) + 2 * j;
              if (i0 < row) w_a = 0.f;
              if (i0 + 1 < row) w_b = 0.f;
              o[j] = pack_bf16(w_a, w_b);
              rest[j] = pack_bf16(w_a - bf16_lo(o[j]), w_b - bf16_hi(o[j]));
            }
            const uint32_t at = lane_off + col_of(hf, x) / 2;
            tmem_st4(tmem + BK_P + at, o[0], o[1], o[2], o[3]);
            tmem_st4(tmem + BK_PLO + at, rest[0], rest[1], rest[2], rest[3]);
          }
      tmem_st_wait();
      fence_before_sync();
      warp_arrive(&w_full, lane);
      T += rank;
    }
    w.wait(&v_full, (n_heads - 1) & 1, 0x46);
    fence_after_sync();
    float z[16], v[16];
    tmem_ld16(tmem + BK_V + lane_off + d0, z);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j) f2_unpack(dk[j], v[2 * j], v[2 * j + 1]);
    if (row < nc && !dead) {
      // 16 consecutive dims of a row per thread: whole sectors
      const auto write = [&](float (&x)[16], float* partial, const float* cross, __nv_bfloat16* out) {
        if (partial) {
          float* dst = partial + ((((size_t)b * a.Hkv + kvh) * a.parts + part) * a.N + tok0 + row) * HD + d0;
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(dst + 4 * j) = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        } else if (out) {
          const size_t o = (koff + row) * HD + d0;
          if (cross && tok0 + row < a.cross_end) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float4 t = *reinterpret_cast<const float4*>(cross + o + 4 * j);
              x[4 * j] += t.x; x[4 * j + 1] += t.y; x[4 * j + 2] += t.z; x[4 * j + 3] += t.w;
            }
          }
#pragma unroll
          for (int j = 0; j < 2; ++j)
            *reinterpret_cast<uint4*>(out + o + 8 * j) =
                make_uint4(pack_bf16(x[8 * j], x[8 * j + 1]), pack_bf16(x[8 * j + 2], x[8 * j + 3]),
                           pack_bf16(x[8 * j + 4], x[8 * j + 5]), pack_bf16(x[8 * j + 6], x[8 * j + 7]));
        }
      };
      write(v, a.dk_part, a.dk_cross, a.dk);
      write(z, a.dv_part, a.dv_cross, a.dv);
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
}

// dk / dv = cross-chunk part (tokens before cross_end) + sum over the parts (groups of query heads of the KV head) of
// their shares, fixed order, cast to bf16.  One thread per 4 consecutive dims of one key token; blockIdx.y: dk, then dv.
struct KvReduceArgs {
  const float *part[2], *cross[2];
  __nv_bfloat16* out[2];
  int B, Hkv, parts, N, cross_end;
};
__global__ void __launch_bounds__(256) kv_head_reduce_kernel(const KvReduceArgs a) {
  const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x;       // over B*Hkv*N*16
  const size_t total = (size_t)a.B * a.Hkv * a.N * 16;
  __nv_bfloat16* out = a.out[blockIdx.y];
  if (idx >= total || !out) return;
  const float *part = a.part[blockIdx.y], *cross = a.cross[blockIdx.y];
  const int d4 = (int)(idx & 15);
  const size_t tok = idx >> 4;                                     // (b*Hkv + kvh)*N + n
  const int n = (int)(tok % a.N);
  const size_t bk = tok / a.N;
  float4 acc = n < a.cross_end ? *reinterpret_cast<const float4*>(cross + tok * HD + 4 * d4) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float* src = part + ((bk * a.parts) * a.N + n) * HD + 4 * d4;
#pragma unroll 8
  for (int r = 0; r < a.parts; ++r) {
    const float4 t = *reinterpret_cast<const float4*>(src + (size_t)r * a.N * HD);
    acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
  }
  *reinterpret_cast<uint2*>(out + tok * HD + 4 * d4) = make_uint2(pack_bf16(acc.x, acc.y), pack_bf16(acc.z, acc.w));
}

IntraBwdArgs bwd_args(const RowImages& rows, const void* gimg, const void* factors,
                      int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups) {
  IntraBwdArgs a{};
  a.q_image = static_cast<const unsigned char*>(rows.q_image); a.k_image = static_cast<const unsigned char*>(rows.k_image);
  a.u_image = static_cast<const unsigned char*>(rows.u_image); a.gimg = static_cast<const unsigned char*>(gimg);
  a.factors = static_cast<const HeadFactor*>(factors);
  a.status = status;
  a.N = N; a.NB = NB; a.Hq = Hq; a.Hkv = Hkv; a.rep = Hq / Hkv; a.rank = groups + 1;
  a.gimg_lo_offset = (size_t)B * Hq * NB * SLAB_S_BYTES;
  return a;
}

}  // namespace

int intra_row_blocks(int N) { return (N + 31) / 32; }

cudaError_t intra_backward_q(const RowImages& rows, const void* gimg, const void* factors, void* dq, const float* dq_init,
                             float* coef_partial, int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups, float scale,
                             int cross_from, cudaStream_t st) {
  cudaError_t e = allow_smem<intra_bwd_q_kernel>(BQ_SMEM);
  if (e != cudaSuccess) return e;
  IntraBwdArgs a = bwd_args(rows, gimg, factors, status, B, Hq, Hkv, N, NB, groups);
  a.scale = scale;
  a.dq = static_cast<__nv_bfloat16*>(dq); a.dq_init = dq_init; a.coef_partial = coef_partial; a.cross_from = cross_from;
  intra_bwd_q_kernel<<<dim3(NB, B * Hkv, Hq / Hkv), BQ_THREADS, BQ_SMEM, st>>>(a);
  return cudaGetLastError();
}

// Heads of a KV head per CTA of the key/value side: all of them when that still fills the machine (dk and dv then
// leave the kernel finished: no fp32 partials of every head, no reduction kernel), else the fewest parts that do.
int intra_kv_parts(int B, int Hq, int Hkv, int NB) {
  const int rep = Hq / Hkv, groups = B * Hkv * NB, sms = sm_count();
  int best = 1;
  double best_cost = 1e30;
  for (int parts = 1; parts <= rep; ++parts) {
    const int heads = (rep + parts - 1) / parts;
    if (parts > 1 && (rep + heads - 1) / heads != parts) continue;       // the same split with fewer parts
    const int waves = (groups * parts + sms - 1) / sms;
    // a head costs one unit, the CTA's own prologue and epilogue about half of one, partials another third per head
    const double cost = waves * (heads + 0.5) + (parts > 1 ? 0.3 * groups * parts / sms : 0.);
    if (cost < best_cost) { best_cost = cost; best = parts; }
  }
  return best;
}

cudaError_t intra_backward_kv(const RowImages& rows, const void* gimg, const void* factors,
                              void* dk, void* dv, const float* dk_cross, const float* dv_cross, int cross_end, float* dk_part,
                              float* dv_part, int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups,
                              cudaStream_t st) {
  const bool fine = groups > 8;
  cudaError_t e = fine ? allow_smem<intra_bwd_kv_kernel<true>>(BK_SMEM) : allow_smem<intra_bwd_kv_kernel<false>>(BK_SMEM);
  if (e != cudaSuccess) return e;
  IntraBwdArgs a = bwd_args(rows, gimg, factors, status, B, Hq, Hkv, N, NB, groups);
  a.parts = intra_kv_parts(B, Hq, Hkv, NB);
  a.heads_per_cta = (Hq / Hkv + a.parts - 1) / a.parts;
  a.cross_end = cross_end;
  if (a.parts > 1) {
    a.dk_part = dk ? dk_part : nullptr;
    a.dv_part = dv ? dv_part : nullptr;
  } else {
    a.dk = static_cast<__nv_bfloat16*>(dk); a.dv = static_cast<__nv_bfloat16*>(dv);
    a.dk_cross = dk_cross; a.dv_cross = dv_cross;
  }
  const dim3 grid(NB, B * Hkv, a.parts);
  if (fine) intra_bwd_kv_kernel<true><<<grid, BW_THREADS, BK_SMEM, st>>>(a);
  else intra_bwd_kv_kernel<false><<<grid, BW_THREADS, BK_SMEM, st>>>(a);
  if (a.parts == 1 || (e = cudaGetLastError()) != cudaSuccess) return cudaGetLastError();
  KvReduceArgs r{{dk_part, dv_part}, {dk_cross, dv_cross}, {static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv)},
                 B, Hkv, a.parts, N, cross_end};
  const size_t total = (size_t)B * Hkv * N * 16;
  kv_head_reduce_kernel<<<dim3((unsigned)((total + 255) / 256), 2), 256, 0, st>>>(r);
  return cudaGetLastError();
}

}  // namespace oal
