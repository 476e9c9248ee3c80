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
// A call of one chunk that wants coefficient gradients takes the terms of the factored weight instead (oal_intra.cuh; u_r as
// the forward formed it, from the scaled rows of q):
//   X_r = dW u_r,  dq += 2 sgn_r l_r * Z_r,  D[r][r'] = sum dW u_r u_r' from y_r,  dC = t D t^T,  dB = t sum dW u_r
// The forward's weights carry the rounding of its scaled rows, about 5e-6 of a row's numerator and denominator, and so does
// dW.  With the same terms sum_j dW_ij w_ij still cancels; with exact scores it does not, and where no bf16 features (2e-3 of
// dfactor from 129 tokens on) hide it what is left was the largest error.  dfactor against 64 bits, 14 heads, 33 to 128
// tokens, geometric mean of 40 inputs, terms / scores: 8 groups 1.13 / 1.22e-5, 12 groups 0.92 / 1.08e-5, 16 groups 0.94 /
// 1.19e-5; from 129 tokens on the same within 0.2 %.  The kernel at N = 128: 8 groups 22 / 17 us, 16 groups 38 / 26 us.
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
// first and last phase of a tile.  One barrier of the compute warps per r: it says at once that
// the scores have been read, X is written, the next masked rows are in place and the Z before last has been drained.
// 14 / 2 heads, 8 groups, B = 4, N = 4096: 353 -> 194 us against walking the terms of the factored weight (scaled rows as value +
// remainder, twice the MMA steps and six barriers per term).
// Warps 0..15 compute (with eight of twice the keys and dims 201 us), warp 16 issues; 17..19 only help to load and fill the
// issuer's warpgroup, whose registers the compute warps take: 640 threads x 96 at launch = 512 x 112 + 128 x 32.
constexpr int BQ_SUBS = 4, BQ_COMPUTE = 4 * BQ_SUBS, BQ_ISSUER = BQ_COMPUTE, BQ_THREADS = (BQ_COMPUTE + 4) * 32;
// tensor memory: scores (128; first dW) | X hi (64) | X lo (64) | two Z (64) | two slots of masked rows (32) or terms (64)
constexpr uint32_t BQ_S = 0, BQ_X = 128, BQ_XLO = 192, BQ_Z = 256, BQ_ROWS = 384, BQ_ROW_COLS = 32;
static_assert(BQ_ROWS + 2 * TERM_COLS <= 512, "tensor-memory columns of the query-side kernel");
// shared memory: images of q, k, [v | 1] and G (hi, lo), then of each quadrant's head
constexpr int BQ_K = ROW_IMAGE_BYTES, BQ_U = BQ_K + ROW_IMAGE_BYTES, BQ_G = BQ_U + SLAB_S_BYTES;
constexpr int BQ_E = BQ_G + 2 * SLAB_S_BYTES;                           // e_r[d], [quadrant][r][64] fp32
constexpr int BQ_MASK = BQ_E + 4 * RMAX_ALL * HD * 4;                   // dims of a group, [quadrant][group][32] words of two bf16
constexpr int BQ_ORDER = BQ_MASK + 4 * GMAX * (HD / 2) * 4;
constexpr int BQ_SMEM = BQ_ORDER + 4 * (int)sizeof(HeadOrder);
// TERMS: l, t and the scalars in the places of e, the masks and the order
constexpr int BQ_Y = 4 * RMAX_ALL * HD, BQ_D = RMAX_ALL * RMAX_ALL;       // floats: y sums; D or t D of a quadrant
static_assert((BQ_Y + 8 * BQ_D) * 4 <= 2 * SLAB_S_BYTES, "the y sums, D and t D take the place of the images of G");
static_assert(sizeof(HeadFactor::t) <= GMAX * (HD / 2) * 4 && sizeof(HeadScalars) <= sizeof(HeadOrder), "a quadrant's tables of either form");

template <bool TERMS>
__global__ void __launch_bounds__(BQ_THREADS, 1) intra_bwd_q_kernel(const IntraBwdArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Qimg = smem;
  float* e_s = reinterpret_cast<float*>(smem + BQ_E);
  uint32_t* mask_s = reinterpret_cast<uint32_t*>(smem + BQ_MASK);
  float* ys = reinterpret_cast<float*>(smem + BQ_G);            // [quadrant][r][64], dims sorted by group; G is dead once dW is complete
  __shared__ float sum_s[BQ_COMPUTE], cls_s[TERMS ? 1 : 4][RMAX_ALL * GMAX], n_s[TERMS ? BQ_COMPUTE : 1][RMAX_ALL];
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
                                        4 * ((8 + 2 * (EP / 8)) * 512 + a.rank * HD * 4 +
                                             (TERMS ? (int)(sizeof(HeadFactor::t) + sizeof(HeadScalars)) : G * (HD / 2) * 4 + (int)sizeof(HeadOrder))));
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
    } else if (y == PER - 3) bulk_g2s(e_s + quadrant * RMAX_ALL * HD, TERMS ? &f->l[0][0] : &f->e[0][0], a.rank * HD * 4, &in_full);
    else if (y == PER - 2) {
      if (TERMS) bulk_g2s(mask_s + quadrant * GMAX * (HD / 2), &f->t[0][0], (int)sizeof(f->t), &in_full);
      else bulk_g2s(mask_s + quadrant * GMAX * (HD / 2), &f->mask[0][0], G * (HD / 2) * 4, &in_full);
    } else if (y == PER - 1) {
      unsigned char* dst_head = smem + BQ_ORDER + quadrant * (int)sizeof(HeadOrder);
      if (TERMS) bulk_g2s(dst_head, &f->s, (int)sizeof(HeadScalars), &in_full);
      else bulk_g2s(dst_head, &f->order, (int)sizeof(HeadOrder), &in_full);
    }
    else if (x == 4 * PER) bulk_g2s(smem + BQ_K, a.k_image + unit * ROW_IMAGE_BYTES, ROW_IMAGE_BYTES, &in_full);
    else if (x == 4 * PER + 1) bulk_g2s(smem + BQ_U, a.u_image + unit * SLAB_S_BYTES, SLAB_S_BYTES, &in_full);
  }
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);
  const uint32_t lane_off = (uint32_t)(32 * qd) << 16;
  const bool want_coef = TERMS || a.coef_partial != nullptr;
  constexpr int FIRST = TERMS ? 0 : 1;                // first r whose X is a product with scores
  constexpr uint32_t SLOT_COLS = TERMS ? TERM_COLS : BQ_ROW_COLS;
  w.wait(&in_full, 0, 0x20);
  __syncwarp();

  if (warp >= BQ_ISSUER) {
    registers_down_to<32>();
    if (warp == BQ_ISSUER && elect_one()) {
      const uint32_t k_addr = smem_u32(smem + BQ_K), g_addr = smem_u32(smem + BQ_G), u_addr = smem_u32(smem + BQ_U);
      const uint64_t du = smem_desc(u_addr, ROW_PLANE, 128), dk_rows = smem_desc(k_addr, ROW_PLANE, 128), dk_dims = smem_desc(k_addr, 128, ROW_PLANE);
      const uint32_t idesc_s = instr_desc_bf16(128, cols, 0, 0), idesc_z = instr_desc_bf16(128, HD, 0, 1);
      issue_dw(tmem + BQ_S, smem_desc(g_addr, ROW_PLANE, 128), smem_desc(g_addr + SLAB_S_BYTES, ROW_PLANE, 128), 2 * ROW_PLANE, du, du,
               2 * ROW_PLANE, cols);
      mma_commit(&dw_full);
      for (int r = FIRST - 1, phase = 0; r <= G; ++r) {
        w.wait(&x_full, phase++ & 1, 0x21);
        fence_after_sync();
        if (r < G) {
          const uint32_t slot = tmem + BQ_ROWS + ((r + 1) & 1) * SLOT_COLS;
          if (TERMS) {
            issue_term<ROW_PLANE>(tmem + BQ_S, slot, k_addr, cols);
          } else {
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks)
              mma_bf16_ts(tmem + BQ_S, slot + 8 * ks, desc_advance(dk_rows, ks * 2 * ROW_PLANE), idesc_s, ks > 0);
          }
          mma_commit(&s_full);
        }
        if (r < 0) continue;
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
    registers_up_to<112>();
    constexpr int BLOCKS = 8 / BQ_SUBS, DIMS = HD / BQ_SUBS, PIECES = DIMS / 8;     // of 16 keys, dims and pieces of 8 dims per warp
    const int sub = warp >> 2, m = lane & 3, d0 = DIMS * sub;
    const int my_key = 32 * my_rb + lane;
    // this warp's keys: blocks of 16, half of some 32s; blocks behind the diagonal stay zero in X
    const auto block_of = [&](int x) { return x * (BQ_SUBS / 2) + (sub >> 1); };
    const auto key_of = [&](int x) { return 32 * block_of(x) + 16 * (sub & 1); };
    const auto exists = [&](int x) { return 32 * block_of(x) < cols; };
    const auto on = [&](int x) { return exists(x) && block_of(x) <= my_rb; };
    // TERMS: c_r, signs, l and t of the quadrant's head
    const HeadScalars& hs = *reinterpret_cast<const HeadScalars*>(smem + BQ_ORDER + qd * (int)sizeof(HeadOrder));
    const float* l = e_s + qd * RMAX_ALL * HD;
    const int rpos = TERMS ? uniform(hs.rpos) : 0;
    // rows of q with only the dims of group r - 1, or scaled by l_r, as the A operand
    const auto build = [&](int r) {
      if constexpr (TERMS) {
        static_assert(DIMS == 16, "a piece of a term");
        build_term16<ROW_PLANE>(tmem + BQ_ROWS + (r & 1) * SLOT_COLS + lane_off, Qimg + row * 16, l + r * HD, d0);
        return;
      }
      const uint32_t* mask = mask_s + (qd * GMAX + r - 1) * (HD / 2) + d0 / 2;
      const uint32_t slot = tmem + BQ_ROWS + (r & 1) * BQ_ROW_COLS + lane_off + d0 / 2;
#pragma unroll
      for (int c = 0; c < PIECES; c += 2) {
        uint32_t o[8];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const uint4 x = *reinterpret_cast<const uint4*>(Qimg + (d0 / 8 + c + y) * ROW_PLANE + row * 16);
          const uint4 k = *reinterpret_cast<const uint4*>(mask + 4 * (c + y));
          o[4 * y] = x.x & k.x; o[4 * y + 1] = x.y & k.y; o[4 * y + 2] = x.z & k.z; o[4 * y + 3] = x.w & k.w;
        }
        tmem_st8(slot + 4 * c, o);
      }
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
    uint32_t qp[4][PIECES];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int i = 0; i < PIECES; ++i)
        qp[t][i] = *reinterpret_cast<const uint32_t*>(Qimg + (d0 / 8 + i) * ROW_PLANE + (32 * qd + (lane >> 2) + 8 * t) * 16 + 4 * m);
    // the dimension whose sum this lane ends up with, in group order
    const HeadOrder& order = *reinterpret_cast<const HeadOrder*>(smem + BQ_ORDER + qd * (int)sizeof(HeadOrder));
    const int my_dim = d0 + 8 * (lane >> 4) + 2 * m + ((lane >> 3) & 1);
    float* y_out = ys + qd * RMAX_ALL * HD + (TERMS ? my_dim : order.pos[my_dim]);
    build(FIRST);
    {
      const uint32_t zero[8] = {};
#pragma unroll
      for (int x = 0; x < BLOCKS; ++x)
        if (exists(x) && !on(x)) store_x(x, zero, zero);
    }
    f32x2 dw[BLOCKS][8];
    f32x2 sum2 = 0ull;
    w.wait(&dw_full, 0, 0x22);
    __syncwarp();
    fence_after_sync();
#pragma unroll
    for (int x = 0; x < BLOCKS; ++x)
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
        if constexpr (TERMS) continue;
        uint32_t hi[8], lo[8];
        split(dw[x], hi, lo);
        store_x(x, hi, lo);
      }
    tmem_st_wait();
    fence_before_sync();
    warp_arrive(&x_full, lane);
    f32x2 dq[4][PIECES];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int i = 0; i < PIECES; ++i) dq[t][i] = 0ull;
    // Z_r: dq, and the sums over the 32 rows of q * Z (one warp holds all rows of its block)
    const auto drain = [&](int r) {
      float z[2][4 * PIECES];
      const uint32_t at = tmem + BQ_Z + (r & 1) * HD + lane_off + d0;
      tmem_ld_rows(at, z[0]);
      tmem_ld_rows(at + (16u << 16), z[1]);
      const float* e = e_s + (qd * RMAX_ALL + r) * HD + d0 + 2 * m;
      f32x2 ev[PIECES], y[PIECES];
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        ev[i] = *reinterpret_cast<const f32x2*>(e + 8 * i);
        if (TERMS) ev[i] = f2_mul(ev[i], f2_bcast(r < rpos ? 2.f : -2.f));
      }
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < PIECES; ++i)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const f32x2 z2 = f2_pack(z[t >> 1][4 * i + 2 * (t & 1)], z[t >> 1][4 * i + 2 * (t & 1) + 1]);
          dq[t][i] = f2_fma(ev[i], z2, dq[t][i]);
          const f32x2 q2 = f2_pack(bf16_lo(qp[t][i]), bf16_hi(qp[t][i]));
          y[i] = t ? f2_fma(q2, z2, y[i]) : f2_mul(q2, z2);
        }
      if (!want_coef) return;
      // over the eight lanes with the same dims, halving what is carried: first the pieces, then the two elements
      const bool b4 = lane & 16, b3 = lane & 8;
      float v0, v1;
      static_assert(PIECES == 2, "lane bit 4 picks the piece, bit 3 the element");
      f2_unpack(f2_add(b4 ? y[1] : y[0], f2_shfl_xor(b4 ? y[0] : y[1], 16)), v0, v1);
      float v = (b3 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, b3 ? v0 : v1, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      if ((lane & 4) == 0) y_out[r * HD] = v;
    };
    for (int r = FIRST; r <= G; ++r) {
      // the next rows' slot was last read for the scores of r - 1, which have arrived
      if (r < G) build(r + 1);
      const f32x2 c2 = f2_bcast(TERMS ? hs.c[r] : 0.f);
      f32x2 n2 = 0ull;
      w.wait(&s_full, (r - FIRST) & 1, 0x23);
      __syncwarp();
      fence_after_sync();
      uint32_t hi[BLOCKS / 2][8], lo[BLOCKS / 2][8];
      const auto products = [&](int x, int k) {
        float sc[16];
        tmem_ld16(tmem + BQ_S + lane_off + key_of(x), sc);
        tmem_ld_wait();
        f32x2 t[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const f32x2 s2 = f2_pack(sc[2 * j], sc[2 * j + 1]);
          t[j] = f2_mul(dw[x][j], TERMS ? f2_add(s2, c2) : s2);
          if (TERMS) n2 = f2_add(n2, t[j]);
        }
        split(t, hi[k], lo[k]);
      };
#pragma unroll
      for (int x = 0; x < BLOCKS / 2; ++x)
        if (on(x)) products(x, x);
      if (r > 0) w.wait(&z_full, (r - 1) & 1, 0x24);            // X of r - 1 has been read
      __syncwarp();
      fence_after_sync();
#pragma unroll
      for (int x = 0; x < BLOCKS / 2; ++x)
        if (on(x)) store_x(x, hi[x], lo[x]);
#pragma unroll
      for (int x = BLOCKS / 2; x < BLOCKS; ++x)
        if (on(x)) {
          products(x, x - BLOCKS / 2);
          store_x(x, hi[x - BLOCKS / 2], lo[x - BLOCKS / 2]);
        }
      tmem_st_wait();
      fence_before_sync();
      warp_arrive(&x_full, lane);
      if (r > 0) drain(r - 1);
      if constexpr (TERMS) {
        float n0, n1;
        f2_unpack(n2, n0, n1);
        n0 += n1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) n0 += __shfl_xor_sync(0xffffffffu, n0, o);
        if (lane == 0) n_s[warp][r] = n0;
      }
    }
    const int rows = max(tile.nc - 32 * my_rb, 0);            // of the row block that exist
    const size_t out0 = (((size_t)tile.b * a.Hq + my_head) * a.N + tok0 + 32 * my_rb + (lane >> 2)) * HD + d0 + 2 * m;
    float2 cross[4][PIECES];
    const bool add_cross = a.dq && a.dq_init && tile.c >= a.cross_from;
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int i = 0; i < PIECES; ++i)
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
        for (int i = 0; i < PIECES; ++i)
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
      // the quadrant's warps: dA, dB and the upper triangle of dC from the sums (symmetrised: both orders are the same sum)
      const auto quadrant_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + qd), "n"(BQ_SUBS * 32) : "memory"); };
      const auto triangle = [](int x, int n, int& i, int& j) {      // x-th entry of an upper triangle, row-major
        i = 0;
        while (x >= n - i) { x -= n - i; ++i; }
        j = i + x;
      };
      quadrant_sync();
      const float* y = ys + qd * RMAX_ALL * HD;
      const int slots = 1 + G + G * (G + 1) / 2, blocks = (a.N + 31) / 32, first = sub * 32 + lane;
      float* dst = a.coef_partial + (((size_t)tile.b * a.Hq + my_head) * blocks + tile.c * 4 + my_rb) * slots;
      if constexpr (TERMS) {
        const auto n_of = [&](int r) { return (n_s[qd][r] + n_s[4 + qd][r]) + (n_s[8 + qd][r] + n_s[12 + qd][r]); };
        const float* t = reinterpret_cast<const float*>(mask_s + qd * GMAX * (HD / 2));
        float *D = ys + BQ_Y + 2 * qd * BQ_D, *tD = D + BQ_D;
        const int rank = a.rank;
        for (int x = first; x < rank * (rank + 1) / 2; x += BQ_SUBS * 32) {
          int r, r2;
          triangle(x, rank, r, r2);
          float s = fmaf(hs.c[r2], n_of(r), hs.c[r] * n_of(r2));
#pragma unroll 4
          for (int k = 0; k < HD; k += 4) {
            const int d = (k + 4 * lane) % HD;                      // rows start in the same bank: every lane elsewhere
            const float4 la = *reinterpret_cast<const float4*>(l + r * HD + d), lb = *reinterpret_cast<const float4*>(l + r2 * HD + d);
            const float4 ya = *reinterpret_cast<const float4*>(y + r * HD + d), yb = *reinterpret_cast<const float4*>(y + r2 * HD + d);
            s = fmaf(lb.x, ya.x, fmaf(lb.y, ya.y, fmaf(lb.z, ya.z, fmaf(lb.w, ya.w, s))));
            s = fmaf(la.x, yb.x, fmaf(la.y, yb.y, fmaf(la.z, yb.z, fmaf(la.w, yb.w, s))));
          }
          D[r * RMAX_ALL + r2] = D[r2 * RMAX_ALL + r] = 0.5f * s;
        }
        quadrant_sync();
        for (int x = first; x < G * rank; x += BQ_SUBS * 32) {
          const int g = x / rank, r2 = x % rank;
          float s = 0.f;
#pragma unroll 4
          for (int r = 0; r < rank; ++r) s = fmaf(t[(1 + g) * T_PITCH + r], D[r * RMAX_ALL + r2], s);
          tD[g * RMAX_ALL + r2] = s;
        }
        quadrant_sync();
        for (int x = first; x < slots && rows > 0; x += BQ_SUBS * 32) {
          float s = 0.f;
          if (x == 0) {
            s = (sum_s[qd] + sum_s[4 + qd]) + (sum_s[8 + qd] + sum_s[12 + qd]);
          } else if (x <= G) {
            for (int r = 0; r < rank; ++r) s = fmaf(t[x * T_PITCH + r], n_of(r), s);
          } else {
            int g, g2;
            triangle(x - 1 - G, G, g, g2);
#pragma unroll 4
            for (int r = 0; r < rank; ++r) s = fmaf(tD[g * RMAX_ALL + r], t[(1 + g2) * T_PITCH + r], s);
          }
          dst[x] = s;
        }
      } else {
        for (int x = first; x < a.rank * G; x += BQ_SUBS * 32) {     // sums of y over the dims of each group
          const int r = x / G, g = x % G, end = order.start[g + 1];
          float t = 0.f;
#pragma unroll 4
          for (int p = order.start[g]; p < end; ++p) t += y[r * HD + p];
          cls_s[qd][x] = t;
        }
        quadrant_sync();
        for (int x = first; x < slots && rows > 0; x += BQ_SUBS * 32) {
          float t;
          if (x == 0) {
            t = 0.f;
#pragma unroll
            for (int y = 0; y < BQ_SUBS; ++y) t += sum_s[4 * y + qd];
          } else if (x <= G) {
            t = a.scale * cls_s[qd][x - 1];
          } else {
            int g, g2;
            triangle(x - 1 - G, G, g, g2);
            t = 0.5f * a.scale * a.scale * (cls_s[qd][(1 + g) * G + g2] + cls_s[qd][(1 + g2) * G + g]);
          }
          dst[x] = t;
        }
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  w.settle();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
}

// ---------------------------------------------------------------------------
// key / value side: one CTA per (chunk, KV head, batch row) and group of query heads; rows are keys
// ---------------------------------------------------------------------------
// What bounds it: as on the query side, the chain of a term (products, hand-over, Z), most of all on the quadrant of keys 0 to
// 31, which meets all queries (its scheduler issues 1.8 times the mean).  One barrier of the compute warps per term says that U has been read, P^T is written, the next
// term's rows are in place and the Z before last is drained; the next head's dW^T is computed while W^T of this one is stored.
//
// Compute warps: four per quadrant, or two where P^T has remainders (with 112 registers a thread these spill: 16 groups, B = 1,
// N = 4096: 159 us against 148; 8 groups, B = 4: 242 against 248).  The next warp issues, three more only fill its warpgroup, whose
// registers the compute warps take: 640 threads x 96 at launch = 512 x 112 + 128 x 32, 384 x 168 = 256 x 232 + 128 x 40.
template <bool FINE>
struct KvWarps {
  static constexpr int SUBS = FINE ? 2 : 4, COMPUTE = 4 * SUBS, ISSUER = COMPUTE, THREADS = (COMPUTE + 4) * 32;
  static constexpr int REGS = FINE ? 232 : 112, REGS_REST = FINE ? 40 : 32;
};
// tensor memory: U (128; first dW^T of a head) | P^T (64), later W^T | their remainders (64) | Z (64) | dU (64) | two term
// slots (64).  Where P^T has no remainders their columns are a second Z until W^T is stored.
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
__global__ void __launch_bounds__(KvWarps<FINE>::THREADS, 1) intra_bwd_kv_kernel(const IntraBwdArgs a) {
  constexpr int SUBS = KvWarps<FINE>::SUBS;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Kimg = smem;
  unsigned char* Uimg = Kimg + ROW_IMAGE_BYTES;
  unsigned char* heads = Uimg + SLAB_S_BYTES;                   // two sets of a head's operands
  __shared__ __align__(16) HeadScalars sc[2];
  __shared__ uint64_t u_in, head_in[2], dw_full, ready, u_full, z_full, w_full, v_full;
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int part = blockIdx.z, c = blockIdx.x, b = blockIdx.y / a.Hkv, kvh = blockIdx.y - b * a.Hkv;
  const int h0 = part * a.heads_per_cta, n_heads = min(a.heads_per_cta, a.rep - h0), rank = a.rank;
  const int qd = warp & 3, row = 32 * qd + lane;     // row: key index inside the chunk
  const int tok0 = c * CT, nc = min(CT, a.N - tok0), cols = (nc + 31) & ~31;
  const auto head_of = [&](int i) { return kvh * a.rep + h0 + i; };
  if (warp == 0) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    mbar_init(&u_in, 1);
    mbar_init(&head_in[0], 1);
    mbar_init(&head_in[1], 1);
    mbar_init(&dw_full, 1);
    mbar_init(&ready, KvWarps<FINE>::COMPUTE);
    mbar_init(&u_full, 1);
    mbar_init(&z_full, 1);
    mbar_init(&w_full, KvWarps<FINE>::COMPUTE);
    mbar_init(&v_full, 1);
    mbar_fence_init();
    dead = 0;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);
  const uint32_t lane_off = (uint32_t)(32 * qd) << 16;
  // the last Z of a head is in its own columns: those of the remainders are free for W^T
  const auto z_at = [&](int r) { return tmem + (FINE || ((rank - 1 - r) & 1) == 0 ? BK_Z : BK_PLO); };

  if (warp >= KvWarps<FINE>::ISSUER) {
    registers_down_to<KvWarps<FINE>::REGS_REST>();
    if (warp == KvWarps<FINE>::ISSUER && elect_one()) {
      const uint32_t u_addr = smem_u32(Uimg);
      const size_t unit = ((size_t)b * a.Hkv + kvh) * a.NB + c;
      mbar_arrive_expect_tx(&u_in, ROW_IMAGE_BYTES + SLAB_S_BYTES);
      bulk_g2s(Kimg, a.k_image + unit * ROW_IMAGE_BYTES, ROW_IMAGE_BYTES, &u_in);
      bulk_g2s(Uimg, a.u_image + unit * SLAB_S_BYTES, SLAB_S_BYTES, &u_in);
      const auto fetch_head = [&](int i) {                  // rows of q, both images of G, l and scalars of head i
        unsigned char* dst = heads + (i & 1) * BK_HEAD_BYTES;
        const size_t at = ((size_t)b * a.Hq + head_of(i)) * a.NB + c;
        const HeadFactor* f = a.factors + head_of(i);
        uint64_t* bar = &head_in[i & 1];
        mbar_arrive_expect_tx(bar, ROW_IMAGE_BYTES + 2 * SLAB_S_BYTES + rank * HD * 4 + (int)sizeof(HeadScalars));
        bulk_g2s(dst, a.q_image + at * ROW_IMAGE_BYTES, ROW_IMAGE_BYTES, bar);
        bulk_g2s(dst + ROW_IMAGE_BYTES, a.gimg + at * SLAB_S_BYTES, SLAB_S_BYTES, bar);
        bulk_g2s(dst + ROW_IMAGE_BYTES + SLAB_S_BYTES, a.gimg + a.gimg_lo_offset + at * SLAB_S_BYTES, SLAB_S_BYTES, bar);
        bulk_g2s(dst + ROW_IMAGE_BYTES + 2 * SLAB_S_BYTES, &f->l[0][0], rank * HD * 4, bar);
        bulk_g2s(&sc[i & 1], &f->s, (int)sizeof(HeadScalars), bar);
      };
      const uint64_t du = smem_desc(u_addr, ROW_PLANE, 128);
      // dW^T[j, i] = [v|1]_j . g_i: rows from the U image, columns from the hi and lo images of G
      const auto head_dw = [&](int i) {
        const uint32_t g_addr = smem_u32(heads + (i & 1) * BK_HEAD_BYTES) + ROW_IMAGE_BYTES;
        w.wait(&head_in[i & 1], (i >> 1) & 1, 0x31);
        fence_after_sync();
        issue_dw(tmem + BK_U, du, du, 2 * ROW_PLANE, smem_desc(g_addr, ROW_PLANE, 128), smem_desc(g_addr + SLAB_S_BYTES, ROW_PLANE, 128),
                 2 * ROW_PLANE, cols);
        mma_commit(&dw_full);
      };
      fetch_head(0);
      if (n_heads > 1) fetch_head(1);
      w.wait(&u_in, 0, 0x32);
      head_dw(0);
      int T = 0, phase = 0;                                 // terms so far, over all heads; phases of `ready`
      for (int i = 0; i < n_heads; ++i) {
        const uint32_t q_addr = smem_u32(heads + (i & 1) * BK_HEAD_BYTES), g_addr = q_addr + ROW_IMAGE_BYTES;
        const uint64_t dq = smem_desc(q_addr, 128, ROW_PLANE), dg = smem_desc(g_addr, 128, ROW_PLANE);
        const uint64_t dg_lo = smem_desc(g_addr + SLAB_S_BYTES, 128, ROW_PLANE);
        for (int r = -1; r < rank; ++r) {
          w.wait(&ready, phase++ & 1, 0x33);
          fence_after_sync();
          if (r + 1 < rank) {
            issue_term<ROW_PLANE>(tmem + BK_U, tmem + BK_TERM + ((T + r + 1) & 1) * TERM_COLS, q_addr, cols);
            mma_commit(&u_full);
          }
          if (r < 0) continue;
          const uint32_t z = z_at(r);
          for (int part = 0; part < (FINE ? 2 : 1); ++part)
            for (int ks = 0; ks < cols / 16; ++ks)
              mma_bf16_ts(z, tmem + (part ? BK_PLO : BK_P) + 8 * ks, desc_advance(dq, ks * 256), instr_desc_bf16(128, HD, 0, 1), part + ks > 0);
          mma_commit(&z_full);
          if (r == 0 && i > 0 && i + 1 < n_heads) {
            // head i - 1 no longer reads the set that head i + 1 takes
            if (w.met(&v_full, (i - 1) & 1, 0x34)) fetch_head(i + 1);
          }
        }
        T += rank;
        if (i + 1 < n_heads) head_dw(i + 1);
        w.wait(&w_full, i & 1, 0x35);
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
  } else {
    registers_up_to<KvWarps<FINE>::REGS>();
    constexpr int BLOCKS = 8 / SUBS, DIMS = HD / SUBS, PIECES = DIMS / 8;     // 16 queries, dims and pieces of 8 dims per warp
    const int sub = warp >> 2, m = lane & 3, d0 = DIMS * sub;
    const unsigned char* xrow = Kimg + row * 16;
    // this warp's queries: blocks of 16, half of some 32s; blocks before the diagonal stay zero in P^T and W^T
    const auto block_of = [&](int x) { return x * (SUBS / 2) + (sub >> 1); };
    const auto col_of = [&](int x) { return 32 * block_of(x) + 16 * (sub & 1); };
    const auto exists = [&](int x) { return 32 * block_of(x) < cols; };
    const auto on = [&](int x) { return exists(x) && block_of(x) >= qd; };
    const uint32_t zero[8] = {};
#pragma unroll
    for (int x = 0; x < BLOCKS; ++x)
      if (exists(x) && !on(x)) {
        tmem_st8(tmem + BK_P + lane_off + col_of(x) / 2, zero);
        if (FINE) tmem_st8(tmem + BK_PLO + lane_off + col_of(x) / 2, zero);
      }
    // keys lane / 4 + 8 t, dims d0 + 8 j + 2 m, + 1: the arrangement in which Z is drained
    f32x2 dk[4][PIECES];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int j = 0; j < PIECES; ++j) dk[t][j] = 0ull;
    const auto load_rows_of = [&](uint32_t at, f32x2 (&v)[4][PIECES]) {
      float z[2][4 * PIECES];
      tmem_ld_rows(at + lane_off + d0, z[0]);
      tmem_ld_rows(at + lane_off + d0 + (16u << 16), z[1]);
      tmem_ld_wait();
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int j = 0; j < PIECES; ++j) v[t][j] = f2_pack(z[t >> 1][4 * j + 2 * (t & 1)], z[t >> 1][4 * j + 2 * (t & 1) + 1]);
    };
    w.wait(&u_in, 0, 0x36);
    int T = 0;
    for (int i = 0; i < n_heads; ++i) {
      const float* l = reinterpret_cast<const float*>(heads + (i & 1) * BK_HEAD_BYTES + ROW_IMAGE_BYTES + 2 * SLAB_S_BYTES);
      const HeadScalars& hs = sc[i & 1];
      w.wait(&head_in[i & 1], (i >> 1) & 1, 0x37);
      __syncwarp();
      const int rpos = uniform(hs.rpos);
      const auto build = [&](int r) {
        const uint32_t slot = tmem + BK_TERM + ((T + r) & 1) * TERM_COLS + lane_off;
#pragma unroll
        for (int d = 0; d < DIMS; d += 16) build_term16<ROW_PLANE>(slot, xrow, l + r * HD, d0 + d);
      };
      build(0);
      f32x2 dw[BLOCKS][8], wt[BLOCKS][8];
      const f32x2 w0 = f2_bcast(hs.w0);
      w.wait(&dw_full, i & 1, 0x38);
      __syncwarp();
      fence_after_sync();
#pragma unroll
      for (int x = 0; x < BLOCKS; ++x)
        if (on(x)) {
          float d[16];
          tmem_ld16(tmem + BK_U + lane_off + col_of(x), d);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int i0 = col_of(x) + 2 * j;                 // query not earlier than the key
            dw[x][j] = f2_pack(i0 >= row ? 2.f * d[2 * j] : 0.f, i0 + 1 >= row ? 2.f * d[2 * j + 1] : 0.f);
            wt[x][j] = w0;
          }
        }
      tmem_st_wait();
      fence_before_sync();
      warp_arrive(&ready, lane);
      const auto drain = [&](int r) {
        f32x2 z[4][PIECES], lv[PIECES];
        const f32x2 sgn = f2_bcast(r < rpos ? 1.f : -1.f);
#pragma unroll
        for (int j = 0; j < PIECES; ++j) lv[j] = f2_mul(*reinterpret_cast<const f32x2*>(l + r * HD + d0 + 2 * m + 8 * j), sgn);
        load_rows_of(z_at(r), z);
#pragma unroll
        for (int j = 0; j < PIECES; ++j)
#pragma unroll
          for (int t = 0; t < 4; ++t) dk[t][j] = f2_fma(lv[j], z[t][j], dk[t][j]);
      };
      for (int r = 0; r < rank; ++r) {
        // the next term's slot was last read for U of r - 1, which has arrived
        if (r + 1 < rank) build(r + 1);
        const f32x2 c2 = f2_bcast(hs.c[r]), sgn = f2_bcast(r < rpos ? 1.f : -1.f);
        w.wait(&u_full, (T + r) & 1, 0x39);
        __syncwarp();
        fence_after_sync();
        uint32_t p[BLOCKS / 2][8], rest[BLOCKS / 2][8];
        const auto products = [&](int x, int k) {
          float u[16];
          tmem_ld16(tmem + BK_U + lane_off + col_of(x), u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const f32x2 u2 = f2_add(f2_pack(u[2 * j], u[2 * j + 1]), c2);
            float t0, t1;
            f2_unpack(f2_mul(dw[x][j], u2), t0, t1);
            p[k][j] = pack_bf16(t0, t1);
            if (FINE) rest[k][j] = pack_bf16(t0 - bf16_lo(p[k][j]), t1 - bf16_hi(p[k][j]));
            wt[x][j] = f2_fma(rpos == rank ? u2 : f2_mul(u2, sgn), u2, wt[x][j]);
          }
        };
        const auto store = [&](int x, int k) {
          tmem_st8(tmem + BK_P + lane_off + col_of(x) / 2, p[k]);
          if (FINE) tmem_st8(tmem + BK_PLO + lane_off + col_of(x) / 2, rest[k]);
        };
#pragma unroll
        for (int x = 0; x < BLOCKS / 2; ++x)
          if (on(x)) products(x, x);
        // P^T of the previous term, or W^T of the previous head, has been read
        if (r > 0) w.wait(&z_full, (T + r - 1) & 1, 0x3A);
        else if (i > 0) w.wait(&v_full, (i - 1) & 1, 0x3B);
        __syncwarp();
        fence_after_sync();
#pragma unroll
        for (int x = 0; x < BLOCKS / 2; ++x)
          if (on(x)) store(x, x);
#pragma unroll
        for (int x = BLOCKS / 2; x < BLOCKS; ++x)
          if (on(x)) {
            products(x, x - BLOCKS / 2);
            store(x, x - BLOCKS / 2);
          }
        if (FINE && r > 0) drain(r - 1);
        tmem_st_wait();
        fence_before_sync();
        warp_arrive(&ready, lane);
        if (!FINE && r > 0) drain(r - 1);
      }
      w.wait(&z_full, (T + rank - 1) & 1, 0x3C);
      __syncwarp();
      fence_after_sync();
      drain(rank - 1);
      // W^T and its remainders in the place of P^T and its, or of the second Z, whose readers of this quadrant are done
      fence_before_sync();
      asm volatile("bar.sync %0, %1;" ::"r"(1 + qd), "n"(SUBS * 32) : "memory");
      fence_after_sync();
#pragma unroll
      for (int x = 0; x < BLOCKS; ++x)
        if (on(x)) {
          uint32_t o[8], rest[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float w_a, w_b;
            f2_unpack(wt[x][j], w_a, w_b);
            const int i0 = col_of(x) + 2 * j;
            if (i0 < row) w_a = 0.f;
            if (i0 + 1 < row) w_b = 0.f;
            o[j] = pack_bf16(w_a, w_b);
            rest[j] = pack_bf16(w_a - bf16_lo(o[j]), w_b - bf16_hi(o[j]));
          }
          tmem_st8(tmem + BK_P + lane_off + col_of(x) / 2, o);
          tmem_st8(tmem + BK_PLO + lane_off + col_of(x) / 2, rest);
        } else if (!FINE && exists(x)) {
          tmem_st8(tmem + BK_PLO + lane_off + col_of(x) / 2, zero);
        }
      tmem_st_wait();
      fence_before_sync();
      warp_arrive(&w_full, lane);
      T += rank;
    }
    const int rows = max(nc - 32 * qd, 0);                    // of the quadrant that exist
    const size_t tok = (size_t)tok0 + 32 * qd + (lane >> 2);
    const size_t out0 = (((size_t)b * a.Hkv + kvh) * a.N + tok) * HD + d0 + 2 * m;
    const size_t part0 = ((((size_t)b * a.Hkv + kvh) * a.parts + part) * a.N + tok) * HD + d0 + 2 * m;
    const auto write = [&](const f32x2 (&v)[4][PIECES], float* partial, const float* cross, __nv_bfloat16* out) {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if ((lane >> 2) + 8 * t >= rows) continue;
        const bool add = cross && (int)tok + 8 * t < a.cross_end;
#pragma unroll
        for (int j = 0; j < PIECES; ++j) {
          float x0, x1;
          f2_unpack(v[t][j], x0, x1);
          const size_t at = 8 * t * HD + 8 * j;
          if (partial) {
            *reinterpret_cast<float2*>(partial + part0 + at) = make_float2(x0, x1);
          } else if (out) {
            const float2 z = add ? *reinterpret_cast<const float2*>(cross + out0 + at) : make_float2(0.f, 0.f);
            *reinterpret_cast<uint32_t*>(out + out0 + at) = pack_bf16(x0 + z.x, x1 + z.y);
          }
        }
      }
    };
    if (!dead) write(dk, a.dk_part, a.dk_cross, a.dk);
    w.wait(&v_full, (n_heads - 1) & 1, 0x3D);
    __syncwarp();
    fence_after_sync();
    load_rows_of(tmem + BK_V, dk);
    if (!dead) write(dk, a.dv_part, a.dv_cross, a.dv);
  }
  fence_before_sync();
  __syncthreads();
  w.settle();
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
  const bool terms = coef_partial && NB == 1;
  cudaError_t e = terms ? allow_smem<intra_bwd_q_kernel<true>>(BQ_SMEM) : allow_smem<intra_bwd_q_kernel<false>>(BQ_SMEM);
  if (e != cudaSuccess) return e;
  IntraBwdArgs a = bwd_args(rows, gimg, factors, status, B, Hq, Hkv, N, NB, groups);
  a.scale = scale;
  a.dq = static_cast<__nv_bfloat16*>(dq); a.dq_init = dq_init; a.coef_partial = coef_partial; a.cross_from = cross_from;
  const dim3 grid(NB, B * Hkv, Hq / Hkv);
  if (terms) intra_bwd_q_kernel<true><<<grid, BQ_THREADS, BQ_SMEM, st>>>(a);
  else intra_bwd_q_kernel<false><<<grid, BQ_THREADS, BQ_SMEM, st>>>(a);
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
  if (fine) intra_bwd_kv_kernel<true><<<grid, KvWarps<true>::THREADS, BK_SMEM, st>>>(a);
  else intra_bwd_kv_kernel<false><<<grid, KvWarps<false>::THREADS, BK_SMEM, st>>>(a);
  if (a.parts == 1 || (e = cudaGetLastError()) != cudaSuccess) return cudaGetLastError();
  KvReduceArgs r{{dk_part, dv_part}, {dk_cross, dv_cross}, {static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv)},
                 B, Hkv, a.parts, N, cross_end};
  const size_t total = (size_t)B * Hkv * N * 16;
  kv_head_reduce_kernel<<<dim3((unsigned)((total + 255) / 256), 2), 256, 0, st>>>(r);
  return cudaGetLastError();
}

}  // namespace oal
