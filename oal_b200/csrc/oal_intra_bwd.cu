// Intra-chunk term of the chunked scan on the tensor cores (tcgen05 / TMEM), backward.
//
// Both kernels walk the terms r of the factored weight (oal_intra.cuh).  The scaled rows are carried as bf16
// value + bf16 remainder, two MMA chains into u_r: the coefficient gradient is a sum of strongly cancelling terms
// (sum_j dW_ij w_ij = 0 for every row) and needs u to more than 8 bits, and on the key side the rounding of the
// scaled keys would act like a perturbation that is the same for every query.
//
// Query side (rows are query rows, columns are keys), dW = G [v|1]^T once (G as hi + lo bf16), then per term:
//   P_r = 2 dW u_r             registers -> tensor memory, bf16 value + remainder
//   Z_r = P_r K                one accumulator per term;  n_r = sum of P_r, registers
//   dq  += sgn_r l_r * Z_r     registers (element-wise in the dimension)
//   y_r  = sum over rows of q * Z_r, one 64-vector per row block
// The coefficient gradient needs D'[r][r'] = sum_ij 2 dW u_r u_r' = sum_d l_r'[d] y_r[d] + c_r' n_r: 64 sums per
// term instead of R (R + 1) / 2 products per pair.  P_r's remainder keeps these sums at the 16 bits they had when
// they were formed from fp32 products.
//
// Key / value side (rows are keys, columns are the queries of one head): per head and term
//   P_r^T as above (bf16 value; with its remainder above 8 groups),  Z_r = P_r^T Q,  dk += sgn_r l_r * Z_r,  w += sgn_r u_r^2 in registers,
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
  const __nv_bfloat16 *q, *k, *v;
  const __nv_bfloat16* gimg;        // [2][B*Hq, NB, 10, 128, 8]: bf16(g) image, then the image of g - bf16(g)
  size_t gimg_lo_offset;            // bytes from the hi image to the lo image
  const HeadFactor* factors;
  __nv_bfloat16* dq;                // may be null
  const float* dq_init;             // fp32 cross part, or null
  float* coef_partial;              // [B][Hq][row blocks][NQ] or null: D upper triangle, n_r, sum 2 dW
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

// hi / lo bf16 pairs of eight products
__device__ __forceinline__ void split8(const f32x2 (&t)[4], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a, b;
    f2_unpack(t[j], a, b);
    hi[j] = pack_bf16(a, b);
    lo[j] = pack_bf16(a - bf16_lo(hi[j]), b - bf16_hi(hi[j]));
  }
}

// ---------------------------------------------------------------------------
// query side
// ---------------------------------------------------------------------------
// tensor memory: U (two halves of 64; first dW) | P hi (64) | P lo (64) | two Z (64) | two term slots (64)
constexpr uint32_t BQ_U = 0, BQ_P = 128, BQ_PLO = 192, BQ_Z = 256, BQ_TERM = 384;
static_assert(BQ_TERM + 2 * TERM_COLS <= 512, "tensor-memory columns of the query-side kernel");
constexpr int BQ_L_FLOATS = 4 * RMAX_ALL * HD;
constexpr int BQ_SMEM = 2 * X_BYTES + 3 * XA_BYTES + BQ_L_FLOATS * 4;
static_assert(BQ_L_FLOATS * 4 <= XA_BYTES, "the y sums take the place of an image of G");

__global__ void __launch_bounds__(BW_THREADS, 1) intra_bwd_q_kernel(const IntraBwdArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Qimg = smem;
  unsigned char* Kimg = Qimg + X_BYTES;
  unsigned char* Uimg = Kimg + X_BYTES;
  unsigned char* Gimg = Uimg + XA_BYTES;                        // hi, lo; dead once dW is complete
  float* lq = reinterpret_cast<float*>(Gimg + 2 * XA_BYTES);    // [quadrant][term][64]
  float* ys = reinterpret_cast<float*>(Gimg);                   // [quadrant][term][64]
  __shared__ __align__(16) HeadScalars sc[4];
  __shared__ float nq[BW_COMPUTE][RMAX_ALL], sq[BW_COMPUTE];
  __shared__ uint64_t dw_full, dw_free, u_full[2], u_free[2], term_full[2], p_full[2], z_half[2], z_free[2];
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const QueryTile tile(a.Hkv, a.N, a.rep);
  if (tile.empty()) return;
  const int qd = warp & 3, sub = (warp >> 2) & 3, row = 32 * qd + lane;
  const int tok0 = tile.c * CT, cols = tile.columns(), rank = a.rank;
  const int my_rb = tile.rb(qd), my_head = tile.head(qd);
  {
    const size_t koff = ((size_t)tile.b * a.Hkv + tile.kvh) * a.N + tok0;
    const size_t qoff = ((size_t)tile.b * a.Hq + my_head) * a.N + tok0 + min(32 * my_rb, tile.nc - 1);
    const int fifth = (warp >> 2) * 32 + lane;                  // five warps load a quadrant's rows and table
    const unsigned char* gsrc = reinterpret_cast<const unsigned char*>(a.gimg) +
                                (((size_t)tile.b * a.Hq + my_head) * a.NB + tile.c) * SLAB_S_BYTES + 32 * my_rb * 16;
    for (int x = fifth; x < 2 * (EP / 8) * 32; x += 160) {
      const int r = x & 31, e = (x >> 5) % (EP / 8), lo = x >= (EP / 8) * 32;
      async_copy16(Gimg + lo * XA_BYTES + e * CP + (32 * qd + r) * 16, gsrc + lo * a.gimg_lo_offset + e * (CT * 16) + r * 16, true);
    }
    load_rows(Uimg, 0, a.v + koff * VD, cols, tile.nc, tid, BW_THREADS);
    load_rows(Qimg, 32 * qd, a.q + qoff * HD, 32, max(tile.nc - 32 * my_rb, 0), fifth, 160);
    load_rows(Kimg, 0, a.k + koff * HD, cols, tile.nc, tid, BW_THREADS);
    load_head(lq + qd * RMAX_ALL * HD, &sc[qd], a.factors + my_head, rank, fifth, 160);
  }
  augment_rows(Uimg, tile.nc, tid, BW_THREADS);
  if (warp == 0) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&u_full[s], 1);
      mbar_init(&u_free[s], BW_COMPUTE);
      mbar_init(&term_full[s], BW_COMPUTE);
      mbar_init(&p_full[s], BW_COMPUTE);
      mbar_init(&z_half[s], 1);
      mbar_init(&z_free[s], BW_COMPUTE);
    }
    mbar_init(&dw_full, 1);
    mbar_init(&dw_free, BW_COMPUTE);
    mbar_fence_init();
    dead = 0;
  }
  async_copies_wait();
  fence_async_smem();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);
  const uint32_t lane_off = (uint32_t)(32 * qd) << 16;
  const int na = min(cols, 64), nb2 = cols - na;              // columns of the two halves
  const bool want_coef = a.coef_partial != nullptr;

  if (warp >= BW_ISSUER) {
    registers_down_to<24>();
    if (warp == BW_ISSUER) {
      const uint32_t k_addr = smem_u32(Kimg), g_addr = smem_u32(Gimg), u_addr = smem_u32(Uimg);
      if (elect_one()) {
        const uint64_t du = smem_desc(u_addr, CP, 128), dk = smem_desc(k_addr, 128, CP);
        issue_dw(tmem + BQ_U, smem_desc(g_addr, CP, 128), smem_desc(g_addr + XA_BYTES, CP, 128), 2 * CP, du, du, 2 * CP, cols);
        mma_commit(&dw_full);
        // half hf of the keys of Z_r = (P hi + P lo) K
        const auto issue_z = [&](int r, int hf) {
          w.wait(&p_full[hf], r & 1, 0x21);
          if (hf == 0 && r >= 2) w.wait(&z_free[r & 1], ((r >> 1) - 1) & 1, 0x22);
          fence_after_sync();
          const uint32_t z = tmem + BQ_Z + (r & 1) * HD, idesc = instr_desc_bf16(128, HD, 0, 1);
          const int k0 = hf ? 4 : 0, k1 = hf ? 4 + nb2 / 16 : na / 16;
          for (int ks = k0; ks < k1; ++ks) {
            mma_bf16_ts(z, tmem + BQ_P + 8 * ks, desc_advance(dk, ks * 256), idesc, ks > 0);
            mma_bf16_ts(z, tmem + BQ_PLO + 8 * ks, desc_advance(dk, ks * 256), idesc, 1);
          }
          mma_commit(&z_half[hf]);
        };
        for (int r = 0; r < rank; ++r) {
          const uint32_t slot = tmem + BQ_TERM + (r & 1) * TERM_COLS;
          w.wait(&term_full[r & 1], (r >> 1) & 1, 0x23);
          if (r > 0) w.wait(&u_free[0], (r - 1) & 1, 0x24);
          else w.wait(&dw_free, 0, 0x25);
          fence_after_sync();
          issue_term(tmem + BQ_U, slot, k_addr, na);
          mma_commit(&u_full[0]);
          if (r > 0) {
            issue_z(r - 1, 0);
            w.wait(&u_free[1], (r - 1) & 1, 0x26);
          }
          if (nb2) {
            fence_after_sync();
            issue_term(tmem + BQ_U + 64, slot, k_addr + 64 * 16, nb2);
          }
          mma_commit(&u_full[1]);            // also: the term's slot has been read
          if (r > 0) issue_z(r - 1, 1);
        }
        issue_z(rank - 1, 0);
        issue_z(rank - 1, 1);
      }
      __syncwarp();
    }
  } else {
    registers_up_to<112>();
    const unsigned char* xrow = Qimg + row * 16;
    const float* l = lq + qd * RMAX_ALL * HD;
    const int rpos = uniform(sc[qd].rpos);
    const int last_key = 32 * my_rb + 31, my_key = 32 * my_rb + lane;
    const int d0 = 16 * sub;
    const auto build = [&](int r) {
      build_term16(tmem + BQ_TERM + (r & 1) * TERM_COLS + lane_off, xrow, l + r * HD, d0);
      tmem_st_wait();
      fence_before_sync();
      warp_arrive(&term_full[r & 1], lane);
    };
    build(0);
    // this warp's keys: a quarter of each half, in blocks of 8; blocks behind the diagonal stay zero in P
    const auto key_of = [&](int hf, int x) { return 64 * hf + sub * ((hf ? nb2 : na) / 4) + 8 * x; };
    const auto exists = [&](int hf, int x) { return 32 * x < (hf ? nb2 : na); };
    const auto on = [&](int hf, int x) { return exists(hf, x) && key_of(hf, x) <= last_key; };
    f32x2 dw[2][2][4];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (exists(hf, x) && !on(hf, x)) {
          tmem_st4(tmem + BQ_P + lane_off + key_of(hf, x) / 2, 0u, 0u, 0u, 0u);
          tmem_st4(tmem + BQ_PLO + lane_off + key_of(hf, x) / 2, 0u, 0u, 0u, 0u);
        }
    w.wait(&dw_full, 0, 0x27);
    fence_after_sync();
    f32x2 sum2 = 0ull;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (on(hf, x)) {
          float d[8];
          tmem_ld8(tmem + BQ_U + lane_off + key_of(hf, x), d);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int kj = key_of(hf, x) + 2 * j;
            dw[hf][x][j] = f2_pack(kj <= my_key ? 2.f * d[2 * j] : 0.f, kj + 1 <= my_key ? 2.f * d[2 * j + 1] : 0.f);
            sum2 = f2_add(sum2, dw[hf][x][j]);
          }
        }
    fence_before_sync();
    warp_arrive(&dw_free, lane);
    f32x2 dq[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) dq[j] = 0ull;
    // Z of term r: dq, and the sums over the 32 rows of q * Z (one warp holds all rows of its block)
    const auto drain = [&](int r) {
      float z[16];
      tmem_ld16(tmem + BQ_Z + (r & 1) * HD + lane_off + d0, z);
      tmem_ld_wait();
      fence_before_sync();
      warp_arrive(&z_free[r & 1], lane);
      const f32x2 sgn = f2_bcast(r < rpos ? 1.f : -1.f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const ulonglong2 lv = *reinterpret_cast<const ulonglong2*>(l + r * HD + d0 + 4 * j);
        dq[2 * j] = f2_fma(f2_mul(lv.x, sgn), f2_pack(z[4 * j], z[4 * j + 1]), dq[2 * j]);
        dq[2 * j + 1] = f2_fma(f2_mul(lv.y, sgn), f2_pack(z[4 * j + 2], z[4 * j + 3]), dq[2 * j + 1]);
      }
      if (!want_coef) return;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint4 raw = *reinterpret_cast<const uint4*>(xrow + (d0 / 8 + k) * CP);
        const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          z[8 * k + 2 * j] *= bf16_lo(rw[j]);
          z[8 * k + 2 * j + 1] *= bf16_hi(rw[j]);
        }
      }
      // butterfly that halves the values it carries: 16 shuffles for 16 sums over 32 lanes
#pragma unroll
      for (int o = 16; o >= 2; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < o / 2; ++j) {
          const float send = up ? z[j] : z[j + o / 2], keep = up ? z[j + o / 2] : z[j];
          z[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      z[0] += __shfl_xor_sync(0xffffffffu, z[0], 1);
      if ((lane & 1) == 0) ys[(qd * RMAX_ALL + r) * HD + d0 + (lane >> 1)] = z[0];
    };
    for (int r = 0; r < rank; ++r) {
      // the next term is built while the MMAs of this one run; its slot's last reader was term r - 1, complete
      // since u_full[1](r - 1)
      if (r + 1 < rank) build(r + 1);
      const f32x2 c2 = f2_bcast(sc[qd].c[r]);
      f32x2 n2 = 0ull;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        w.wait(&u_full[hf], r & 1, 0x28 + hf);
        fence_after_sync();
        float u[2][8];
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (on(hf, x)) tmem_ld8(tmem + BQ_U + lane_off + key_of(hf, x), u[x]);
        tmem_ld_wait();
        fence_before_sync();
        warp_arrive(&u_free[hf], lane);
        uint32_t hi[2][4], lo[2][4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (on(hf, x)) {
            f32x2 t[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              t[j] = f2_mul(dw[hf][x][j], f2_add(f2_pack(u[x][2 * j], u[x][2 * j + 1]), c2));
              n2 = f2_add(n2, t[j]);
            }
            split8(t, hi[x], lo[x]);
          }
        if (r > 0) {                           // the previous term's P has been read
          w.wait(&z_half[hf], (r - 1) & 1, 0x2A + hf);
          fence_after_sync();
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (on(hf, x)) {
            tmem_st4(tmem + BQ_P + lane_off + key_of(hf, x) / 2, hi[x][0], hi[x][1], hi[x][2], hi[x][3]);
            tmem_st4(tmem + BQ_PLO + lane_off + key_of(hf, x) / 2, lo[x][0], lo[x][1], lo[x][2], lo[x][3]);
          }
        tmem_st_wait();
        fence_before_sync();
        warp_arrive(&p_full[hf], lane);
      }
      if (r > 0) drain(r - 1);
      if (want_coef) {
        float n, n1;
        f2_unpack(n2, n, n1);
        n += n1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
        if (lane == 0) nq[warp][r] = n;
      }
    }
    w.wait(&z_half[0], (rank - 1) & 1, 0x2C);
    w.wait(&z_half[1], (rank - 1) & 1, 0x2D);
    fence_after_sync();
    drain(rank - 1);
    if (want_coef) {
      float s0, s1;
      f2_unpack(sum2, s0, s1);
      s0 += s1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      if (lane == 0) sq[warp] = s0;
    }
    if (a.dq && my_key < tile.nc && !dead) {
      // 16 consecutive dims of a row per thread: whole 32- and 64-byte sectors
      const size_t o = (((size_t)tile.b * a.Hq + my_head) * a.N + tok0 + my_key) * HD + d0;
      float v[16];
#pragma unroll
      for (int j = 0; j < 8; ++j) f2_unpack(dq[j], v[2 * j], v[2 * j + 1]);
      if (a.dq_init && tile.c >= a.cross_from) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 t = *reinterpret_cast<const float4*>(a.dq_init + o + 4 * j);
          v[4 * j] += t.x; v[4 * j + 1] += t.y; v[4 * j + 2] += t.z; v[4 * j + 3] += t.w;
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
        *reinterpret_cast<uint4*>(a.dq + o + 8 * j) =
            make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                       pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
    }
    if (want_coef) {
      // the quadrant's four warps turn its sums into D' (symmetrised: both orders are the same sum), n', s'
      asm volatile("bar.sync %0, 128;" ::"r"(1 + qd) : "memory");
      const auto n_of = [&](int r) { return (nq[qd][r] + nq[4 + qd][r]) + (nq[8 + qd][r] + nq[12 + qd][r]); };
      const int nu = rank * (rank + 1) / 2, stride = nu + rank + 1, blocks = (a.N + 31) / 32;
      float* dst = a.coef_partial + (((size_t)tile.b * a.Hq + my_head) * blocks + tile.c * 4 + my_rb) * stride;
      const float* y = ys + qd * RMAX_ALL * HD;
      for (int x = sub * 32 + lane; x < stride && 32 * my_rb < tile.nc; x += 128) {
        float t;
        if (x < nu) {
          int r = 0, rest = x;
          while (rest >= rank - r) { rest -= rank - r; ++r; }
          const int r2 = r + rest;
          t = fmaf(sc[qd].c[r2], n_of(r), sc[qd].c[r] * n_of(r2));
#pragma unroll 4
          for (int d = 0; d < HD; d += 4) {
            const float4 la = *reinterpret_cast<const float4*>(l + r * HD + d), lb = *reinterpret_cast<const float4*>(l + r2 * HD + d);
            const float4 ya = *reinterpret_cast<const float4*>(y + r * HD + d), yb = *reinterpret_cast<const float4*>(y + r2 * HD + d);
            t = fmaf(lb.x, ya.x, fmaf(lb.y, ya.y, fmaf(lb.z, ya.z, fmaf(lb.w, ya.w, t))));
            t = fmaf(la.x, yb.x, fmaf(la.y, yb.y, fmaf(la.z, yb.z, fmaf(la.w, yb.w, t))));
          }
          t *= 0.5f;
        } else if (x < nu + rank) {
          t = n_of(x - nu);
        } else {
          t = (sq[qd] + sq[4 + qd]) + (sq[8 + qd] + sq[12 + qd]);
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
constexpr int BK_HEAD_BYTES = X_BYTES + 2 * SLAB_S_BYTES + BK_HEAD_L;       // Q image, G hi, G lo, l: one head's operands
constexpr int BK_SMEM = X_BYTES + XA_BYTES + 2 * BK_HEAD_BYTES;
static_assert(BK_HEAD_BYTES % 16 == 0 && BK_SMEM <= 227 * 1024, "shared memory of the key/value-side kernel");

// FINE: P^T with its remainders and W^T against both images of G, for heads of more than 8 groups.  Their weights were
// formed and summed in fp32 (oal_pairs.cu) before these kernels took them over, and the bf16 values alone were up to 1.24
// times as far from 64 bits in dv and 1.18 times in dk (14 / 2 heads, N = 347, 16 groups: 2.13e-3 -> 2.64e-3 and 2.14e-3 ->
// 2.52e-3); up to 8 groups the bf16 values are nearer than the tiles that they replaced (dk 3.3e-3 -> 2.8e-3).
template <bool FINE>
__global__ void __launch_bounds__(BW_THREADS, 1) intra_bwd_kv_kernel(const IntraBwdArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Kimg = smem;
  unsigned char* Uimg = Kimg + X_BYTES;
  unsigned char* heads = Uimg + XA_BYTES;                       // two sets of a head's operands
  __shared__ __align__(16) HeadScalars sc[2];
  __shared__ uint64_t q_full[2], g_full[2], dw_full, dw_free, u_full[2], u_free[2], term_full[2], p_full[2], z_half[2], z_free, w_full, v_full;
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int part = blockIdx.z, c = blockIdx.x, b = blockIdx.y / a.Hkv, kvh = blockIdx.y - b * a.Hkv;
  const int h0 = part * a.heads_per_cta, n_heads = min(a.heads_per_cta, a.rep - h0), rank = a.rank;
  const int qd = warp & 3, sub = (warp >> 2) & 3, row = 32 * qd + lane;     // row: key index inside the chunk
  const int tok0 = c * CT, nc = min(CT, a.N - tok0), cols = (nc + 31) & ~31;
  const size_t koff = ((size_t)b * a.Hkv + kvh) * a.N + tok0;
  const auto head_of = [&](int i) { return kvh * a.rep + h0 + i; };
  // Q image, l and scalars of head i: asynchronous copies by threads tid of n
  const auto fetch_q = [&](int i, int n) {
    unsigned char* set = heads + (i & 1) * BK_HEAD_BYTES;
    load_rows(set, 0, a.q + (((size_t)b * a.Hq + head_of(i)) * a.N + tok0) * HD, cols, nc, tid, n);
    load_head(reinterpret_cast<float*>(set + X_BYTES + 2 * SLAB_S_BYTES), &sc[i & 1], a.factors + head_of(i), rank, tid, n);
  };
  load_rows(Kimg, 0, a.k + koff * HD, CT, nc, tid, BW_THREADS);
  load_rows(Uimg, 0, a.v + koff * VD, CT, nc, tid, BW_THREADS);
  if (warp < BW_COMPUTE) fetch_q(0, BW_COMPUTE * 32);
  augment_rows(Uimg, nc, tid, BW_THREADS);
  if (warp == 0) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], BW_COMPUTE);
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
    mbar_fence_init();
    dead = 0;
  }
  async_copies_wait();
  fence_async_smem();
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
        const auto fetch_g = [&](int i) {                     // both G images of head i (bulk copies)
          unsigned char* dst = heads + (i & 1) * BK_HEAD_BYTES + X_BYTES;
          const unsigned char* src = reinterpret_cast<const unsigned char*>(a.gimg) + (((size_t)b * a.Hq + head_of(i)) * a.NB + c) * SLAB_S_BYTES;
          mbar_arrive_expect_tx(&g_full[i & 1], 2 * SLAB_S_BYTES);
          bulk_g2s(dst, src, SLAB_S_BYTES, &g_full[i & 1]);
          bulk_g2s(dst + SLAB_S_BYTES, src + a.gimg_lo_offset, SLAB_S_BYTES, &g_full[i & 1]);
        };
        fetch_g(0);
        int T = 0;                                            // terms issued so far, over all heads
        for (int i = 0; i < n_heads; ++i) {
          const uint32_t q_addr = smem_u32(heads + (i & 1) * BK_HEAD_BYTES), g_addr = q_addr + X_BYTES;
          if (i + 1 < n_heads) {
            if (i > 0) w.wait(&v_full, (i - 1) & 1, 0x30);    // head i - 1 no longer reads the set that head i + 1 takes
            fetch_g(i + 1);
          }
          w.wait(&g_full[i & 1], (i >> 1) & 1, 0x31);
          w.wait(&q_full[i & 1], (i >> 1) & 1, 0x32);
          if (T > 0) {
            w.wait(&u_free[0], (T - 1) & 1, 0x33);
            w.wait(&u_free[1], (T - 1) & 1, 0x34);
          }
          fence_after_sync();
          // dW^T[j, i] = [v|1]_j . g_i: rows from the U image, columns from the hi and lo images of G
          const uint64_t du = smem_desc(u_addr, CP, 128);
          issue_dw(tmem + BK_U, du, du, 2 * CP, smem_desc(g_addr, CT * 16, 128), smem_desc(g_addr + SLAB_S_BYTES, CT * 16, 128),
                   2 * CT * 16, cols);
          mma_commit(&dw_full);
          const uint64_t dq = smem_desc(q_addr, 128, CP), dg = smem_desc(g_addr, 128, CT * 16);
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
            issue_term(tmem + BK_U, slot, q_addr, na);
            mma_commit(&u_full[0]);
            if (r > 0) {
              issue_z(T - 1, 0);
              w.wait(&u_free[1], (T - 1) & 1, 0x3A);
            }
            if (nb2) {
              fence_after_sync();
              issue_term(tmem + BK_U + 64, slot, q_addr + 64 * 16, nb2);
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
    f32x2 dk[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) dk[j] = 0ull;
    int T = 0;
    for (int i = 0; i < n_heads; ++i) {
      const float* l = reinterpret_cast<const float*>(heads + (i & 1) * BK_HEAD_BYTES + X_BYTES + 2 * SLAB_S_BYTES);
      const HeadScalars& hs = sc[i & 1];
      async_copies_wait();
      fence_async_smem();
      warp_arrive(&q_full[i & 1], lane);
      // every warp reads l and the scalars below: all copies have arrived
      w.wait(&q_full[i & 1], (i >> 1) & 1, 0x3C);
      if (i > 0) w.wait(&v_full, (i - 1) & 1, 0x3D);          // W^T of the previous head has been read; so has its operand set
      if (i + 1 < n_heads) fetch_q(i + 1, BW_COMPUTE * 32);
      const int rpos = uniform(hs.rpos);
      const auto build = [&](int r) {
        build_term16(tmem + BK_TERM + ((T + r) & 1) * TERM_COLS + lane_off, xrow, l + r * HD, d0);
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

IntraBwdArgs bwd_args(const void* q, const void* k, const void* v, const void* gimg, const void* factors,
                      int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups) {
  IntraBwdArgs a{};
  a.q = static_cast<const __nv_bfloat16*>(q); a.k = static_cast<const __nv_bfloat16*>(k);
  a.v = static_cast<const __nv_bfloat16*>(v); a.gimg = static_cast<const __nv_bfloat16*>(gimg);
  a.factors = static_cast<const HeadFactor*>(factors);
  a.status = status;
  a.N = N; a.NB = NB; a.Hq = Hq; a.Hkv = Hkv; a.rep = Hq / Hkv; a.rank = groups + 1;
  a.gimg_lo_offset = (size_t)B * Hq * NB * SLAB_S_BYTES;
  return a;
}

}  // namespace

int intra_row_blocks(int N) { return (N + 31) / 32; }

cudaError_t intra_backward_q(const void* q, const void* k, const void* v, const void* gimg,
                             const void* factors, void* dq, const float* dq_init, float* coef_partial,
                             int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups, int cross_from,
                             cudaStream_t st) {
  cudaError_t e = allow_smem<intra_bwd_q_kernel>(BQ_SMEM);
  if (e != cudaSuccess) return e;
  IntraBwdArgs a = bwd_args(q, k, v, gimg, factors, status, B, Hq, Hkv, N, NB, groups);
  a.dq = static_cast<__nv_bfloat16*>(dq); a.dq_init = dq_init; a.coef_partial = coef_partial; a.cross_from = cross_from;
  intra_bwd_q_kernel<<<dim3(NB, B * Hkv, Hq / Hkv), BW_THREADS, BQ_SMEM, st>>>(a);
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

cudaError_t intra_backward_kv(const void* q, const void* k, const void* v, const void* gimg, const void* factors,
                              void* dk, void* dv, const float* dk_cross, const float* dv_cross, int cross_end, float* dk_part,
                              float* dv_part, int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups,
                              cudaStream_t st) {
  const bool fine = groups > 8;
  cudaError_t e = fine ? allow_smem<intra_bwd_kv_kernel<true>>(BK_SMEM) : allow_smem<intra_bwd_kv_kernel<false>>(BK_SMEM);
  if (e != cudaSuccess) return e;
  IntraBwdArgs a = bwd_args(q, k, v, gimg, factors, status, B, Hq, Hkv, N, NB, groups);
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
