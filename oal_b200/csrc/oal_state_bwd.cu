// Backward of the inter-chunk state path on the tensor cores (tcgen05 / TMEM).
//
//   dstate_heads : Z_h[u,c] = phi_raw(q_h)^T G_h per query head (raw = coefficient-free features),
//                  dCarry[u,c] = sum_h diag(coef_h) Z_h accumulated in tensor memory, and the
//                  per-feature coefficient gradient  dcoef_h[f] += sum_e carry[u,c][f,e] Z_h[f,e]
//                  (reference: oal_attention/hd_block_gemm_backward.py:764-877 dCarry with GQA sum;
//                  coefficient partial sums oal_attention/hd_block_gemm_feature_backward.py:134-474)
//   feature_grad : dphi[i, f] = A_i . state[f, :]  with A = G (query side, state = carry) or
//                  A = [v | 1] (key side, state = reverse-scanned dCarry), folded on the fly through
//                  the feature map into dq / dk
//                  (reference: hd_block_gemm_backward_wave.py:335-342 and hd_block_gemm_backward.py:911-964
//                  contractions, hd_block_gemm_feature_backward.py:59-131,157-422 folds)
// The reverse scan and the key-side phi_k . dT contraction reuse state_scan / cross_read.
#include "oal_features.cuh"
#include "oal_kernels.h"

namespace oal {
namespace {

using namespace umma;

__device__ __forceinline__ void unpack_bf16x8(const uint4 t, float (&o)[8]) {
  const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[j]);
    o[2 * j] = __low2float(h);
    o[2 * j + 1] = __high2float(h);
  }
}

// ---------------------------------------------------------------------------
// dstate_heads
// ---------------------------------------------------------------------------
struct DStateArgs {
  const unsigned char* q_image;    // [B*Hq, NB, 8, 128, 8]
  const __nv_bfloat16* gimg;       // [B*Hq, NB, 10, 128, 8]
  const __nv_bfloat16* carry_img;  // [units, NB, 19, 10, 128, 8] or null (no coefficient gradients)
  const __nv_bfloat16* carry_lo;   // same layout: bf16(state - bf16(state)); the dot products below see hi + lo,
                                   // because they are sums of strongly cancelling terms
  const float* coef_table;         // [Hq, F_ROWS]
  float* dcarry;                   // [units, NB] chunks of F_ROWS x EP floats in state_inc_offset order
  float* dcoef_partial;            // [B, NC, 2 column halves, Hq, F_ROWS] or null
  int NB, Hq, Hkv, units;
  int c0, NC;                      // chunks [c0, c0 + NC) of each sequence (no one reads dCarry of the others)
  float scale;
  int32_t* status;
};

// Persistent, warp-specialised kernel.  Work items are (batch x KV head, chunk, feature slab); CTA k
// takes items k, k + gridDim.x, ... and walks the query heads of the KV head for each, so the flat
// iteration `it` = (item, head) drives four pipelined roles:
//   warps 0-7   thread = (token, half of the slab): generate the coefficient-free, unscaled feature slab of (item, head)
//               from the q rows into A[it % 3]
//   warp  17    lane 0 streams the head's G image and coefficients into slot it % 3 of a ring and, an item ahead, the
//               slab's carry and remainder images (bulk copies)
//   warp  16    lane 0 issues the MMAs  Z[it % 3] = A^T G  once A and G are there and Z[it % 3] is drained
//   warps 8-15  drain Z, thread = (feature row, part of the used columns): dot with the carry row for
//               the coefficient gradient, acc += coef_h * Z in registers; after the last head
//               acc -> dCarry
// A, G and Z share the index it % 3 and one barrier per direction: `ready` counts the generator and drain warps and the
// loader, and the MMA-completion barrier tells the generators "A is free", the loader "G is free" and the drain warps
// "Z is ready".  (Every wait and every commit costs the issuing thread 50 to 100 clocks.)
constexpr int DS_GEN_WARPS = 8, DS_EPI_WARPS = 8;
constexpr int DS_ISSUER = DS_GEN_WARPS + DS_EPI_WARPS, DS_LOADER = DS_ISSUER + 1;
// What bounds it: the drain (about 1400 clocks per iteration) and the generators, latency rather than issue slots.  The carry
// rows were loaded by the drain warps at the head of an item, 5000 of its 15000 clocks.  14 / 2 heads, B = 4, N = 4096:
// 268 -> 188 us (221 with the pieces of q from the rows themselves).
// Two warps more only fill the issuer's warpgroup, whose registers the drain warps take: 640 threads x 96 at launch =
// 256 x 80 + 256 x 144 + 128 x 24 and 1024 to spare.
constexpr int DS_THREADS = (DS_LOADER + 3) * 32;
constexpr int DS_RING = 3;      // A and G slots in shared memory, Z buffers in tensor memory
// shared memory: A slots | G slots (the MMA reads 8 columns past the used ones: in bounds, into columns of Z that no one
// reads) | carry and its remainders | coefficients.  A coefficient slot is written again six iterations later,
// behind mma_done of the third one after its own: the drain warps had read it before they let that MMA have Z.
constexpr int DS_G = DS_RING * SLAB_A_BYTES, DS_CARRY = DS_G + DS_RING * SLAB_U_BYTES;
constexpr int DS_COEF = DS_CARRY + 2 * SLAB_U_BYTES, DS_CRING = 2 * DS_RING;
constexpr int DS_SMEM = DS_COEF + DS_CRING * 128 * 4;
constexpr int DS_COLS = EP / 2; // columns per drain thread; the second half has EU - DS_COLS used ones
static_assert(DS_GEN_WARPS * 32 == 2 * CT, "a generator thread per token and half of a slab");
static_assert(DS_GEN_WARPS % 4 == 0, "drain warp w must sit on tensor-memory lane quadrant w % 4");

// (item, head) cursor of one role; the divisions happen only when the item changes
struct DsCursor {
  int u, c, slab, hh, item;
  int b, h0;          // batch row and first query head of the item's KV head
  __device__ __forceinline__ void set_item(int it_item, int c0, int NC, int Hkv, int rep) {
    item = it_item;
    slab = item % F_SLABS;
    const int r = item / F_SLABS;
    c = c0 + r % NC;
    u = r / NC;
    b = u / Hkv;
    h0 = (u - b * Hkv) * rep;
  }
  __device__ __forceinline__ void start(int c0, int NC, int Hkv, int rep) {
    hh = 0;
    set_item(blockIdx.x, c0, NC, Hkv, rep);
  }
  __device__ __forceinline__ void next(int rep, int c0, int NC, int Hkv) {
    if (++hh == rep) {
      hh = 0;
      set_item(item + gridDim.x, c0, NC, Hkv, rep);
    }
  }
};

__global__ void __launch_bounds__(DS_THREADS, 1) dstate_heads_kernel(const DStateArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Abuf = smem;                              // DS_RING x SLAB_A_BYTES
  unsigned char* Gbuf = smem + DS_G;
  __shared__ uint64_t ready[DS_RING], mma_done[DS_RING], carry_full, carry_free;
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int rep = a.Hq / a.Hkv;
  const int n_items = F_SLABS * a.NC * a.units;
  const int my_items = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  const int T = my_items * rep;
  if (warp == DS_ISSUER) tmem_alloc(&tmem_base, 256);
  if (tid == 0) {
    for (int s = 0; s < DS_RING; ++s) {
      mbar_init(&ready[s], DS_GEN_WARPS + DS_EPI_WARPS + 1);
      mbar_init(&mma_done[s], 1);
    }
    mbar_init(&carry_full, 1);
    mbar_init(&carry_free, DS_EPI_WARPS);
    mbar_fence_init();
    dead = 0;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);

  if (warp < DS_GEN_WARPS) {
    // ---------------- generators ----------------
    registers_down_to<80>();
    // The two pieces of its token's row that a thread needs for (item, head) come from the row image, an iteration ahead.
    // (From the rows themselves: 32 cache lines per load, 1000 clocks.  Through shared memory with cp.async: as long.)
    const int half = warp >> 2, token = 32 * (warp & 3) + lane;
    DsCursor cur;
    cur.start(a.c0, a.NC, a.Hkv, rep);
    const uint4* row = nullptr;                // the token's pieces, ROW_PLANE apart
    uint4 r4 = make_uint4(0u, 0u, 0u, 0u), c4 = r4;
    const auto fetch = [&]() {
      const HalfBlock blk = half_block(min(2 * cur.slab + half, F_PAIR_BLOCKS - 1));
      row = reinterpret_cast<const uint4*>(a.q_image + ((size_t)(cur.b * a.Hq + cur.h0 + cur.hh) * a.NB + cur.c) * ROW_IMAGE_BYTES) + token;
      r4 = load_ahead(row + blk.rb * CT);
      c4 = load_ahead(row + blk.cb * CT);
    };
    if (T > 0) fetch();
    int s = 0, use = 0;                       // ring slot of `it` and how often it has been used before
    for (int it = 0; it < T; ++it) {
      const int hs = 2 * cur.slab + half;
      const uint4 r_now = r4, c_now = c4;
      const uint4* row_now = row;
      cur.next(rep, a.c0, a.NC, a.Hkv);
      if (it + 1 < T) fetch();
      if (use > 0) w.wait(&mma_done[s], (use - 1) & 1, 0x31);   // the MMA that read A[s] has completed
      uint4* tile = reinterpret_cast<uint4*>(Abuf + s * SLAB_A_BYTES) + 8 * half * CT + token;
      raw_half_slab(hs, r_now, c_now, [&](int j) { return __ldg(row_now + j * CT); },
                    [&](int j, uint4 f) { tile[j * CT] = f; });
      fence_async_smem();
      warp_arrive(&ready[s], lane);
      if (++s == DS_RING) { s = 0; ++use; }
    }
  } else if (warp < DS_ISSUER) {
    // ---------------- drain warps ----------------
    registers_up_to<144>();
    const int fr = 32 * (warp & 3) + lane, ch = (warp - DS_GEN_WARPS) >> 2, col0 = ch * DS_COLS;
    const uint32_t lane_off = (uint32_t)(32 * (warp & 3)) << 16;
    // packed fp32 pairs: the drain is bound by issue slots, and a packed multiply-add is one slot for two columns
    f32x2 acc[DS_COLS / 2];        // this thread's part of the dCarry row, summed over the heads of the item
    f32x2 carry[DS_COLS / 2];      // this thread's part of the carry row (value + remainder), fp32, once per item
#pragma unroll
    for (int j = 0; j < DS_COLS / 2; ++j) carry[j] = 0ull;
    DsCursor d, dn;
    d.start(a.c0, a.NC, a.Hkv, rep);
    dn = d;
    int s = 0, use = 0;
    const int blocks = ch == 0 ? DS_COLS / 8 : (EU - DS_COLS) / 8;      // of 8 used columns
    if (lane == 0)
      for (int x = 0; x < DS_RING; ++x) mbar_arrive(&ready[x]);         // the Z buffers are empty
    int items = 0;
    for (int it = 0; it < T; ++it) {
      const int b = d.b, h = d.h0 + d.hh, f = d.slab * 128 + fr;
      const float fs = feature_scale_factor(f, a.scale);   // d(table entry) / d(coefficient)
      dn.next(rep, a.c0, a.NC, a.Hkv);
      if (d.hh == 0 && a.carry_img) {
        const uint4* cp = reinterpret_cast<const uint4*>(smem + DS_CARRY);
        const uint4* cl = reinterpret_cast<const uint4*>(smem + DS_CARRY + SLAB_U_BYTES);
        w.wait(&carry_full, items & 1, 0x37);
        ++items;
        uint4 cpk[DS_COLS / 8], cpl[DS_COLS / 8];
#pragma unroll
        for (int e = 0; e < DS_COLS / 8; ++e) {
          cpk[e] = cpl[e] = make_uint4(0u, 0u, 0u, 0u);
          if (e >= blocks) continue;
          cpk[e] = cp[(col0 / 8 + e) * 128 + fr];
          cpl[e] = cl[(col0 / 8 + e) * 128 + fr];
        }
#pragma unroll
        for (int e = 0; e < DS_COLS / 8; ++e) {
          float c0[8], c1[8];
          unpack_bf16x8(cpk[e], c0);
          unpack_bf16x8(cpl[e], c1);
#pragma unroll
          for (int j = 0; j < 4; ++j) carry[4 * e + j] = f2_pack(c0[2 * j] + c1[2 * j], c0[2 * j + 1] + c1[2 * j + 1]);
        }
        warp_arrive(&carry_free, lane);
      }
      w.wait(&mma_done[s], use & 1, 0x32);
      fence_after_sync();
      const uint32_t tz = tmem + EP * s + col0;
      if (d.hh == 0) {
#pragma unroll
        for (int j = 0; j < DS_COLS / 2; ++j) acc[j] = 0ull;
      }
      f32x2 dot[2] = {0ull, 0ull};
      const f32x2 cf2 = f2_bcast(reinterpret_cast<const float*>(smem + DS_COEF)[it % DS_CRING * 128 + fr]);
      // two register stages: the loads of the next 8 columns are in flight while these are combined
      float z[2][8];
      tmem_ld8(tz + lane_off, z[0]);
#pragma unroll
      for (int r = 0; r < DS_COLS / 8; ++r) {
        if (r >= blocks) continue;
        tmem_ld_wait();
        if (r + 1 < blocks) tmem_ld8(tz + lane_off + 8 * (r + 1), z[(r + 1) & 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 z2 = f2_pack(z[r & 1][2 * j], z[r & 1][2 * j + 1]);
          dot[j & 1] = f2_fma(z2, carry[4 * r + j], dot[j & 1]);
          acc[4 * r + j] = f2_fma(cf2, z2, acc[4 * r + j]);
        }
      }
      fence_before_sync();
      warp_arrive(&ready[s], lane);                // every lane has its Z values in registers
      float d0, d1, d2, d3;
      f2_unpack(dot[0], d0, d1);
      f2_unpack(dot[1], d2, d3);
      const float dot_sum = (d0 + d2) + (d1 + d3);
      if (a.dcoef_partial)      // one partial per column half, summed by the reduction over (batch, chunk, half)
        a.dcoef_partial[((((size_t)b * a.NC + d.c - a.c0) * 2 + ch) * a.Hq + h) * F_ROWS + f] =
            fs * dot_sum;
      if (d.hh == rep - 1) {
        // dCarry rows of this slab -> HBM; the next group of 8 columns of a row lies one 128-row block further
        float* dst = a.dcarry + ((size_t)d.u * a.NB + d.c) * F_ROWS * EP + state_inc_offset(f, col0);
#pragma unroll
        for (int r = 0; r < DS_COLS / 8; ++r) {
          if (r >= blocks) continue;
          float o[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) f2_unpack(acc[4 * r + j], o[2 * j], o[2 * j + 1]);
          *reinterpret_cast<float4*>(dst + r * 1024) = make_float4(o[0], o[1], o[2], o[3]);
          *reinterpret_cast<float4*>(dst + r * 1024 + 4) = make_float4(o[4], o[5], o[6], o[7]);
        }
      }
      d = dn;
      if (++s == DS_RING) { s = 0; ++use; }
    }
  } else {
    registers_down_to<24>();
    if (warp == DS_ISSUER && elect_one()) {
      // ---------------- MMA issue ----------------
      const uint32_t idesc = instr_desc_bf16(128, EP, 1, 1);
      // descriptors of slot 0 of both rings, advanced by adds: this thread is the serial path of every slab
      const uint64_t da0 = smem_desc(smem_u32(Abuf), 128, CT * 16), dg0 = smem_desc(smem_u32(Gbuf), 128, CT * 16);
      int s = 0, use = 0;
      for (int it = 0; it < T; ++it) {
        const uint64_t da = desc_advance(da0, s * SLAB_A_BYTES), dg = desc_advance(dg0, s * SLAB_U_BYTES);
        const uint32_t tz = tmem + EP * s;
        w.wait(&ready[s], use & 1, 0x33);
        fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < CT / 16; ++ks)
          mma_bf16_ss(tz, desc_advance(da, ks * 256), desc_advance(dg, ks * 256), idesc, ks > 0);
        mma_commit(&mma_done[s]);
        if (++s == DS_RING) { s = 0; ++use; }
      }
    }
    if (warp == DS_LOADER && elect_one()) {
      // ---------------- G image, carry and coefficient stream ----------------
      DsCursor d;
      d.start(a.c0, a.NC, a.Hkv, rep);
      int s = 0, use = 0, fetched = 0;
      const auto fetch_carry = [&](const DsCursor& x) {
        const size_t at = (((size_t)x.u * a.NB + x.c) * F_SLABS + x.slab) * SLAB_S_BYTES;
        if (fetched > 0 && !w.met(&carry_free, (fetched - 1) & 1, 0x38)) return;      // in registers of the drain warps
        ++fetched;
        mbar_arrive_expect_tx(&carry_full, 2 * SLAB_U_BYTES);
        bulk_g2s(smem + DS_CARRY, reinterpret_cast<const unsigned char*>(a.carry_img) + at, SLAB_U_BYTES, &carry_full);
        bulk_g2s(smem + DS_CARRY + SLAB_U_BYTES, reinterpret_cast<const unsigned char*>(a.carry_lo) + at, SLAB_U_BYTES, &carry_full);
      };
      if (T > 0 && a.carry_img) fetch_carry(d);
      for (int it = 0; it < T; ++it) {
        const int h = d.h0 + d.hh;
        const unsigned char* src =
            reinterpret_cast<const unsigned char*>(a.gimg) + ((size_t)(d.b * a.Hq + h) * a.NB + d.c) * SLAB_S_BYTES;
        if (use > 0 && !w.met(&mma_done[s], (use - 1) & 1, 0x36)) break;
        mbar_arrive_expect_tx(&ready[s], SLAB_U_BYTES + 128 * 4);
        bulk_g2s(Gbuf + s * SLAB_U_BYTES, src, SLAB_U_BYTES, &ready[s]);
        bulk_g2s(smem + DS_COEF + it % DS_CRING * 128 * 4, a.coef_table + (size_t)h * F_ROWS + d.slab * 128, 128 * 4, &ready[s]);
        const bool last = d.hh == rep - 1;
        d.next(rep, a.c0, a.NC, a.Hkv);
        if (last && it + 1 < T && a.carry_img) fetch_carry(d);
        if (++s == DS_RING) { s = 0; ++use; }
      }
    }
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  w.settle();
  if (warp == DS_ISSUER) tmem_dealloc(tmem_base, 256);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
}

// ---------------------------------------------------------------------------
// fold of dphi (tensor memory, thread = token, columns = the features of a half slab) through the feature map into dx.
// Per block of x x^T, with t = dphi (* coef):
//   dx[r] += sum_c t[r][c] x[c]        dx[c] += sum_r t[r][c] x[r]
// dx lies in shared memory (fp32, this thread's token); the sums of the column block stay in registers while it does
// not change.  Entries above the diagonal of a diagonal block add zeros: their coefficients are zero, and so are the rows
// of dCarry that belong to them.
// ---------------------------------------------------------------------------
struct FoldColumns {
  int cb;                        // column block, < 0: none yet
  f32x2 x[4], dx[4];
};

__device__ __forceinline__ void fold_add8(unsigned char* dx_token, int block, const f32x2 (&v)[4]) {
  ulonglong2* p0 = reinterpret_cast<ulonglong2*>(dx_token + 2 * block * CP);
  ulonglong2* p1 = reinterpret_cast<ulonglong2*>(dx_token + (2 * block + 1) * CP);
  ulonglong2 a = *p0, b = *p1;
  a.x = f2_add(a.x, v[0]); a.y = f2_add(a.y, v[1]);
  b.x = f2_add(b.x, v[2]); b.y = f2_add(b.y, v[3]);
  *p0 = a;
  *p1 = b;
}

// `taddr`: the half slab's 64 columns at this warp's lanes; `loaded` runs once every lane has its values in registers.
template <bool QUERY, class Loaded>
__device__ __forceinline__ void fold_half_slab(int hs, uint32_t taddr, const unsigned char* xrow, const float* coef,
                                               unsigned char* dx_token, FoldColumns& col, Loaded loaded) {
  if (hs == HALF_CONST) {                // the constant has no gradient
    loaded();
    return;
  }
  const float* cf = coef + F_BLOCK * hs;
  float va[2][16];
  tmem_ld16(taddr, va[0]);
  // 16 columns: a pair of columns of the block and its eight rows
  const auto products = [&](int i, f32x2 (&t)[8]) {
#pragma unroll
    for (int r = 0; r < 8; ++r) t[r] = f2_pack(va[i & 1][2 * r], va[i & 1][2 * r + 1]);
    if constexpr (QUERY) {
#pragma unroll
      for (int r = 0; r < 8; r += 2) {
        const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(cf + 16 * i + 2 * r);
        t[r] = f2_mul(t[r], c.x);
        t[r + 1] = f2_mul(t[r + 1], c.y);
      }
    }
  };
  if (hs == HALF_LINEAR) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      tmem_ld_wait();
      if (i < 3) tmem_ld16(taddr + 16 * (i + 1), va[(i + 1) & 1]);
      else loaded();
      f32x2 t[8];
      products(i, t);
      const f32x2 lo[4] = {t[0], t[1], t[2], t[3]}, hi[4] = {t[4], t[5], t[6], t[7]};
      fold_add8(dx_token, 2 * i, lo);
      fold_add8(dx_token, 2 * i + 1, hi);
    }
    return;
  }
  const HalfBlock blk = half_block(hs);
  if (blk.cb != col.cb) {
    if (col.cb >= 0) fold_add8(dx_token, col.cb, col.dx);
    col.cb = blk.cb;
    const uint4 c4 = *reinterpret_cast<const uint4*>(xrow + blk.cb * ROW_PLANE);
    const uint32_t cw[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      col.x[k] = f2_pack(bf16_lo(cw[k]), bf16_hi(cw[k]));
      col.dx[k] = 0ull;
    }
  }
  const uint4 r4 = *reinterpret_cast<const uint4*>(xrow + blk.rb * ROW_PLANE);
  const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w};
  f32x2 xr[8], sum[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) xr[j] = f2_bcast((j & 1) ? bf16_hi(rw[j / 2]) : bf16_lo(rw[j / 2]));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    tmem_ld_wait();
    if (i < 3) tmem_ld16(taddr + 16 * (i + 1), va[(i + 1) & 1]);
    else loaded();
    f32x2 t[8];
    products(i, t);
    f32x2 other = f2_mul(t[7], xr[7]);         // two chains
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      sum[r] = i ? f2_fma(t[r], col.x[i], sum[r]) : f2_mul(t[r], col.x[i]);
      if (r & 1) { if (r < 7) other = f2_fma(t[r], xr[r], other); }
      else col.dx[i] = f2_fma(t[r], xr[r], col.dx[i]);
    }
    col.dx[i] = f2_add(col.dx[i], other);
  }
  f32x2 rows[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float a0, a1, b0, b1;
    f2_unpack(sum[2 * k], a0, a1);
    f2_unpack(sum[2 * k + 1], b0, b1);
    rows[k] = f2_pack(a0 + a1, b0 + b1);
  }
  fold_add8(dx_token, blk.rb, rows);
}

// ---------------------------------------------------------------------------
// feature_grad: persistent, warp-specialised.  Work items are (batch, head, chunk) with the heads of
// one state unit adjacent; CTA k takes items k, k + gridDim.x, ...  Roles:
//   warps 0-7  fold: thread = (token, half of the slab's 128 features); drains dphi of slab `s` from
//              tensor memory (four buffers) into its dx row in shared memory; halves are combined per item
//   warp  8    lane 0 issues  dphi[s] = A . S[s]^T  (M = tokens, N = 128 features, K = 80)
//   warp  9    lane 0 streams the state slab images (four slots) and, per item, the A operand
//              image (G, or [v | 1] for keys) and, for queries, the head's coefficient table (two buffers each)
// A state slot and a dphi buffer share their index and one barrier per direction (see cross_read_kernel).
// What bounds it: the fold's instruction latency (two warps per scheduler, 1500 clocks per slab; the MMAs are four slabs
// ahead).  14 / 2 heads, B = 4, N = 4096: 187 -> 164 us (QUERY), 38 -> 29 (not).
// ---------------------------------------------------------------------------
struct FeatGradArgs {
  const unsigned char* x_image;  // rows of q (QUERY) or k  [B*H, NB, 8, 128, 8]
  const unsigned char* a_image;  // A operand: image of G (QUERY) or [v | 1]  [B*H, NB, 10, 128, 8]
  const __nv_bfloat16* image;    // state image [units, NB, 19, 10, 128, 8]: carry (QUERY) / dT (KEY)
  const float* coef_table;       // QUERY
  float* dx;                     // [B,H,N,64] fp32
  int N, NB, H, rep, B;
  int c0, NC;                    // chunks [c0, c0 + NC) of each sequence (the others meet a zero state)
  int32_t* status;
};

constexpr int FG_FOLD_WARPS = 8, FG_ISSUER = FG_FOLD_WARPS, FG_LOADER = FG_ISSUER + 1;
constexpr int FG_THREADS = (FG_LOADER + 1) * 32;
constexpr int FG_RING = 4;

struct FgItem {
  int b, h, c;
};
__device__ __forceinline__ FgItem fg_item(int item, int H, int rep, int NC, int c0) {
  FgItem r;
  const int hh = item % rep, t = item / rep;
  r.c = c0 + t % NC;
  const int unit = t / NC, units_per_b = H / rep;
  r.b = unit / units_per_b;
  r.h = (unit % units_per_b) * rep + hh;
  return r;
}

template <bool QUERY>
__global__ void __launch_bounds__(FG_THREADS, 1) feature_grad_kernel(const FeatGradArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Sbuf = smem;                                        // FG_RING x SLAB_S_BYTES
  unsigned char* Aimg = Sbuf + FG_RING * SLAB_S_BYTES;              // 2 x SLAB_S_BYTES: [10][128 tokens][8 e]
  float* coef_s = reinterpret_cast<float*>(Aimg + 2 * SLAB_S_BYTES); // 2 x F_ROWS
  unsigned char* ximg = reinterpret_cast<unsigned char*>(coef_s + 2 * F_ROWS);     // rows of x
  unsigned char* dx_s = ximg + ROW_IMAGE_BYTES;                              // per half: [16][128 tokens][4] fp32, plane pitch CP
  __shared__ uint64_t ready[FG_RING], done[FG_RING], a_full[2], a_free[2], coef_full[2], coef_free[2];
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int n_items = a.B * a.H * a.NC;
  const int my_items = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  if (warp == FG_ISSUER) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    for (int s = 0; s < FG_RING; ++s) {
      mbar_init(&ready[s], FG_FOLD_WARPS + 1);
      mbar_init(&done[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&a_free[s], 1);
      mbar_init(&coef_full[s], 1);
      mbar_init(&coef_free[s], FG_FOLD_WARPS);
    }
    mbar_fence_init();
    dead = 0;
  }
  // the last block of columns is not copied: zeros for both operands
  for (int x = tid; x < (FG_RING + 2) * CT; x += FG_THREADS)
    *reinterpret_cast<uint4*>(Sbuf + (x / CT) * SLAB_S_BYTES + SLAB_U_BYTES + (x % CT) * 16) = make_uint4(0u, 0u, 0u, 0u);
  fence_async_smem();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);

  if (warp < FG_FOLD_WARPS) {
    // ---------------- fold warps ----------------
    constexpr int T = FG_FOLD_WARPS * 32, PIECES = CT * 8 / T;
    const int half = warp >> 2, token = 32 * (warp & 3) + lane;
    const uint32_t lane_off = (uint32_t)(32 * (warp & 3)) << 16;
    const unsigned char* xrow = ximg + token * 16;
    unsigned char* dx_token = dx_s + half * 16 * CP + token * 16;
    uint4 next[PIECES];                                   // this thread's share of the next item's rows
    const auto fetch = [&](int k) {
      const FgItem it = fg_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
      const uint4* src = reinterpret_cast<const uint4*>(a.x_image + ((size_t)(it.b * a.H + it.h) * a.NB + it.c) * ROW_IMAGE_BYTES);
#pragma unroll
      for (int j = 0; j < PIECES; ++j) next[j] = load_ahead(src + tid + j * T);
    };
    const auto store_rows = [&]() {
#pragma unroll
      for (int j = 0; j < PIECES; ++j) reinterpret_cast<uint4*>(ximg)[tid + j * T] = next[j];
    };
    if (my_items > 0) fetch(0);
    store_rows();
    for (int x = tid; x < 2 * 16 * CP / 16; x += T) reinterpret_cast<uint4*>(dx_s)[x] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
    if (lane == 0)
      for (int x = 0; x < FG_RING; ++x) mbar_arrive(&ready[x]);         // the dphi buffers are empty
    int ds = 0, duse = 0;
    for (int k = 0; k < my_items; ++k) {
      const FgItem it = fg_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
      const size_t head_off = (size_t)(it.b * a.H + it.h) * a.N;
      if (k + 1 < my_items) fetch(k + 1);
      const float* coef = coef_s + (k & 1) * F_ROWS;
      if (QUERY) w.wait(&coef_full[k & 1], (k >> 1) & 1, 0x52);
      FoldColumns col;
      col.cb = -1;
      for (int s = 0; s < F_SLABS; ++s) {
        w.wait(&done[ds], duse & 1, 0x53);
        __syncwarp();
        fence_after_sync();
        fold_half_slab<QUERY>(2 * s + half, tmem + ds * 128 + 64 * half + lane_off, xrow, coef, dx_token, col, [&]() {
          fence_before_sync();
          warp_arrive(&ready[ds], lane);
        });
        if (++ds == FG_RING) { ds = 0; ++duse; }
      }
      if (QUERY) warp_arrive(&coef_free[k & 1], lane);
      fold_add8(dx_token, col.cb, col.dx);
      asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
      // the halves of every token together, whole rows per warp, and zeros for the next item
      store_rows();
#pragma unroll
      for (int j = 0; j < 2 * PIECES; ++j) {
        const int x = tid + j * T, row = x >> 4;
        float4* p = reinterpret_cast<float4*>(dx_s + (x & 15) * CP + row * 16);
        float4* p2 = reinterpret_cast<float4*>(dx_s + (16 + (x & 15)) * CP + row * 16);
        const float4 u = *p, v = *p2;
        *p = *p2 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (it.c * CT + row < a.N && !dead)
          *reinterpret_cast<float4*>(a.dx + (head_off + it.c * CT) * HD + 4 * x) = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
    }
  } else if (warp == FG_ISSUER) {
    // ---------------- MMA issue ----------------
    if (elect_one()) {
      const uint32_t idesc = instr_desc_bf16(128, 128, 0, 0);
      const uint64_t da0 = smem_desc(smem_u32(Aimg), CT * 16, 128), ds0 = smem_desc(smem_u32(Sbuf), 128 * 16, 128);
      int s4 = 0, use = 0;
      for (int k = 0; k < my_items; ++k) {
        const uint64_t da = desc_advance(da0, (k & 1) * SLAB_S_BYTES);
        w.wait(&a_full[k & 1], (k >> 1) & 1, 0x54);
        for (int s = 0; s < F_SLABS; ++s) {
          const uint64_t dsl = desc_advance(ds0, s4 * SLAB_S_BYTES);
          w.wait(&ready[s4], use & 1, 0x55);
          fence_after_sync();
#pragma unroll
          for (int ks = 0; ks < EP / 16; ++ks)
            mma_bf16_ss(tmem + s4 * 128, desc_advance(da, ks * 2 * CT * 16), desc_advance(dsl, ks * 2 * 128 * 16), idesc,
                        ks > 0);
          mma_commit(&done[s4]);
          if (++s4 == FG_RING) { s4 = 0; ++use; }
        }
        mma_commit(&a_free[k & 1]);
      }
    }
    __syncwarp();
  } else {
    // ---------------- image / table stream ----------------
    if (elect_one()) {
      int s4 = 0, use = 0;
      const auto fetch_item = [&](int k) {
        const FgItem it = fg_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
        if (k >= 2) {
          if (!w.met(&a_free[k & 1], ((k >> 1) - 1) & 1, 0x57)) return;
          if (QUERY && !w.met(&coef_free[k & 1], ((k >> 1) - 1) & 1, 0x58)) return;
        }
        mbar_arrive_expect_tx(&a_full[k & 1], SLAB_U_BYTES);
        bulk_g2s(Aimg + (k & 1) * SLAB_S_BYTES, a.a_image + ((size_t)(it.b * a.H + it.h) * a.NB + it.c) * SLAB_S_BYTES, SLAB_U_BYTES,
                 &a_full[k & 1]);
        if (!QUERY) return;
        mbar_arrive_expect_tx(&coef_full[k & 1], F_ROWS * (uint32_t)sizeof(float));
        bulk_g2s(coef_s + (k & 1) * F_ROWS, a.coef_table + (size_t)it.h * F_ROWS, F_ROWS * (uint32_t)sizeof(float),
                 &coef_full[k & 1]);
      };
      if (my_items > 0) fetch_item(0);
      for (int k = 0; k < my_items && !w.gave_up(); ++k) {
        const FgItem it = fg_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
        const int unit = (it.b * a.H + it.h) / a.rep;
        const unsigned char* img = reinterpret_cast<const unsigned char*>(a.image) +
                                   ((size_t)unit * a.NB + it.c) * F_SLABS * SLAB_S_BYTES;
        for (int s = 0; s < F_SLABS; ++s) {
          // the next item's operand and table while there is time: their buffers' last reader was item k-1
          if (s == 2 * F_SLABS / 3 && k + 1 < my_items) fetch_item(k + 1);
          if (use > 0 && !w.met(&done[s4], (use - 1) & 1, 0x59)) break;
          mbar_arrive_expect_tx(&ready[s4], SLAB_U_BYTES);
          bulk_g2s(Sbuf + s4 * SLAB_S_BYTES, img + (size_t)s * SLAB_S_BYTES, SLAB_U_BYTES, &ready[s4]);
          if (++s4 == FG_RING) { s4 = 0; ++use; }
        }
      }
    }
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  w.settle();
  if (warp == FG_ISSUER) tmem_dealloc(tmem_base, 512);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
}

// ---------------------------------------------------------------------------
// coefficient gradients of the cross-chunk term: per-feature sums -> (A, B_g, C_gg') slots
// ---------------------------------------------------------------------------
// block = 32 feature rows x 8 segments of the outer index; the segments are added in fixed order
__global__ void __launch_bounds__(256) dcoef_sum_kernel(const float* partial, int outer /* B*NC*2 */, int Hq,
                                                        float* dcoef) {
  __shared__ float seg_sum[8][32];
  const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
  const int f = blockIdx.x * 32 + lane, h = blockIdx.y;
  const int per = (outer + 7) / 8, o0 = seg * per, o1 = min(outer, o0 + per);
  float t = 0.f;
#pragma unroll 4
  for (int o = o0; o < o1; ++o) t += partial[((size_t)o * Hq + h) * F_ROWS + f];
  seg_sum[seg][lane] = t;
  __syncthreads();
  if (seg == 0) {
    float r = 0.f;
#pragma unroll
    for (int x = 0; x < 8; ++x) r += seg_sum[x][lane];
    dcoef[(size_t)h * F_ROWS + f] = r;
  }
}

__device__ __forceinline__ int tri_slot(int g, int g2) { return g * GMAX - (g * (g - 1)) / 2 + (g2 - g); }

// One block per head.  A warp walks all features once per coefficient slot, so the sums need no atomics and
// their order is fixed: lane partial sums over features lane, lane + 32, ..., then the butterfly.
constexpr int SLOT_WARPS = 32;
__global__ void __launch_bounds__(32 * SLOT_WARPS) dcoef_slots_kernel(const float* dcoef, const int32_t* dim_perm,
                                                                      const int32_t* group_start, int G,
                                                                      float* slots /* [Hq][NCOEF] */) {
  __shared__ int gdim[HD];
  __shared__ short fslot[F_ROWS];
  __shared__ float fval[F_ROWS];
  const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < HD) {
    const int p = threadIdx.x;
    int g = 0;
    while (g < GMAX - 1 && p >= group_start[h * (GMAX + 1) + g + 1]) ++g;
    gdim[dim_perm[h * HD + p]] = g;
  }
  __syncthreads();
  for (int f = threadIdx.x; f < F_ROWS; f += blockDim.x) {
    int slot = -1;
    float wgt = 0.f;
    const FeatureId id = feature_id(f);
    if (id.kind == 0 && id.live) {
      const int ga = min(gdim[id.r], gdim[id.c]), gb = max(gdim[id.r], gdim[id.c]);
      slot = 1 + GMAX + tri_slot(ga, gb);
      wgt = (ga == gb && id.r != id.c) ? 2.f : 1.f;
    } else if (id.kind == 1) {
      slot = 1 + gdim[id.r];
      wgt = 1.f;
    } else if (id.kind == 2) {
      slot = 0;
      wgt = 1.f;
    }
    fslot[f] = (short)slot;
    fval[f] = slot >= 0 ? wgt * dcoef[(size_t)h * F_ROWS + f] : 0.f;
  }
  __syncthreads();
  const int live = 1 + G + G * (G + 1) / 2;      // slots that groups 0 .. G-1 can reach, in (A, B, C rows) order
  for (int x = warp; x < live; x += SLOT_WARPS) {
    int s = x;
    if (x > G) {
      int g = 0, rest = x - 1 - G;
      while (rest >= G - g) { rest -= G - g; ++g; }
      s = 1 + GMAX + tri_slot(g, g + rest);
    }
    float t = 0.f;
#pragma unroll 4
    for (int f = lane; f < F_ROWS; f += 32) t += fslot[f] == s ? fval[f] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) slots[(size_t)h * NCOEF + s] = t;
  }
}

// normalisation VJP writing the bf16 operand images of G (hi, lo), and the image of the rows of q that the backward
// kernels fetch with bulk copies (copied by threads, 16 bytes each with cp.async, a tile's rows took 5000 clocks)
//   CTA = 32 consecutive tokens of one (head, chunk); warp = 8 consecutive columns, lane = token, so a
//   warp stores 512 contiguous bytes of an image chunk.  Rows are enumerated over padded chunks so
//   that tail tokens of the last chunk are zeroed.
__global__ void __launch_bounds__(256) norm_vjp_image_kernel(const void* grad_out, int out_dt, const float* grad_num,
                                                             const float* grad_den, const float* num,
                                                             const float* den, float floor_v, __nv_bfloat16* gimg, int N, int NB, int heads,
                                                             int tm_heads, const RowImages img_rows, int32_t* status) {
  __shared__ float part[8][32];
  if (status && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;     // first kernel of the backward
  const int ec = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t per_head = (size_t)NB * CT;
  const size_t r = (size_t)blockIdx.x * 32 + lane;          // grid covers heads * per_head rows exactly
  const size_t bh = r / per_head;
  const int t = (int)(r % per_head);
  const int cidx = t / CT, tl = t % CT;
  const bool live = t < N;
  const size_t row = bh * N + t;
  // row of the upstream gradient of out: head-first [B, Hq, N, 64], or token-major [B, N, Hq, 64] (tm_heads = Hq)
  const size_t grow = tm_heads > 0 ? ((bh / tm_heads) * N + t) * tm_heads + bh % tm_heads : row;
  float gv[8], dot = 0.f, dn = 1.f, dw = 1.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) gv[j] = 0.f;
  if (live) {
    dn = den[row];
    dw = fmaxf(dn, floor_v);
    if (grad_out) {
      float go[8];
      if (out_dt == OAL_DTYPE_BF16) {
        const uint4 w = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(grad_out) + grow * VD + 8 * ec);
        unpack_bf16x8(w, go);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) go[j] = load_elem(grad_out, grow * VD + 8 * ec + j, out_dt);
      }
      const float4 n0 = *reinterpret_cast<const float4*>(num + row * VD + 8 * ec);
      const float4 n1 = *reinterpret_cast<const float4*>(num + row * VD + 8 * ec + 4);
      const float nn[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        dot = fmaf(go[j], nn[j], dot);
        gv[j] = go[j] / dw;
      }
    }
    if (grad_num) {
      const float4 a0 = *reinterpret_cast<const float4*>(grad_num + row * VD + 8 * ec);
      const float4 a1 = *reinterpret_cast<const float4*>(grad_num + row * VD + 8 * ec + 4);
      gv[0] += a0.x; gv[1] += a0.y; gv[2] += a0.z; gv[3] += a0.w;
      gv[4] += a1.x; gv[5] += a1.y; gv[6] += a1.z; gv[7] += a1.w;
    }
  }
  part[ec][lane] = dot;
  reinterpret_cast<uint4*>(static_cast<unsigned char*>(img_rows.q_image) + (bh * NB + cidx) * ROW_IMAGE_BYTES)[ec * CT + tl] =
      live ? *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(img_rows.q) + row * HD + 8 * ec) : make_uint4(0u, 0u, 0u, 0u);
  // hi image = bf16(g); lo image = bf16(g - hi): dW = g . [v|1] is formed from both, because its two
  // large terms (dout.v / den and dout.num / den^2) nearly cancel
  uint4* img = reinterpret_cast<uint4*>(gimg + (bh * NB + cidx) * (size_t)(SLAB_S_BYTES / 2));
  uint4* img_lo = reinterpret_cast<uint4*>(gimg + ((size_t)heads * NB + bh * NB + cidx) * (size_t)(SLAB_S_BYTES / 2));
  {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __nv_bfloat16 h0 = __float2bfloat16_rn(gv[2 * k]), h1 = __float2bfloat16_rn(gv[2 * k + 1]);
      hi[k] = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
      lo[k] = pack_bf16(gv[2 * k] - __bfloat162float(h0), gv[2 * k + 1] - __bfloat162float(h1));
    }
    img[ec * CT + tl] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    img_lo[ec * CT + tl] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
  __syncthreads();
  if (ec < 2) {            // columns 64..79: [d den, 0 x 15]
    float gd = 0.f;
    if (ec == 0 && live) {
      float d = 0.f;
#pragma unroll
      for (int x = 0; x < 8; ++x) d += part[x][lane];
      if (grad_out) gd = (dn >= floor_v) ? -(d / dw) / dw : 0.f;
      if (grad_den) gd += grad_den[row];
    }
    const __nv_bfloat16 h0 = __float2bfloat16_rn(gd);
    img[(VD / 8 + ec) * CT + tl] = make_uint4((uint32_t)__bfloat16_as_ushort(h0), 0u, 0u, 0u);
    img_lo[(VD / 8 + ec) * CT + tl] = make_uint4(pack_bf16(gd - __bfloat162float(h0), 0.f), 0u, 0u, 0u);
  }
}

}  // namespace

cudaError_t dstate_heads(const void* q_image, const void* gimg, const void* carry_img, const void* carry_lo, const float* coef_table,
                         float* dcarry, float* dcoef_partial, int B, int Hq, int Hkv, int NB, int c0, int NC, float scale,
                         int32_t* status, cudaStream_t st) {
  cudaError_t e = allow_smem<dstate_heads_kernel>(DS_SMEM);
  if (e != cudaSuccess) return e;
  const int sms = sm_count(), items = F_SLABS * NC * B * Hkv;
  DStateArgs a{static_cast<const unsigned char*>(q_image), static_cast<const __nv_bfloat16*>(gimg),
               static_cast<const __nv_bfloat16*>(carry_img), static_cast<const __nv_bfloat16*>(carry_lo), coef_table,
               dcarry, dcoef_partial, NB, Hq, Hkv, B * Hkv, c0, NC, scale, status};
  dstate_heads_kernel<<<items < sms ? items : sms, DS_THREADS, DS_SMEM, st>>>(a);
  return cudaGetLastError();
}

cudaError_t feature_grad(bool query, const void* x_image, const void* a_image, const void* image,
                         const float* coef_table, float* dx, int B, int H, int rep, int N, int NB, int c0, int NC,
                         int32_t* status, cudaStream_t st) {
  const int smem = FG_RING * SLAB_S_BYTES + 2 * SLAB_S_BYTES + 2 * F_ROWS * (int)sizeof(float) + ROW_IMAGE_BYTES + 2 * 16 * CP;
  FeatGradArgs a{static_cast<const unsigned char*>(x_image), static_cast<const unsigned char*>(a_image),
                 static_cast<const __nv_bfloat16*>(image), coef_table, dx, N, NB, H, rep, B, c0, NC, status};
  cudaError_t e;
  const int sms = sm_count(), items = B * H * NC, grid = items < sms ? items : sms;
  if (query) {
    if ((e = allow_smem<feature_grad_kernel<true>>(smem)) != cudaSuccess) return e;
    feature_grad_kernel<true><<<grid, FG_THREADS, smem, st>>>(a);
  } else {
    if ((e = allow_smem<feature_grad_kernel<false>>(smem)) != cudaSuccess) return e;
    feature_grad_kernel<false><<<grid, FG_THREADS, smem, st>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t dcoef_reduce(const float* partial, int outer, int Hq, int G, const int32_t* dim_perm,
                         const int32_t* group_start, float* dcoef, float* slots, cudaStream_t st) {
  dcoef_sum_kernel<<<dim3(F_ROWS / 32, Hq), 256, 0, st>>>(partial, outer, Hq, dcoef);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  dcoef_slots_kernel<<<Hq, 32 * SLOT_WARPS, 0, st>>>(dcoef, dim_perm, group_start, G, slots);
  return cudaGetLastError();
}

cudaError_t norm_vjp_image(const void* grad_out, int out_dt, const float* grad_num, const float* grad_den,
                           const float* num, const float* den, float floor_v, void* gimg, int heads,
                           int N, int NB, int token_major_heads, const RowImages& rows, int32_t* clear_status,
                           cudaStream_t st) {
  norm_vjp_image_kernel<<<(unsigned)((size_t)heads * NB * CT / 32), 256, 0, st>>>(grad_out, out_dt, grad_num, grad_den, num, den, floor_v,
                                                                                  static_cast<__nv_bfloat16*>(gimg), N, NB, heads,
                                                                                  token_major_heads, rows, clear_status);
  return cudaGetLastError();
}

}  // namespace oal
