// Inter-chunk state kernels on the tensor cores (tcgen05 / TMEM).
//
// Chunked causal scan of the reference (oal_attention/hd_block_gemm_runtime.py:271-320
// block totals and exclusive cumsum, :552-560 cross contraction phi_q x carry) with 128-token
// chunks:
//   state_update : dS[u,c] = phi_k(chunk c)^T [v | 1]          (features are the MMA M dimension)
//   state_scan   : carry[u,c] = state_in + sum_{c'<c} dS[u,c'] (fp32), stored as the bf16
//                  operand image the MMAs read
//   cross_read   : Y[i,:] = phi_q(i) . carry[u,c(i)]           (tokens are the MMA M dimension)
// Feature tiles are generated on chip (oal_features.cuh), in shared memory or, for the cross read, straight in tensor
// memory, and never touch HBM.
// The fp32 accumulators live in tensor memory; state images are streamed with 1-D bulk
// async copies.  Every mbarrier wait is bounded (oal_umma.cuh).
#include "oal_features.cuh"
#include "oal_kernels.h"
#include "oal_prologue.cuh"

namespace oal {
namespace {

using namespace umma;

// the 19 slabs are processed by four CTAs per (chunk, unit): slab groups 5, 5, 5, 4
constexpr int SU_GROUPS = 4;
__device__ __forceinline__ int group_first_slab(int g) { return 5 * g; }
__device__ __forceinline__ int group_slab_count(int g) { return g < 3 ? 5 : F_SLABS - 15; }

// ---------------------------------------------------------------------------
// per-head coefficient table in feature order (fp32 [Hq][F_ROWS]), query scale folded in:
// pair rows carry scale^2, linear rows scale (the query-side kernels read the unscaled q)
// ---------------------------------------------------------------------------
__global__ void coef_table_kernel(const int32_t* dim_perm, const int32_t* group_start, const float* A,
                                  const float* Bc, const float* Cc, int G, float scale, float* table) {
  __shared__ int gdim[HD];
  const int h = blockIdx.x;
  if (threadIdx.x < HD) {
    const int p = threadIdx.x;
    int g = 0;
    while (g < GMAX - 1 && p >= group_start[h * (GMAX + 1) + g + 1]) ++g;
    gdim[dim_perm[h * HD + p]] = g;
  }
  __syncthreads();
  for (int f = threadIdx.x; f < F_ROWS; f += blockDim.x) {
    float v = 0.f;
    const FeatureId id = feature_id(f);
    if (id.kind == 0 && id.live) {
      const int gr = min(gdim[id.r], G - 1), gc = min(gdim[id.c], G - 1);
      v = (id.r == id.c ? 1.f : 2.f) * Cc[((size_t)h * G + gr) * G + gc];
    } else if (id.kind == 1) {
      v = Bc[h * G + min(gdim[id.r], G - 1)];
    } else if (id.kind == 2) {
      v = A[h];
    }
    table[(size_t)h * F_ROWS + f] = v * feature_scale_factor(f, scale);
  }
}

// ---------------------------------------------------------------------------
// state_update: dS[u,c][slab rows] = phi_k^T U
//   one block per (slab group of 4, chunk, unit); 256 threads, thread = (token, half of the slab's chunks).
//   The first `n_prologue` blocks compute the per-head prologue instead (oal_prologue.cuh): it has no input in
//   common with this kernel, both are needed next, and one launch costs less than two and a fork.
// ---------------------------------------------------------------------------
struct StateUpdateArgs {
  const __nv_bfloat16 *k, *v;   // [units, N, 64]
  float* ds;                    // [units, NB] chunks of F_ROWS x EP floats in state_inc_offset order
  int N, NB, NC;                // chunks of the sequence; chunks whose increment is computed (the first NC)
  int32_t* status;
  int32_t* block_status;        // with a prologue that clears `status` in this launch: a word per block instead, see state_scan
};

__global__ void __launch_bounds__(GEN_THREADS, 2) state_update_kernel(const StateUpdateArgs a, const PrologueArgs pro,
                                                                      int n_prologue) {
  extern __shared__ __align__(128) unsigned char smem[];
  if ((int)blockIdx.x < n_prologue) {
    head_prologue(pro, blockIdx.x, *reinterpret_cast<PrologueSmem*>(smem), threadIdx.x, GEN_THREADS);
    return;
  }
  unsigned char* Abuf = smem;                          // 2 x SLAB_A_BYTES
  unsigned char* Uimg = smem + 2 * SLAB_A_BYTES;       // [10][128 tokens][8 e]
  __shared__ uint64_t mma_done[2];
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int item = (int)blockIdx.x - n_prologue;
  const int grp = item % SU_GROUPS, c = (item / SU_GROUPS) % a.NC, u = item / SU_GROUPS / a.NC;
  const int token = tid & 127, half = tid >> 7;
  if (warp == 0) tmem_alloc(&tmem_base, 256);
  if (tid == 0) {
    mbar_init(&mma_done[0], 1);
    mbar_init(&mma_done[1], 1);
    mbar_fence_init();
    dead = 0;
  }
  const int i = c * CT + token;
  const __nv_bfloat16* kbase = a.k + (size_t)u * a.N * HD;
  const __nv_bfloat16* vbase = a.v + (size_t)u * a.N * VD;
  uint32_t xp[HD / 2];
  load_row_packed(xp, kbase, i, a.N);
  for (int idx = tid; idx < (EP / 8) * CT; idx += GEN_THREADS) {
    const int ec = idx >> 7, t = idx & 127, j = c * CT + t;
    reinterpret_cast<uint4*>(Uimg)[idx] = u_image_chunk(vbase + (size_t)j * VD, ec, j < a.N);
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);
  const uint32_t tacc = tmem;
  const int s0 = group_first_slab(grp), ns = group_slab_count(grp);
  const uint32_t idesc = instr_desc_bf16(128, EP, 1, 1);
  const uint32_t u_addr = smem_u32(Uimg);
  float* ds_base = a.ds + ((size_t)u * a.NB + c) * F_ROWS * EP;

  auto epilogue = [&](int it) {
    w.wait(&mma_done[it & 1], (it >> 1) & 1);
    fence_after_sync();
    if (warp >= 8) return;          // warps 0-7 cover the 128 lanes x 80 columns
    const int row = (s0 + it) * 128 + 32 * (warp & 3) + lane;
    const int col0 = warp < 4 ? 0 : 48, ncol = warp < 4 ? 48 : 32;
    const uint32_t t = tacc + (uint32_t)((it & 1) * EP) + ((uint32_t)(32 * (warp & 3)) << 16) + col0;
    for (int cc = 0; cc < ncol; cc += 16) {
      float vv[16];
      tmem_ld16(t + cc, vv);
      tmem_ld_wait();
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        *reinterpret_cast<float4*>(ds_base + state_inc_offset(row, col0 + cc + 4 * q4)) =
            make_float4(vv[4 * q4], vv[4 * q4 + 1], vv[4 * q4 + 2], vv[4 * q4 + 3]);
    }
    fence_before_sync();
  };

  for (int it = 0; it < ns; ++it) {
    const int buf = it & 1;
    // A[buf] and accumulator buf were released by epilogue(it-2), which every thread has passed
    keep_in_loop(xp);
    write_half_slab_raw(s0 + it, half, xp, reinterpret_cast<uint4*>(Abuf + buf * SLAB_A_BYTES) + token);
    fence_async_smem();
    __syncthreads();
    if (warp == 0 && elect_one()) {
      fence_after_sync();
      const uint64_t da = smem_desc(smem_u32(Abuf + buf * SLAB_A_BYTES), 128, CT * 16);
      const uint64_t du = smem_desc(u_addr, 128, CT * 16);
#pragma unroll
      for (int ks = 0; ks < CT / 16; ++ks)
        mma_bf16_ss(tacc + buf * EP, desc_advance(da, ks * 256), desc_advance(du, ks * 256), idesc, ks > 0);
      mma_commit(&mma_done[buf]);
    }
    if (it >= 1) epilogue(it - 1);
  }
  epilogue(ns - 1);
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 256);
  if (tid == 0) {
    const int32_t bits = dead ? w.status_bits() : 0;
    if (a.block_status) a.block_status[item] = bits;
    else if (bits) atomicOr(a.status, bits);
  }
}

// ---------------------------------------------------------------------------
// state_scan: exclusive prefix over chunks (forward) or suffix (reverse), fp32 running sum,
// result stored as the bf16 MMA operand image  [u][c][slab][e/8][128 rows][8 e].
//   Increments and images have the same element order, so a thread owns four consecutive elements and walks the
//   chunks: grid (F_ROWS * EP / 4 / 256, units).  Bound by HBM at many units, by the latency of the walk at few:
//   the loads of SCAN_AHEAD chunks are in flight together.  `trim`: the first chunk visited meets a zero state and
//   nothing reads its image, and the increment of the last one visited reaches no image: neither is touched.
// image_lo (optional): a second image of the rounding remainders, bf16(state - bf16(state)); the
// coefficient-gradient dot products of the backward read state = image + image_lo.
// block_status (optional): words left by the blocks of a state update whose launch also cleared `status`; nothing orders
// that store against an atomic of the same launch, so they are merged into it here.
// ---------------------------------------------------------------------------
constexpr int SCAN_AHEAD = 4;

__global__ void __launch_bounds__(256) state_scan_kernel(const float* ds, __nv_bfloat16* image,
                                                         __nv_bfloat16* image_lo, const float* state_in,
                                                         float* state_total, int NB, int reverse, int trim,
                                                         const int32_t* block_status, int n_status, int32_t* status) {
  constexpr size_t CHUNK = (size_t)F_ROWS * EP;
  static_assert(CHUNK % 1024 == 0, "the grid covers a chunk exactly");
  const size_t x = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;      // element inside a chunk, image order
  const size_t u = blockIdx.y;
  // row-major position of the same element in state_in / state_total
  const int tile = (int)(x >> 10), within = (int)(x & 1023);          // 1024 = 128 rows x 8 columns
  const size_t rm = (size_t)((tile / (EP / 8)) * 128 + (within >> 3)) * EP + (tile % (EP / 8)) * 8 + (within & 7);
  for (size_t b = (size_t)blockIdx.y * (CHUNK / 4) + x / 4; b < (size_t)n_status; b += (size_t)gridDim.y * (CHUNK / 4))
    if (block_status[b]) atomicOr(status, block_status[b]);
  float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
  if (state_in) run = *reinterpret_cast<const float4*>(state_in + u * CHUNK + rm);
  const float* src = ds + u * NB * CHUNK + x;
  const size_t dst = u * NB * CHUNK + x;
  for (int n0 = 0; n0 < NB; n0 += SCAN_AHEAD) {
    float4 inc[SCAN_AHEAD];
#pragma unroll
    for (int k = 0; k < SCAN_AHEAD; ++k) {
      const int n = n0 + k, c = reverse ? NB - 1 - n : n;
      if (n < NB - trim) inc[k] = __ldcs(reinterpret_cast<const float4*>(src + c * CHUNK));
    }
#pragma unroll
    for (int k = 0; k < SCAN_AHEAD; ++k) {
      const int n = n0 + k, c = reverse ? NB - 1 - n : n;
      if (n >= NB) break;
      if (image && n >= trim) {
        const uint2 hi = make_uint2(pack_bf16(run.x, run.y), pack_bf16(run.z, run.w));
        *reinterpret_cast<uint2*>(image + dst + c * CHUNK) = hi;
        if (image_lo)
          *reinterpret_cast<uint2*>(image_lo + dst + c * CHUNK) =
              make_uint2(pack_bf16(run.x - bf16_lo(hi.x), run.y - bf16_hi(hi.x)),
                         pack_bf16(run.z - bf16_lo(hi.y), run.w - bf16_hi(hi.y)));
      }
      if (n < NB - trim) {
        run.x += inc[k].x; run.y += inc[k].y; run.z += inc[k].z; run.w += inc[k].w;
      }
    }
  }
  if (state_total) *reinterpret_cast<float4*>(state_total + u * CHUNK + rm) = run;
}

// ---------------------------------------------------------------------------
// cross_read: Y[i, 0:80] = phi(i) . state_image[u, c]   (sum over all slabs)
//   QUERY : phi = phi_q of head h (coefficient table with the query scale folded in), x = q, output num/den
//   !QUERY: phi = phi_k, x = k, output columns 0..63 (the value part) to out64
// ---------------------------------------------------------------------------
struct CrossReadArgs {
  const __nv_bfloat16* x;        // q [B,Hq,N,64] or k [B,Hkv,N,64]
  const __nv_bfloat16* image;    // [units, NB, 19, 10, 128, 8]
  const float* coef_table;       // [Hq, F_ROWS] (QUERY)
  float* out64;                  // [B,H,N,64]
  float* out1;                   // [B,H,N] (QUERY: denominator)
  int N, NB, H, rep, B;          // rep = heads per state unit (Hq/Hkv for QUERY, 1 otherwise)
  int c0, NC;                    // chunks [c0, c0 + NC) of each sequence (the others meet a zero state)
  int32_t* status;
};

// Persistent, warp-specialised kernel.  Work items are (batch, head, chunk) with the heads of one
// state unit adjacent, so CTAs running at the same time read the same state image from L2.  CTA k
// takes items k, k + gridDim.x, ...; the flat iteration `it` = (item, slab) drives four roles:
//   warps 0-7   generate feature slab `slab` of the item's 128 tokens into tensor memory, A[it % 4]
//   warp  13    lane 0 streams the state slab images into a 6-slot ring and the head's coefficient
//               table into one of two buffers (bulk copies)
//   warp  12    lane 0 issues the MMAs  acc[item & 1] += A . S  once both are full
//   warps 8-11  after the item's last slab: accumulator -> HBM, then release it
// What bounded it: shared memory.  With the slabs there an MMA of 128 x 80 x 16 reads 6.5 KB (53 clocks at 128 bytes
// per clock), a slab is written and read at 32 KB each beside the 20 KB of state that arrive and are read: 970 of the
// 1550 clocks a slab took.  A token is a tensor-memory lane and its thread writes the slab's columns itself, which
// leaves the state image alone in shared memory.  Generating with 16 warps
// and copying a quarter of the state changed nothing before that.  14 / 2 heads, B = 4, N = 4096: 187 -> 156 us
// (QUERY), 32 -> 26 (not).
constexpr int CR_GEN_WARPS = 8, CR_EPI_WARPS = 4;
constexpr int CR_ISSUER = CR_GEN_WARPS + CR_EPI_WARPS, CR_LOADER = CR_ISSUER + 1;
constexpr int CR_THREADS = (CR_LOADER + 1) * 32;
constexpr int CR_ARING = 4, CR_SRING = 6;
// tensor memory: ring of feature slabs (128 features of the 128 tokens, two per column), two accumulators
constexpr uint32_t CR_SLAB_COLS = 64, CR_ACC = CR_ARING * CR_SLAB_COLS;
static_assert(CR_ACC + 2 * EP <= 512, "tensor-memory columns of the cross-read kernel");
static_assert(CR_GEN_WARPS * 32 == GEN_THREADS, "the slab generator is written for GEN_THREADS threads");

struct CrItem {
  int b, h, c;
};
// item index -> (batch, head, chunk): the `rep` heads of a state unit are adjacent, then chunks
__device__ __forceinline__ CrItem cr_item(int item, int H, int rep, int NC, int c0) {
  CrItem r;
  const int hh = item % rep, t = item / rep;
  r.c = c0 + t % NC;
  const int unit = t / NC, units_per_b = H / rep;
  r.b = unit / units_per_b;
  r.h = (unit % units_per_b) * rep + hh;
  return r;
}

template <bool QUERY>
__global__ void __launch_bounds__(CR_THREADS, 1) cross_read_kernel(const CrossReadArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Sbuf = smem;                                   // CR_SRING x SLAB_S_BYTES, then the head's coefficient table
  __shared__ uint64_t full_a[CR_ARING], a_free[CR_ARING], s_full[CR_SRING], s_free[CR_SRING], acc_full[2], acc_free[2];
  __shared__ uint64_t coef_full[2], coef_free[2];
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int n_items = a.B * a.H * a.NC;
  const int my_items = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  if (warp == CR_ISSUER) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    for (int s = 0; s < CR_ARING; ++s) {
      mbar_init(&full_a[s], CR_GEN_WARPS);
      mbar_init(&a_free[s], 1);
    }
    for (int s = 0; s < CR_SRING; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_free[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_free[s], CR_EPI_WARPS);
      mbar_init(&coef_full[s], 1);
      mbar_init(&coef_free[s], CR_GEN_WARPS);
    }
    mbar_fence_init();
    dead = 0;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);

  if (warp < CR_GEN_WARPS) {
    // ---------------- generators: thread = (token, half of the slab's chunks) ----------------
    const int token = tid & 127, half = warp >> 2;
    int s3 = 0, use = 0;
    for (int k = 0; k < my_items; ++k) {
      const CrItem it = cr_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
      // this head's coefficient table, brought in by the loader warp (two buffers)
      const float* coef = reinterpret_cast<const float*>(Sbuf + CR_SRING * SLAB_S_BYTES) + (k & 1) * F_ROWS;
      if constexpr (QUERY) w.wait(&coef_full[k & 1], (k >> 1) & 1, 0x47);
      uint32_t xp[HD / 2];
      load_row_packed(xp, a.x + (size_t)(it.b * a.H + it.h) * a.N * HD, it.c * CT + token, a.N);
      f32x2 xq[QUERY ? HD / 2 : 1];
      if constexpr (QUERY) unpack_row(xp, xq);
      for (int s = 0; s < F_SLABS; ++s) {
        if (use > 0) w.wait(&a_free[s3], (use - 1) & 1, 0x41);      // the MMAs that read A[s3] have completed
        __syncwarp();
        fence_after_sync();
        const uint32_t slot = tmem + s3 * CR_SLAB_COLS + ((uint32_t)(32 * (warp & 3)) << 16);
        if constexpr (QUERY) {
          keep_in_loop(xq);
          store_half_slab_coef(s, half, xq, coef, slot);
        } else {
          keep_in_loop(xp);
          store_half_slab_raw(s, half, xp, slot);
        }
        tmem_st_wait();
        fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_a[s3]);
        if (++s3 == CR_ARING) { s3 = 0; ++use; }
      }
      if constexpr (QUERY) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&coef_free[k & 1]);     // this warp no longer reads the table
      }
    }
  } else if (warp < CR_ISSUER) {
    // ---------------- accumulator -> HBM ----------------
    const uint32_t lane_off = (uint32_t)(32 * (warp & 3)) << 16;
    for (int k = 0; k < my_items; ++k) {
      const CrItem it = cr_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
      const int row = it.c * CT + 32 * (warp & 3) + lane;
      const size_t orow = (size_t)(it.b * a.H + it.h) * a.N + row;
      w.wait(&acc_full[k & 1], (k >> 1) & 1, 0x42);
      fence_after_sync();
      const uint32_t t = tmem + CR_ACC + (k & 1) * EP + lane_off;
#pragma unroll
      for (int cc = 0; cc < EP; cc += 16) {
        if (cc < VD || QUERY) {
          float vv[16];
          tmem_ld16(t + cc, vv);
          tmem_ld_wait();
          if (row < a.N && !dead) {
            if (cc < VD) {
#pragma unroll
              for (int q4 = 0; q4 < 4; ++q4)
                *reinterpret_cast<float4*>(a.out64 + orow * VD + cc + 4 * q4) =
                    make_float4(vv[4 * q4], vv[4 * q4 + 1], vv[4 * q4 + 2], vv[4 * q4 + 3]);
            } else if (QUERY) {
              a.out1[orow] = vv[0];
            }
          }
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_free[k & 1]);
    }
  } else if (warp == CR_ISSUER) {
    // ---------------- MMA issue ----------------
    if (elect_one()) {
      const uint32_t idesc = instr_desc_bf16(128, EP, 0, 1);
      // descriptor of slot 0 of the image ring, advanced by adds: this thread is the serial path of every slab
      const uint64_t ds0 = smem_desc(smem_u32(Sbuf), 128, 128 * 16);
      int s3 = 0, use = 0, gs = 0, guse = 0;
      for (int k = 0; k < my_items; ++k) {
        const uint32_t tacc = tmem + CR_ACC + (k & 1) * EP;
        if (k >= 2) w.wait(&acc_free[k & 1], ((k >> 1) - 1) & 1, 0x43);   // item k-2 has left this accumulator
        for (int s = 0; s < F_SLABS; ++s) {
          const uint64_t dsl = desc_advance(ds0, gs * SLAB_S_BYTES);
          const uint32_t slab = tmem + s3 * CR_SLAB_COLS;
          w.wait(&full_a[s3], use & 1, 0x44);
          w.wait(&s_full[gs], guse & 1, 0x45);
          fence_after_sync();
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)       // 16 features per step
            mma_bf16_ts(tacc, slab + 8 * ks, desc_advance(dsl, ks * 256), idesc, (s > 0 || ks > 0));
          mma_commit(&a_free[s3]);
          mma_commit(&s_free[gs]);
          if (s == F_SLABS - 1) mma_commit(&acc_full[k & 1]);
          if (++s3 == CR_ARING) { s3 = 0; ++use; }
          if (++gs == CR_SRING) { gs = 0; ++guse; }
        }
      }
    }
    __syncwarp();
  } else {
    // ---------------- state image stream ----------------
    if (elect_one()) {
      int gs = 0, guse = 0;
      for (int k = 0; k < my_items; ++k) {
        const CrItem it = cr_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
        const int unit = (it.b * a.H + it.h) / a.rep;
        const unsigned char* img = reinterpret_cast<const unsigned char*>(a.image) +
                                   ((size_t)unit * a.NB + it.c) * F_SLABS * SLAB_S_BYTES;
        if constexpr (QUERY) {
          if (k >= 2) w.wait(&coef_free[k & 1], ((k >> 1) - 1) & 1, 0x48);   // item k-2 no longer reads this buffer
          mbar_arrive_expect_tx(&coef_full[k & 1], F_ROWS * (uint32_t)sizeof(float));
          bulk_g2s(Sbuf + CR_SRING * SLAB_S_BYTES + (k & 1) * F_ROWS * sizeof(float),
                   a.coef_table + (size_t)it.h * F_ROWS, F_ROWS * (uint32_t)sizeof(float), &coef_full[k & 1]);
        }
        for (int s = 0; s < F_SLABS; ++s) {
          if (guse > 0) w.wait(&s_free[gs], (guse - 1) & 1, 0x46);
          mbar_arrive_expect_tx(&s_full[gs], SLAB_S_BYTES);
          bulk_g2s(Sbuf + gs * SLAB_S_BYTES, img + (size_t)s * SLAB_S_BYTES, SLAB_S_BYTES, &s_full[gs]);
          if (++gs == CR_SRING) { gs = 0; ++guse; }
        }
      }
    }
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  if (warp == CR_ISSUER) tmem_dealloc(tmem_base, 512);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
}

}  // namespace

// ---------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------
cudaError_t build_coef_table(const int32_t* dim_perm, const int32_t* group_start, const float* A,
                             const float* Bc, const float* Cc, int Hq, int G, float scale, float* table,
                             cudaStream_t st) {
  coef_table_kernel<<<Hq, 256, 0, st>>>(dim_perm, group_start, A, Bc, Cc, G, scale, table);
  return cudaGetLastError();
}

int state_update_blocks(int units, int NC) { return SU_GROUPS * NC * units; }

cudaError_t state_update(const void* k, const void* v, float* ds, int units, int N, int NB, int NC, const PrologueArgs* prologue,
                         int q_heads, int32_t* status, int32_t* block_status, cudaStream_t st) {
  const int smem = 2 * SLAB_A_BYTES + SLAB_S_BYTES;
  cudaError_t e = allow_smem<state_update_kernel>(smem);
  if (e != cudaSuccess) return e;
  StateUpdateArgs a{static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), ds, N, NB, NC, status, block_status};
  const int n_pro = prologue ? q_heads : 0;
  state_update_kernel<<<n_pro + state_update_blocks(units, NC), GEN_THREADS, smem, st>>>(a, prologue ? *prologue : PrologueArgs{}, n_pro);
  return cudaGetLastError();
}

cudaError_t state_scan(const float* ds, void* image, void* image_lo, const float* state_in, float* state_total,
                       int units, int NB, int reverse, bool trim, const int32_t* block_status, int n_status, int32_t* status,
                       cudaStream_t st) {
  state_scan_kernel<<<dim3(F_ROWS * EP / 1024, units), 256, 0, st>>>(
      ds, static_cast<__nv_bfloat16*>(image), static_cast<__nv_bfloat16*>(image_lo), state_in, state_total, NB, reverse,
      trim ? 1 : 0, block_status, block_status ? n_status : 0, status);
  return cudaGetLastError();
}

cudaError_t cross_read(bool query, const void* x, const void* image, const float* coef_table, float* out64,
                       float* out1, int B, int H, int rep, int N, int NB, int c0, int NC, int32_t* status,
                       cudaStream_t st) {
  const int smem = CR_SRING * SLAB_S_BYTES + 2 * F_ROWS * (int)sizeof(float);
  CrossReadArgs a{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(image), coef_table,
                  out64, out1, N, NB, H, rep, B, c0, NC, status};
  cudaError_t e;
  const int sms = sm_count(), items = B * H * NC, grid = items < sms ? items : sms;
  if (query) {
    if ((e = allow_smem<cross_read_kernel<true>>(smem)) != cudaSuccess) return e;
    cross_read_kernel<true><<<grid, CR_THREADS, smem, st>>>(a);
  } else {
    if ((e = allow_smem<cross_read_kernel<false>>(smem)) != cudaSuccess) return e;
    cross_read_kernel<false><<<grid, CR_THREADS, smem, st>>>(a);
  }
  return cudaGetLastError();
}

size_t state_rows() { return F_ROWS; }
size_t state_image_bytes_per_chunk() { return (size_t)F_SLABS * SLAB_S_BYTES; }
size_t state_slab_image_bytes() { return SLAB_S_BYTES; }

}  // namespace oal
