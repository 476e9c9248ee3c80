// Inter-chunk state kernels on the tensor cores (tcgen05 / TMEM).
//
// Chunked causal scan of the reference (oal_attention/hd_block_gemm_runtime.py:271-320
// block totals and exclusive cumsum, :552-560 cross contraction phi_q x carry) with 128-token
// chunks:
//   state_walk   : dS[u,c] = phi_k(chunk c)^T [v | 1]          (features are the MMA M dimension),
//                  carry[u,c] = state_in + sum_{c'<c} dS[u,c'] (fp32), stored as the bf16
//                  operand image the MMAs read
//   state_update, state_scan : the same in two steps, increments in memory between them, for a range of a longer sequence
//                  (the totals of the ranges are exchanged between the two) and as the reverse scan of the backward
//   cross_read   : Y[i,:] = phi_q(i) . carry[u,c(i)]           (tokens are the MMA M dimension)
// Feature tiles are generated on chip (oal_features.cuh), in shared memory or, for the cross read, straight in tensor
// memory, and never touch HBM.
// The fp32 accumulators live in tensor memory; state images are streamed with 1-D bulk
// async copies.  Every mbarrier wait is bounded (oal_umma.cuh).
#include <algorithm>

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
// First launch of a forward: the first `n_prologue` blocks compute the per-head prologue (oal_prologue.cuh), the others write
// the rows of k and of [v | 1 | 0] as operand images, which the state walk and the backward kernels fetch with bulk copies.
//   Image blocks: 32 consecutive tokens of one (unit, chunk); warp = 8 consecutive columns, lane = token, so a warp stores 512
//   contiguous bytes.  Rows are enumerated over padded chunks: zeros past the end of the sequence.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) rows_prologue_kernel(const PrologueArgs pro, int n_prologue, const RowImages rows, int N, int NB) {
  __shared__ PrologueSmem smem;
  if ((int)blockIdx.x < n_prologue) {
    head_prologue(pro, blockIdx.x, smem, threadIdx.x, 256);
    return;
  }
  const int ec = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t per_unit = (size_t)NB * CT, r = (size_t)(blockIdx.x - n_prologue) * 32 + lane, u = r / per_unit;
  const int t = (int)(r % per_unit), tl = t % CT;
  const bool live = t < N;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const size_t at = (u * N + t) * HD + 8 * ec, chunk = u * NB + t / CT;
  uint4* k_out = reinterpret_cast<uint4*>(static_cast<unsigned char*>(rows.k_image) + chunk * ROW_IMAGE_BYTES);
  uint4* u_out = reinterpret_cast<uint4*>(static_cast<unsigned char*>(rows.u_image) + chunk * SLAB_S_BYTES);
  k_out[ec * CT + tl] = live ? *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(rows.k) + at) : zero;
  u_out[ec * CT + tl] = live ? *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(rows.v) + at) : zero;
  if (ec < 2) u_out[(VD / 8 + ec) * CT + tl] = make_uint4(ec == 0 && live ? 0x00003F80u : 0u, 0u, 0u, 0u);
}

// ---------------------------------------------------------------------------
// state_update: dS[u,c][slab rows] = phi_k^T U
//   one block per (slab group of 4, chunk, unit); 256 threads, thread = (token, half of the slab)
// ---------------------------------------------------------------------------
struct StateUpdateArgs {
  const __nv_bfloat16 *k, *v;   // [units, N, 64]
  float* ds;                    // [units, NB] chunks of F_ROWS x EP floats in state_inc_offset order
  int N, NB, NC;                // chunks of the sequence; chunks whose increment is computed (the first NC)
  int32_t* status;
};

constexpr int GEN_THREADS = 256;      // (token, half of a slab)

__global__ void __launch_bounds__(GEN_THREADS, 2) state_update_kernel(const StateUpdateArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Abuf = smem;                          // 2 x SLAB_A_BYTES
  unsigned char* Uimg = smem + 2 * SLAB_A_BYTES;       // [10][128 tokens][8 e]
  unsigned char* Ximg = Uimg + SLAB_S_BYTES;           // rows of k
  __shared__ uint64_t mma_done[2];
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int item = blockIdx.x;
  const int grp = item % SU_GROUPS, c = (item / SU_GROUPS) % a.NC, u = item / SU_GROUPS / a.NC;
  const int token = tid & 127, half = tid >> 7;
  if (warp == 0) tmem_alloc(&tmem_base, 256);
  if (tid == 0) {
    mbar_init(&mma_done[0], 1);
    mbar_init(&mma_done[1], 1);
    mbar_fence_init();
    dead = 0;
  }
  const __nv_bfloat16* vbase = a.v + (size_t)u * a.N * VD;
  load_rows(Ximg, 0, a.k + ((size_t)u * a.N + c * CT) * HD, CT, a.N - c * CT, tid, GEN_THREADS);
  for (int idx = tid; idx < (EP / 8) * CT; idx += GEN_THREADS) {
    const int ec = idx >> 7, t = idx & 127, j = c * CT + t;
    reinterpret_cast<uint4*>(Uimg)[idx] = u_image_chunk(vbase + (size_t)j * VD, ec, j < a.N);
  }
  async_copies_wait();
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
    const int row = (s0 + it) * 128 + 32 * (warp & 3) + lane;
    const int col0 = warp < 4 ? 0 : 40, ncol = warp < 4 ? 40 : EU - 40;
    const uint32_t t = tacc + (uint32_t)((it & 1) * EP) + ((uint32_t)(32 * (warp & 3)) << 16) + col0;
    for (int cc = 0; cc < ncol; cc += 8) {
      float vv[8];
      tmem_ld8(t + cc, vv);
      tmem_ld_wait();
      float* dst = ds_base + state_inc_offset(row, col0 + cc);
      *reinterpret_cast<float4*>(dst) = make_float4(vv[0], vv[1], vv[2], vv[3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(vv[4], vv[5], vv[6], vv[7]);
    }
    fence_before_sync();
  };

  for (int it = 0; it < ns; ++it) {
    const int buf = it & 1;
    // A[buf] and accumulator buf were released by epilogue(it-2), which every thread has passed
    uint4* tile = reinterpret_cast<uint4*>(Abuf + buf * SLAB_A_BYTES) + 8 * half * CT + token;
    const int hs = 2 * (s0 + it) + half;
    const HalfBlock blk = half_block(min(hs, F_PAIR_BLOCKS - 1));
    const auto piece = [&](int j) { return *reinterpret_cast<const uint4*>(Ximg + j * CP + token * 16); };
    raw_half_slab(hs, piece(blk.rb), piece(blk.cb), piece, [&](int j, uint4 f) { tile[j * CT] = f; });
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
  w.settle();
  if (warp == 0) tmem_dealloc(tmem_base, 256);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
}

// ---------------------------------------------------------------------------
// state_scan: exclusive prefix over chunks (forward) or suffix (reverse), fp32 running sum,
// result stored as the bf16 MMA operand image  [u][c][slab][e/8][128 rows][8 e].
//   Increments and images have the same element order, so a thread owns four consecutive elements and walks the
//   chunks: grid (slabs x used blocks of 8 columns, units), one block of 128 rows x 8 columns per CTA.  Bound by HBM at many units, by the latency of the walk at few:
//   the loads of SCAN_AHEAD chunks are in flight together.  `trim`: the first chunk visited meets a zero state and
//   nothing reads its image, and the increment of the last one visited reaches no image: neither is touched.
// image_lo (optional): a second image of the rounding remainders, bf16(state - bf16(state)); the
// coefficient-gradient dot products of the backward read state = image + image_lo.
// ---------------------------------------------------------------------------
constexpr int SCAN_AHEAD = 4;

__global__ void __launch_bounds__(256) state_scan_kernel(const float* ds, __nv_bfloat16* image,
                                                         __nv_bfloat16* image_lo, const float* state_in,
                                                         float* state_total, int NB, int reverse, int trim) {
  constexpr size_t CHUNK = (size_t)F_ROWS * EP;
  const int slab = blockIdx.x / (EU / 8), e8 = blockIdx.x % (EU / 8), within = threadIdx.x * 4;
  const size_t x = (size_t)(slab * (EP / 8) + e8) * 1024 + within;    // element inside a chunk, image order
  const size_t u = blockIdx.y;
  // row-major position of the same element in state_in / state_total
  const size_t rm = (size_t)(slab * 128 + (within >> 3)) * EP + e8 * 8 + (within & 7);
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
  if (state_total) {
    *reinterpret_cast<float4*>(state_total + u * CHUNK + rm) = run;
    if (e8 == EU / 8 - 1) *reinterpret_cast<float4*>(state_total + u * CHUNK + rm + 8) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// ---------------------------------------------------------------------------
// state_walk: the carry images of every chunk, one block per (unit, slab), which walks the chunks with its 128 x 72 state in
// registers.
//   warps 0-3   thread = token: features of chunk c into A[c % 2], the pieces of k two chunks ahead in registers; warp 0 issues
//               the MMA  Z[c % 2] = A^T [v | 1]
//   warps 4-15  thread = (feature row, 24 columns): image c written while the MMA runs, then the increment of chunk c added;
//               warp 4 has the image of [v | 1] two chunks on copied in
// What bounds it: the chain of a chunk (features, MMA, drain) for a block alone on its SM, 1.4 us per chunk with remainder images
// and 1.2 without; with two blocks the stores of an SM, 37 KB per chunk and block at 16 bytes per clock (2350 clocks, whatever
// the generators do: eight warps, or all in one set of warps, are no faster).  In two kernels the increments, twice the images'
// bytes, go to memory and back: 135 -> 77 us at B = 4, N = 4096, 2 KV heads (152 blocks: two on four SMs); one or two units leave
// most SMs without a block, see state_walk_pays().
// ---------------------------------------------------------------------------
struct StateWalkArgs {
  const unsigned char *k_image, *u_image;
  unsigned char *image, *image_lo; // [units, NB, 19, 10, 128, 8]: state, and bf16(state - bf16(state)) or null
  const float* state_in;           // [units, F_ROWS, EP] row-major, or null
  int NB;
  int first_image;                 // 1: nothing reads the image of the first chunk (a zero state)
  int32_t* status;
};
constexpr int SW_GEN_WARPS = 4, SW_DRAIN_WARPS = 12, SW_THREADS = (SW_GEN_WARPS + SW_DRAIN_WARPS) * 32;
constexpr int SW_BLOCKS = EU / 8 / (SW_DRAIN_WARPS / 4);      // blocks of 8 columns per drain warp
static_assert(SW_BLOCKS * (SW_DRAIN_WARPS / 4) * 8 == EU, "the drain warps share the used columns evenly");
// shared memory: two feature slabs, two images of [v | 1] (the MMA reads 8 columns past the used ones: in bounds, into columns
// of Z that no one reads)
constexpr int SW_U = 2 * SLAB_A_BYTES, SW_SMEM = SW_U + SLAB_U_BYTES + SLAB_S_BYTES;

__global__ void __launch_bounds__(SW_THREADS, 2) state_walk_kernel(const StateWalkArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t z_full[2], z_free[2], u_full[2];
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int slab = blockIdx.x % F_SLABS, u = blockIdx.x / F_SLABS;
  const int n = a.NB - 1;                              // the increment of the last chunk reaches no image
  if (warp == 0) tmem_alloc(&tmem_base, 256);
  const auto fetch_u = [&](int c) {                    // one thread
    mbar_arrive_expect_tx(&u_full[c & 1], SLAB_U_BYTES);
    bulk_g2s(smem + SW_U + (c & 1) * SLAB_U_BYTES, a.u_image + ((size_t)u * a.NB + c) * SLAB_S_BYTES, SLAB_U_BYTES, &u_full[c & 1]);
  };
  if (tid == 0) {
    for (int x = 0; x < 2; ++x) {
      mbar_init(&z_full[x], 1);
      mbar_init(&z_free[x], SW_DRAIN_WARPS);
      mbar_init(&u_full[x], 1);
    }
    mbar_fence_init();
    dead = 0;
    for (int c = 0; c < 2 && c < n; ++c) fetch_u(c);
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  Waiter w{&dead};
  const uint32_t tmem = uniform(tmem_base);

  if (warp < SW_GEN_WARPS) {
    // ---------------- generators ----------------
    const HalfBlock blk[2] = {half_block(min(2 * slab, F_PAIR_BLOCKS - 1)), half_block(min(2 * slab + 1, F_PAIR_BLOCKS - 1))};
    const unsigned char* base = a.k_image + (size_t)u * a.NB * ROW_IMAGE_BYTES + tid * 16;
    uint4 r4[2][2], c4[2][2];                          // [chunk parity][half of the slab]
    const auto fetch_k = [&](int c, int x) {
      const unsigned char* at = base + (size_t)min(c, a.NB - 1) * ROW_IMAGE_BYTES;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        r4[x][h] = load_ahead(at + blk[h].rb * ROW_PLANE);
        c4[x][h] = load_ahead(at + blk[h].cb * ROW_PLANE);
      }
    };
    fetch_k(0, 0);
    fetch_k(1, 1);
    const uint32_t idesc = instr_desc_bf16(128, EP, 1, 1);
    for (int c0 = 0; c0 < n; c0 += 2) {
#pragma unroll
      for (int x = 0; x < 2; ++x) {                    // parity: a register set and a buffer each
        const int c = c0 + x;
        if (c >= n) break;
        if (c >= 2) w.wait(&z_full[x], ((c >> 1) - 1) & 1, 0x11);      // the MMA that read A[x] has completed
        __syncwarp();
        uint4* tile = reinterpret_cast<uint4*>(smem + x * SLAB_A_BYTES) + tid;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          raw_half_slab(2 * slab + h, r4[x][h], c4[x][h],
                        [&](int j) { return __ldg(reinterpret_cast<const uint4*>(base + (size_t)c * ROW_IMAGE_BYTES + j * ROW_PLANE)); },
                        [&](int j, uint4 f) { tile[(8 * h + j) * CT] = f; });
        fetch_k(c + 2, x);
        fence_async_smem();
        asm volatile("bar.sync 1, %0;" ::"n"(SW_GEN_WARPS * 32) : "memory");
        if (warp == 0 && elect_one()) {
          w.wait(&u_full[x], (c >> 1) & 1, 0x12);
          if (c >= 2) w.wait(&z_free[x], ((c >> 1) - 1) & 1, 0x13);
          fence_after_sync();
          const uint64_t da = smem_desc(smem_u32(smem + x * SLAB_A_BYTES), 128, CT * 16);
          const uint64_t du = smem_desc(smem_u32(smem + SW_U + x * SLAB_U_BYTES), 128, ROW_PLANE);
#pragma unroll
          for (int ks = 0; ks < CT / 16; ++ks)
            mma_bf16_ss(tmem + x * EP, desc_advance(da, ks * 256), desc_advance(du, ks * 256), idesc, ks > 0);
          mma_commit(&z_full[x]);
        }
        __syncwarp();
      }
    }
  } else {
    // ---------------- state ----------------
    const int fr = 32 * (warp & 3) + lane, e0 = SW_BLOCKS * ((warp - SW_GEN_WARPS) >> 2);       // feature row, first block of 8 columns
    float run[8 * SW_BLOCKS];
#pragma unroll
    for (int e = 0; e < 8 * SW_BLOCKS; ++e) run[e] = 0.f;
    if (a.state_in) {
      const float* src = a.state_in + ((size_t)u * F_ROWS + slab * 128 + fr) * EP + 8 * e0;
#pragma unroll
      for (int e = 0; e < 8 * SW_BLOCKS; e += 4) {
        const float4 t = *reinterpret_cast<const float4*>(src + e);
        run[e] = t.x; run[e + 1] = t.y; run[e + 2] = t.z; run[e + 3] = t.w;
      }
    }
    const size_t at0 = ((size_t)u * a.NB * F_SLABS + slab) * SLAB_S_BYTES + e0 * ROW_PLANE + fr * 16;
    for (int c = 0; c < a.NB; ++c) {
      if (c >= a.first_image) {
        const size_t at = at0 + (size_t)c * F_SLABS * SLAB_S_BYTES;
#pragma unroll
        for (int e8 = 0; e8 < SW_BLOCKS; ++e8) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float x = run[8 * e8 + 2 * j], y = run[8 * e8 + 2 * j + 1];
            hi[j] = pack_bf16(x, y);
            lo[j] = pack_bf16(x - bf16_lo(hi[j]), y - bf16_hi(hi[j]));
          }
          *reinterpret_cast<uint4*>(a.image + at + e8 * ROW_PLANE) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          if (a.image_lo) *reinterpret_cast<uint4*>(a.image_lo + at + e8 * ROW_PLANE) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
      if (c >= n) break;
      w.wait(&z_full[c & 1], (c >> 1) & 1, 0x14);
      if (warp == SW_GEN_WARPS && lane == 0 && c + 2 < n && !w.gave_up()) fetch_u(c + 2);
      __syncwarp();
      fence_after_sync();
      const uint32_t t = tmem + (c & 1) * EP + ((uint32_t)(32 * (warp & 3)) << 16) + 8 * e0;
      float z[SW_BLOCKS][8];
#pragma unroll
      for (int e8 = 0; e8 < SW_BLOCKS; ++e8) tmem_ld8(t + 8 * e8, z[e8]);
      tmem_ld_wait();
      fence_before_sync();
      warp_arrive(&z_free[c & 1], lane);
#pragma unroll
      for (int e = 0; e < 8 * SW_BLOCKS; ++e) run[e] += z[e >> 3][e & 7];
    }
  }
  fence_before_sync();
  __syncthreads();
  w.settle();
  if (warp == 0) tmem_dealloc(tmem_base, 256);
  if (tid == 0 && dead) atomicOr(a.status, w.status_bits());
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
//   generators  write feature slab `slab` of the item's 128 tokens into tensor memory, A[it % 5]; four sets of four
//               warps (32 tokens each) take the slabs in turn
//   loader      lane 0 streams the state slab images into slot it % 5 of a ring and the head's coefficient
//               table into one of two buffers (bulk copies)
//   issuer      lane 0 issues the MMAs  acc[item & 1] += A . S  once both are there
//   epilogue    after the item's last slab: accumulator -> HBM, then release it
// A slot of features and a slot of the state share one barrier per direction: every wait and every commit costs the
// issuing thread 50 to 100 clocks, and with a pair of each it needed 550 clocks per slab without any MMA (a slab's eight
// MMAs take 480).  The epilogue goes through shared memory: stored by the thread of each row, 64 stores of 32 lines held up
// every other shared-memory access of the SM for 3000 clocks per item.
// What bounds it: the issuing thread (about 650 clocks per slab) and a gap of 1500 clocks at each item.  14 / 2 heads, 8 groups,
// B = 4, N = 4096: 157 -> 116 us (QUERY), 30 -> 25 (not).
constexpr int CR_SETS = 4, CR_GEN_WARPS = 4 * CR_SETS, CR_EPI_WARPS = 4;     // whole warpgroups
constexpr int CR_ISSUER = CR_GEN_WARPS + CR_EPI_WARPS, CR_LOADER = CR_ISSUER + 1;
// Two warps more only fill the issuer's warpgroup, whose registers the generators take: 768 threads x 80 at launch =
// 512 x 88 + 128 x 72 + 128 x 40 and 2048 to spare.
constexpr int CR_THREADS = (CR_LOADER + 3) * 32;
constexpr int CR_RING = 5;
// tensor memory: ring of feature slabs (128 features of the 128 tokens, two per column), two accumulators
constexpr uint32_t CR_SLAB_COLS = 64, CR_ACC = CR_RING * CR_SLAB_COLS;
static_assert(CR_ACC + 2 * EP <= 512, "tensor-memory columns of the cross-read kernel");
// shared memory: ring of state slabs, two coefficient tables, two row images, the epilogue's rows (fp32, padded)
constexpr int CR_COEF = CR_RING * SLAB_S_BYTES, CR_X = CR_COEF + 2 * F_ROWS * 4, CR_STAGE = CR_X + 2 * X_BYTES;
constexpr int CR_PITCH = VD + 4, CR_SMEM = CR_STAGE + CT * CR_PITCH * 4;

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
  __shared__ uint64_t full[CR_RING], done[CR_RING], acc_full[2], acc_free[2];
  __shared__ uint64_t coef_full[2], coef_free[2], x_full[2];
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int n_items = a.B * a.H * a.NC;
  const int my_items = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  if (warp == CR_ISSUER) tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    for (int s = 0; s < CR_RING; ++s) {
      mbar_init(&full[s], 4 + 1);          // the warps of a set, and the loader
      mbar_init(&done[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_free[s], CR_EPI_WARPS);
      mbar_init(&coef_full[s], 1);
      mbar_init(&coef_free[s], CR_GEN_WARPS);
      mbar_init(&x_full[s], CR_GEN_WARPS);
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
    // ---------------- generators ----------------
    registers_up_to<88>();
    const int set = warp >> 2;
    unsigned char* ximg = smem + CR_X;
    const auto fetch = [&](int k) {
      const CrItem it = cr_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
      load_rows(ximg + (k & 1) * X_BYTES, 0, a.x + ((size_t)(it.b * a.H + it.h) * a.N + it.c * CT) * HD, CT, a.N - it.c * CT, tid,
                CR_GEN_WARPS * 32);
    };
    if (my_items > 0) fetch(0);
    int flat = set;                                      // slab of this set, over all items
    for (int k = 0; k < my_items; ++k) {
      async_copies_wait();
      warp_arrive(&x_full[k & 1], lane);
      w.wait(&x_full[k & 1], (k >> 1) & 1, 0x49);        // the rows are in, and item k-1 has been generated
      if (k + 1 < my_items) fetch(k + 1);
      // this head's coefficient table, brought in by the loader warp (two buffers)
      const float* coef = reinterpret_cast<const float*>(smem + CR_COEF) + (k & 1) * F_ROWS;
      if constexpr (QUERY) w.wait(&coef_full[k & 1], (k >> 1) & 1, 0x47);
      const unsigned char* xlane = ximg + (k & 1) * X_BYTES + (32 * (warp & 3) + (lane >> 2)) * 16;
      for (; flat < (k + 1) * F_SLABS; flat += CR_SETS) {
        const int slot_i = flat % CR_RING, use = flat / CR_RING, slab = flat - k * F_SLABS;
        if (use > 0) w.wait(&done[slot_i], (use - 1) & 1, 0x41);      // the MMAs that read the slot have completed
        __syncwarp();
        fence_after_sync();
        const uint32_t slot = tmem + slot_i * CR_SLAB_COLS + ((uint32_t)(32 * (warp & 3)) << 16);
        store_half_slab<QUERY>(2 * slab, xlane, coef, slot, lane);
        store_half_slab<QUERY>(2 * slab + 1, xlane, coef, slot + CR_SLAB_COLS / 2, lane);
        tmem_st_wait();
        fence_before_sync();
        warp_arrive(&full[slot_i], lane);
      }
      if constexpr (QUERY) warp_arrive(&coef_free[k & 1], lane);     // this warp no longer reads the table
    }
  } else if (warp < CR_ISSUER) {
    // ---------------- accumulator -> HBM ----------------
    registers_down_to<72>();
    const uint32_t lane_off = (uint32_t)(32 * (warp & 3)) << 16;
    float* stage = reinterpret_cast<float*>(smem + CR_STAGE) + 32 * (warp & 3) * CR_PITCH;      // this warp's 32 rows
    for (int k = 0; k < my_items; ++k) {
      const CrItem it = cr_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
      const int row0 = it.c * CT + 32 * (warp & 3);
      const size_t orow = (size_t)(it.b * a.H + it.h) * a.N + row0;
      w.wait(&acc_full[k & 1], (k >> 1) & 1, 0x42);
      __syncwarp();
      fence_after_sync();
      const uint32_t t = tmem + CR_ACC + (k & 1) * EP + lane_off;
#pragma unroll
      for (int cc = 0; cc < VD; cc += 16) {
        float vv[16];
        tmem_ld16(t + cc, vv);
        tmem_ld_wait();
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4)
          *reinterpret_cast<float4*>(stage + lane * CR_PITCH + cc + 4 * q4) = make_float4(vv[4 * q4], vv[4 * q4 + 1], vv[4 * q4 + 2], vv[4 * q4 + 3]);
      }
      float den[8] = {};
      if constexpr (QUERY) {
        tmem_ld8(t + VD, den);
        tmem_ld_wait();
      }
      fence_before_sync();
      warp_arrive(&acc_free[k & 1], lane);              // (and the staged rows are visible to the warp)
      if (!dead) {
        if (QUERY && row0 + lane < a.N) a.out1[orow + lane] = den[0];
#pragma unroll 4
        for (int x = lane; x < 32 * (VD / 4); x += 32) {
          const int r = x / (VD / 4), c4 = x % (VD / 4);
          if (row0 + r < a.N)
            *reinterpret_cast<float4*>(a.out64 + orow * VD + 4 * x) = *reinterpret_cast<const float4*>(stage + r * CR_PITCH + 4 * c4);
        }
      }
      __syncwarp();
    }
  } else {
    registers_down_to<40>();
    if (warp == CR_ISSUER && elect_one()) {
      // ---------------- MMA issue ----------------
      const uint32_t idesc = instr_desc_bf16(128, EP, 0, 1);
      // descriptor of slot 0 of the image ring, advanced by adds: this thread is the serial path of every slab
      const uint64_t ds0 = smem_desc(smem_u32(smem), 128, 128 * 16);
      int slot = 0, use = 0;
      for (int k = 0; k < my_items; ++k) {
        const uint32_t tacc = tmem + CR_ACC + (k & 1) * EP;
        if (k >= 2) w.wait(&acc_free[k & 1], ((k >> 1) - 1) & 1, 0x43);   // item k-2 has left this accumulator
        for (int s = 0; s < F_SLABS; ++s) {
          const uint64_t dsl = desc_advance(ds0, slot * SLAB_S_BYTES);
          const uint32_t slab = tmem + slot * CR_SLAB_COLS;
          w.wait(&full[slot], use & 1, 0x44);
          fence_after_sync();
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)       // 16 features per step
            if (s < F_SLABS - 1 || ks < LAST_STEPS) mma_bf16_ts(tacc, slab + 8 * ks, desc_advance(dsl, ks * 256), idesc, (s > 0 || ks > 0));
          mma_commit(&done[slot]);
          if (++slot == CR_RING) { slot = 0; ++use; }
        }
        mma_commit(&acc_full[k & 1]);
      }
    }
    if (warp == CR_LOADER && elect_one()) {
      // ---------------- state image and coefficient stream ----------------
      int slot = 0, use = 0;
      const auto fetch_coef = [&](int k) {
        const CrItem it = cr_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
        if (k >= 2 && !w.met(&coef_free[k & 1], ((k >> 1) - 1) & 1, 0x48)) return;   // item k-2 no longer reads this buffer
        mbar_arrive_expect_tx(&coef_full[k & 1], F_ROWS * (uint32_t)sizeof(float));
        bulk_g2s(smem + CR_COEF + (k & 1) * F_ROWS * sizeof(float), a.coef_table + (size_t)it.h * F_ROWS,
                 F_ROWS * (uint32_t)sizeof(float), &coef_full[k & 1]);
      };
      if (QUERY && my_items > 0) fetch_coef(0);
      for (int k = 0; k < my_items && !w.gave_up(); ++k) {
        const CrItem it = cr_item(blockIdx.x + k * gridDim.x, a.H, a.rep, a.NC, a.c0);
        const int unit = (it.b * a.H + it.h) / a.rep;
        const unsigned char* img = reinterpret_cast<const unsigned char*>(a.image) +
                                   ((size_t)unit * a.NB + it.c) * F_SLABS * SLAB_S_BYTES;
        for (int s = 0; s < F_SLABS; ++s) {
          // the next item's table while there is time: its buffer's last reader was item k-1
          if (QUERY && s == 2 * F_SLABS / 3 && k + 1 < my_items) fetch_coef(k + 1);
          if (use > 0 && !w.met(&done[slot], (use - 1) & 1, 0x46)) break;
          // the unused columns of an image only reach unused columns of the accumulator
          mbar_arrive_expect_tx(&full[slot], SLAB_U_BYTES);
          bulk_g2s(smem + slot * SLAB_S_BYTES, img + (size_t)s * SLAB_S_BYTES, SLAB_U_BYTES, &full[slot]);
          if (++slot == CR_RING) { slot = 0; ++use; }
        }
      }
    }
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  w.settle();
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

cudaError_t state_update(const void* k, const void* v, float* ds, int units, int N, int NB, int NC, int32_t* status, cudaStream_t st) {
  const int smem = 2 * SLAB_A_BYTES + SLAB_S_BYTES + X_BYTES;
  cudaError_t e = allow_smem<state_update_kernel>(smem);
  if (e != cudaSuccess) return e;
  StateUpdateArgs a{static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), ds, N, NB, NC, status};
  state_update_kernel<<<SU_GROUPS * NC * units, GEN_THREADS, smem, st>>>(a);
  return cudaGetLastError();
}

// The walk against the two kernels, whose increments go to memory and back: a chunk costs the walk 1.3 us (its blocks' chain)
// and the two kernels 0.36 us per unit and, once, 7.6 us for the second launch and its first loads; a walk of a few units that
// writes more than about 1000 chunks in all loses another 0.9 us per chunk.  Whole forwards as recorded graphs, walk less two
// steps in us, with (without) remainder images:
//   units      4 chunks    8             16            32           64           128          256          512
//     1       -6 (-6)     0 (-2)       +10 (+6)      +30 (+24)    +60 (+48)   +115 (+98)   +231 (+184)  +478 (+393)
//     2       -6 (-5)    -2 (-2)        +7 (+3)      +16 (+12)    +36 (+26)    +67 (+47)   +154 (+111)  +407 (+274)
//     3       -6 (-7)    -3 (-4)        -3 (-4)       -4 (-6)      +3 (-1)      +3 (+1)     +44 (+19)   +185 (+159)
//     4       -7 (-7)    -2 (-4)        -6 (-5)       -7 (-10)    -24 (-20)    -40 (-36)    -25 (-30)    +53 (+73)
//     6       -7 (-7)   -11 (-13)      -22 (-22)     -41 (-32)    -80 (-72)   -108 (-114)  -173 (-138)  -305 (-211)
//    14      -14 (-15)  -30 (-30)      -63 (-54)    -121 (-121)  -221 (-220)  -422 (-387)  -823 (-736)
//    32      -25 (-25)  -71 (-62)     -134 (-126)   -261 (-240)  -532 (-463) -1051 (-906)
bool state_walk_pays(int units, int NB) {
  return NB * (1.3 - 0.36 * units) + 0.9 * std::max(0, NB - 1000 / units) < 7.6;
}

cudaError_t rows_prologue(const RowImages& rows, int units, int N, int NB, const PrologueArgs* prologue, int q_heads, cudaStream_t st) {
  const int n_pro = prologue ? q_heads : 0;
  rows_prologue_kernel<<<n_pro + units * NB * (CT / 32), 256, 0, st>>>(prologue ? *prologue : PrologueArgs{}, n_pro, rows, N, NB);
  return cudaGetLastError();
}

cudaError_t state_walk(const RowImages& rows, void* image, void* image_lo, const float* state_in, int units, int NB, bool trim,
                       int32_t* status, cudaStream_t st) {
  cudaError_t e = allow_smem<state_walk_kernel>(SW_SMEM);
  if (e != cudaSuccess) return e;
  StateWalkArgs a{static_cast<const unsigned char*>(rows.k_image), static_cast<const unsigned char*>(rows.u_image),
                  static_cast<unsigned char*>(image), static_cast<unsigned char*>(image_lo), state_in, NB, trim ? 1 : 0, status};
  state_walk_kernel<<<F_SLABS * units, SW_THREADS, SW_SMEM, st>>>(a);
  return cudaGetLastError();
}

cudaError_t state_scan(const float* ds, void* image, void* image_lo, const float* state_in, float* state_total,
                       int units, int NB, int reverse, bool trim, cudaStream_t st) {
  state_scan_kernel<<<dim3(F_SLABS * (EU / 8), units), 256, 0, st>>>(
      ds, static_cast<__nv_bfloat16*>(image), static_cast<__nv_bfloat16*>(image_lo), state_in, state_total, NB, reverse,
      trim ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t cross_read(bool query, const void* x, const void* image, const float* coef_table, float* out64,
                       float* out1, int B, int H, int rep, int N, int NB, int c0, int NC, int32_t* status,
                       cudaStream_t st) {
  CrossReadArgs a{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(image), coef_table,
                  out64, out1, N, NB, H, rep, B, c0, NC, status};
  cudaError_t e;
  const int sms = sm_count(), items = B * H * NC, grid = items < sms ? items : sms;
  if (query) {
    if ((e = allow_smem<cross_read_kernel<true>>(CR_SMEM)) != cudaSuccess) return e;
    cross_read_kernel<true><<<grid, CR_THREADS, CR_SMEM, st>>>(a);
  } else {
    if ((e = allow_smem<cross_read_kernel<false>>(CR_SMEM)) != cudaSuccess) return e;
    cross_read_kernel<false><<<grid, CR_THREADS, CR_SMEM, st>>>(a);
  }
  return cudaGetLastError();
}

size_t state_rows() { return F_ROWS; }
size_t state_image_bytes_per_chunk() { return (size_t)F_SLABS * SLAB_S_BYTES; }
size_t state_slab_image_bytes() { return SLAB_S_BYTES; }

}  // namespace oal
