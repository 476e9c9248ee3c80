// Quadratic feature map of the chunked scan, laid out for the tensor cores.
//
// The reference materialises phi_k = [1, k_d, k_r k_c (r >= c)] and
// phi_q = [A, B_{g(d)} q_d, m C_{g(r)g(c)} q_r q_c] as [tokens, 2145] matrices in HBM
// (oal_attention/hd_block_gemm_feature_forward.py:225-253, :373-385; pair order
// oal_attention/hd_block_gemm_cache.py:105-121).  Here a feature tile only ever exists in
// shared memory or tensor memory, in bf16.  The feature order is internal (the running state is never exposed): 64
// consecutive features are one 8 x 8 block of x x^T,
//   features 64 hs + 16 (c / 2) + 2 r + c % 2:  x[8 rb + r] * x[8 cb + c],  r, c = 0 .. 7,  rb >= cb
//   blocks hs = 0 .. 35 by cb, then rb; in a diagonal block the entries above the diagonal (c > r) have no meaning
//   features 2304 + d: linear, x[d];   feature 2368: constant;   zeros up to 2432
// Two blocks (128 features) form a slab: 19 slabs, 2432 feature rows.  What the order is for:
//   * a block needs 16 of a token's 64 values, so a thread reads two 16-byte pieces of the token's row from shared memory;
//   * pairs of features (2 r + 16 i, + 1) share r and take adjacent columns: one broadcast and one packed multiply;
//   * in tensor memory an accumulator fragment (.16x256b: thread t of a warp holds, of 16 rows, rows t / 4 and t / 4 + 8,
//     and of every 8 columns, columns 2 (t % 4) and + 1) gives a thread two rows r and all eight columns c of a block for
//     each of four tokens, as bf16 operand (two features per column) and as fp32 accumulator: the coefficients that a thread
//     reads serve four tokens, and sums over c need no exchange.
#pragma once

#include "oal_common.cuh"
#include "oal_umma.cuh"

namespace oal {

constexpr int F_BLOCK = 64;                    // features of a block of x x^T, or half slab
constexpr int F_PAIR_BLOCKS = 36;
constexpr int F_LINEAR = F_PAIR_BLOCKS * F_BLOCK, F_CONST = F_LINEAR + HD;
constexpr int F_SLABS = 19;
constexpr int F_ROWS = F_SLABS * 128;          // 2432
constexpr int LAST_STEPS = (F_CONST - 128 * (F_SLABS - 1)) / 16 + 1;      // 16-feature steps of the last slab before its padding
constexpr int CT = 128;                        // tokens per chunk of the scan
constexpr int SLAB_A_BYTES = 128 * CT * 2;     // feature slab tile  [16 chunks][128 tokens][8] bf16
constexpr int SLAB_S_BYTES = (EP / 8) * 128 * 16;   // state slab image [10][128 features][8 e] bf16
// Columns of [v | 1 | 0] that can be other than zero, in whole blocks of 8.  The last block of an image or increment only
// completes the extent that the MMA wants (a multiple of 16): it is never written, copied or read.
constexpr int EU = (E1 + 7) / 8 * 8;
constexpr int SLAB_U_BYTES = (EU / 8) * 128 * 16;

// Per-chunk fp32 state increments (and state-gradient increments) are stored like the bf16 state
// image, [slab][e / 8][128 rows][8 e], so that a warp whose lanes are consecutive feature rows writes
// and reads contiguous kilobytes.  Float index of (feature row f, column e) inside one chunk:
__host__ __device__ constexpr size_t state_inc_offset(int f, int e) {
  return ((size_t)((f >> 7) * (EP / 8) + (e >> 3)) * 128 + (f & 127)) * 8 + (e & 7);
}

// Row and column block of half slab hs < F_PAIR_BLOCKS.
struct HalfBlock {
  int rb, cb;
};
__host__ __device__ constexpr HalfBlock half_pos(int hs) {
  int cb = 0;
  while (hs >= 8 - cb) {
    hs -= 8 - cb;
    ++cb;
  }
  return HalfBlock{cb + hs, cb};
}

// What feature row f is: kind 0 pair (r, c; `live` false for the repeated entries above the diagonal),
// 1 linear (r = dimension), 2 constant, 3 padding.
struct FeatureId {
  int kind, r, c;
  bool live;
};
__host__ __device__ inline FeatureId feature_id(int f) {
  FeatureId id{3, 0, 0, false};
  if (f < F_LINEAR) {
    const HalfBlock blk = half_pos(f / F_BLOCK);
    const int y = f % F_BLOCK;
    id.kind = 0;
    id.r = 8 * blk.rb + ((y >> 1) & 7);
    id.c = 8 * blk.cb + 2 * (y >> 4) + (y & 1);
    id.live = id.c <= id.r;
  } else if (f < F_CONST) {
    id.kind = 1;
    id.r = f - F_LINEAR;
    id.live = true;
  } else if (f == F_CONST) {
    id.kind = 2;
    id.live = true;
  }
  return id;
}

// Power of the query scale folded into the per-head coefficient table: the query-side kernels work
// on the unscaled q, so pair coefficients carry scale^2 and linear ones scale.
__host__ __device__ inline float feature_scale_factor(int f, float scale) {
  return f < F_LINEAR ? scale * scale : (f < F_CONST ? scale : 1.f);
}

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

constexpr int ROW_PLANE = CT * 16;             // one 16-byte piece of every row of a chunk
constexpr int ROW_IMAGE_BYTES = 8 * ROW_PLANE; // a chunk's rows of 64 as an operand image [8][128][8], zeros past the sequence

// ---- rows in shared memory -----------------------------------------------------------------------
// Chunk planes of an operand image that threads write: 128 rows of 16 bytes and 16 bytes of padding, so that eight
// threads that copy one 128-byte row (coalesced) hit eight different bank groups.
constexpr int CP = CT * 16 + 16;
constexpr int X_BYTES = 8 * CP;

// 16-byte asynchronous copy global -> shared (zero fill when `valid` is false); completion with
// async_copies_wait().  All copies of a thread are in flight together, so an image costs one memory
// latency instead of one per 16 bytes.
__device__ __forceinline__ void async_copy16(void* dst_smem, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::smem_u32(dst_smem)), "l"(src),
               "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void async_copies_wait() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// `rows` rows of 64 bf16 from `src` (consecutive, the first `valid` exist) -> operand image [8][rows][8] at row `row0`,
// plane pitch CP, by threads tid of nthreads (a multiple of 8).  A tile of rows is contiguous: a thread keeps its column
// piece and advances both addresses by constants (with the row computed for every piece, the address arithmetic took
// longer than the copies).
__device__ __forceinline__ void load_rows(unsigned char* img, int row0, const __nv_bfloat16* src, int rows, int valid, int tid,
                                          int nthreads) {
  const int step = nthreads >> 3;
  unsigned char* dst = img + (tid & 7) * CP + (row0 + (tid >> 3)) * 16;
  const __nv_bfloat16* from = src + (size_t)tid * 8;
  for (int r = tid >> 3; r < rows; r += step, dst += step * 16, from += (size_t)nthreads * 8)
    async_copy16(dst, r < valid ? from : src, r < valid);
}

// ---- half slabs -------------------------------------------------------------------------------------
// The code is the same for every half slab.  (The form this replaces, one specialised piece of code per 8 features and the
// row in registers, was 60 to 100 KB of straight-line code and needed the whole row where a half slab uses a quarter of it.)
// Entries above the diagonal are generated too: their coefficients are zero, so they reach no result.
constexpr int HALF_LINEAR = F_PAIR_BLOCKS, HALF_CONST = F_PAIR_BLOCKS + 1;
static_assert(HALF_CONST == 2 * F_SLABS - 1, "the constant starts the last half slab");
constexpr uint64_t half_slab_rows(int word) {          // 4 bits per half slab, 16 half slabs per word
  uint64_t w = 0;
  for (int h = 16 * word; h < 16 * word + 16 && h < F_PAIR_BLOCKS; ++h) w |= (uint64_t)half_pos(h).rb << (4 * (h - 16 * word));
  return w;
}
constexpr uint64_t half_slab_columns(int word) {
  uint64_t w = 0;
  for (int h = 16 * word; h < 16 * word + 16 && h < F_PAIR_BLOCKS; ++h) w |= (uint64_t)half_pos(h).cb << (4 * (h - 16 * word));
  return w;
}
static __constant__ uint64_t kHalfRow[3] = {half_slab_rows(0), half_slab_rows(1), half_slab_rows(2)};
static __constant__ uint64_t kHalfCol[3] = {half_slab_columns(0), half_slab_columns(1), half_slab_columns(2)};
__device__ __forceinline__ HalfBlock half_block(int hs) {      // hs < F_PAIR_BLOCKS, warp-uniform
  const int sh = 4 * (hs & 15);
  return HalfBlock{(int)(kHalfRow[hs >> 4] >> sh) & 15, (int)(kHalfCol[hs >> 4] >> sh) & 15};
}
__device__ __forceinline__ uint32_t bf16_twice(uint32_t word, int high) { return __byte_perm(word, word, high ? 0x3232u : 0x1010u); }

// Coefficient-free features of half slab hs of one token, eight at a time: emit(j, 16 bytes), j = 0 .. 7, from the pieces of
// the token's row that hold the block's rows and columns (`r4`, `c4`) or, for the linear features, piece(j).  The product of
// two bf16 values rounded once to bf16 is what an fp32 multiply followed by a conversion gives, so the packed multiply
// yields those bits at two features per instruction.
template <class Piece, class Emit>
__device__ __forceinline__ void raw_half_slab(int hs, const uint4 r4, const uint4 c4, Piece piece, Emit emit) {
  if (hs < F_PAIR_BLOCKS) {
    const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w};
    uint32_t r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = bf16_twice(rw[j / 2], j & 1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t* rr = r + 4 * (j & 1);
      emit(j, make_uint4(mul_bf16x2(rr[0], c[j / 2]), mul_bf16x2(rr[1], c[j / 2]), mul_bf16x2(rr[2], c[j / 2]), mul_bf16x2(rr[3], c[j / 2])));
    }
  } else if (hs == HALF_LINEAR) {
#pragma unroll
    for (int j = 0; j < 8; ++j) emit(j, piece(j));
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) emit(j, make_uint4(j == 0 ? 0x00003F80u : 0u, 0u, 0u, 0u));   // bf16(1.0) first
  }
}

// Features of half slab hs for the 32 tokens of a warp as the MMA's A operand in tensor memory (32 columns, a feature pair
// each).  A lane works on rows r = 2 (lane % 4) and + 1 of the block for the tokens lane / 4 + 8 t, t = 0 .. 3.  `xlane`
// points at token lane / 4 of the warp in plane 0 of the row image, `slot` at the half slab's first column at the warp's
// lanes.  COEF: times the per-head coefficient table (feature order, query scale folded in, zero above the diagonal and in
// the padding), in fp32 and rounded once.
template <bool COEF>
__device__ __forceinline__ void store_half_slab(int hs, const unsigned char* xlane, const float* coef, uint32_t slot, int lane) {
  const int m = lane & 3;
  const float* cf = coef + F_BLOCK * hs + 4 * m;
  uint32_t o[2][16];                       // [tokens 0, 8 | 16, 24][column pair i: (token, column 2 m), (token, + 1), (token + 8, ..) ..]
  f32x2 ca[4], cb[4];
  const auto load_coefs = [&]() {
    if constexpr (COEF) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(cf + 16 * i);
        ca[i] = c.x;
        cb[i] = c.y;
      }
    }
  };
  const auto pack = [](f32x2 f) {
    float lo, hi;
    f2_unpack(f, lo, hi);
    return umma::pack_bf16(lo, hi);
  };
  if (hs < F_PAIR_BLOCKS) {
    const HalfBlock blk = half_block(hs);
    load_coefs();
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const unsigned char* x = xlane + 128 * t;
      uint32_t* out = &o[t >> 1][2 * (t & 1)];
      const uint32_t r = *reinterpret_cast<const uint32_t*>(x + blk.rb * CP + 4 * m);
      const uint4 c4 = *reinterpret_cast<const uint4*>(x + blk.cb * CP);
      const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
      if constexpr (COEF) {
        const f32x2 xa = f2_bcast(bf16_lo(r)), xb = f2_bcast(bf16_hi(r));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f32x2 xc = f2_pack(bf16_lo(c[i]), bf16_hi(c[i]));
          out[4 * i] = pack(f2_mul(f2_mul(xa, xc), ca[i]));
          out[4 * i + 1] = pack(f2_mul(f2_mul(xb, xc), cb[i]));
        }
      } else {
        const uint32_t xa = bf16_twice(r, 0), xb = bf16_twice(r, 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          out[4 * i] = mul_bf16x2(xa, c[i]);
          out[4 * i + 1] = mul_bf16x2(xb, c[i]);
        }
      }
    }
  } else if (hs == HALF_LINEAR) {
    load_coefs();
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t* out = &o[t >> 1][2 * (t & 1)];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint2 d = *reinterpret_cast<const uint2*>(xlane + 128 * t + (2 * i + (m >> 1)) * CP + 8 * (m & 1));
        out[4 * i] = COEF ? pack(f2_mul(f2_pack(bf16_lo(d.x), bf16_hi(d.x)), ca[i])) : d.x;
        out[4 * i + 1] = COEF ? pack(f2_mul(f2_pack(bf16_lo(d.y), bf16_hi(d.y)), cb[i])) : d.y;
      }
    }
  } else {
    const uint32_t first = COEF ? umma::pack_bf16(cf[0], 0.f) : 0x00003F80u;
#pragma unroll
    for (int x = 0; x < 16; ++x) o[0][x] = o[1][x] = (m == 0 && (x == 0 || x == 2)) ? first : 0u;
  }
  umma::tmem_st_rows16(slot, o[0]);
  umma::tmem_st_rows16(slot + (16u << 16), o[1]);
}

// 16 bytes through the read-only path, issued where it stands: the compiler may move an ordinary load down to its first use,
// behind the waits that it was meant to overlap.
__device__ __forceinline__ uint4 load_ahead(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// Bounded mbarrier waits for one CTA: the first wait that expires raises a shared flag and every
// later wait returns at once, so a kernel always terminates; the flag ends up in the status word.
// A thread that issues bulk copies stops at its first wait that was not met, and a CTA that gave up settles before it frees
// its tensor memory and leaves: a bulk copy that lands in the shared memory of a CTA that has left is a launch failure, and
// the barriers that would tell when the last one is in have lost their phases.  (MMAs touch the CTA's own memory only and
// queue a few deep: their thread runs its loop to the end.  With a check there the cross read took 111 us instead of 108.)
struct Waiter {
  int* dead;          // shared flag: a wait expired somewhere in this CTA (holds the site id, >= 1)
  __device__ __forceinline__ bool gave_up() const { return *reinterpret_cast<volatile int*>(dead) != 0; }
  // whether the phase has completed; false: this or another thread's wait expired
  __device__ __forceinline__ bool met(uint64_t* bar, uint32_t parity, int site) {
    if (umma::mbar_test(bar, parity)) return true;      // already complete: the common case costs one probe
    if (gave_up()) return false;
    if (umma::mbar_wait(bar, parity)) return true;
    *reinterpret_cast<volatile int*>(dead) = site;
    return false;
  }
  __device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity, int site = 1) { met(bar, parity, site); }
  // Every thread, after the last barrier of the CTA.  What is still in flight then (at most the shared memory of an SM, and
  // the queue of MMAs) takes microseconds; the pause is a thousand times that.
  __device__ __forceinline__ void settle() const {
    if (!gave_up()) return;
    for (const long long t0 = clock64(); clock64() - t0 < SETTLE_CLOCKS;) __nanosleep(1000);
  }
  static constexpr long long SETTLE_CLOCKS = 4000000;      // 2 ms
  // status bits to OR into the caller's word: the timeout flag plus the site id in bits 8..15
  __device__ __forceinline__ int status_bits() const {
    const int d = *reinterpret_cast<volatile int*>(dead);
    return d ? (OAL_STATUS_WAIT_TIMEOUT | ((d & 0xFF) << 8)) : 0;
  }
};


// One arrival per warp on an mbarrier after every lane has finished what precedes (shared-memory
// stores made visible to the async proxy, or tensor-memory accesses).
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) umma::mbar_arrive(bar);
}

// 16-byte image chunk (8 consecutive e of one token) of U = [v | 1 | 0]
__device__ __forceinline__ uint4 u_image_chunk(const __nv_bfloat16* vrow, int ec, bool valid) {
  if (!valid) return make_uint4(0u, 0u, 0u, 0u);
  if (ec < VD / 8) return *reinterpret_cast<const uint4*>(vrow + 8 * ec);
  if (ec == VD / 8) return make_uint4(0x00003F80u, 0u, 0u, 0u);   // bf16(1.0) in element 0
  return make_uint4(0u, 0u, 0u, 0u);
}


}  // namespace oal
