// Shared pieces of the tensor-core intra-chunk kernels.
//
// Per token pair (i, j) of one query head the kernel weight is a quadratic form in
// v = [1, s_1 .. s_G], s_g = sum_{d in g} (scale q_i[d]) k_j[d]:
//     w = v^T M v,   M = [[A, B/2], [B/2, C]]          (oal_attention/grouped_reference.py:61-99)
// With the eigen-decomposition M = V diag(sigma) V^T (oal_prologue.cuh for a packed factor,
// head_factor_kernel for explicit coefficients; one per call) and lambda_r = sqrt|sigma_r| the weight is a
// signed sum of squares
//     w = w0 + sum_r sgn_r u_r^2,   u_r(i,j) = c_r + sum_d q_i[d] (l_r[d] k_j[d]),
//     c_r = lambda_r V[0][r],  l_r[d] = scale lambda_r V[1 + g(d)][r],
// so every u_r is one plain 64-long dot product of a per-dimension scaled copy of one side's row with the other
// side's row, and dimension groups need no sorting or padding.
//
// The kernels walk the terms, not the keys: term r scales the 128 rows of the CTA (the MMA's A operand, written
// to tensor memory by the threads that own the rows), one MMA chain gives u_r for all pairs of the chunk at once,
// and the pair weights w (or the products with dW) stay in registers while r advances.  The other side's rows are
// one shared-memory image that every term reads unchanged.  Against walking 16-key tiles with all R scaled copies
// of the tile stacked in shared memory (the form this replaces) that is a third of the instructions, no
// shared-memory rebuild and no weight hand-over per tile, code that does not depend on R (any number of groups),
// and the coefficient gradient as sums over rows instead of R (R + 1) / 2 products per pair (intra_bwd).
#pragma once

#include "oal_features.cuh"

namespace oal {

constexpr int RMAX_ALL = OAL_MAX_GROUPS + 1;         // 17: extent of the per-head factor table
constexpr int T_PITCH = 20;
constexpr int XA_BYTES = 10 * CP;                    // [v | 1 | 0]

// What a kernel keeps of a head's table besides l.
struct HeadScalars {
  float c[RMAX_ALL];                 // c_r
  float w0;                          // constant added to the weight (the packed-factor form keeps its eps out of the terms)
  int rank;                          // R = G + 1
  int rpos;                          // terms r < rpos enter with +, the others with -
};
static_assert(sizeof(HeadScalars) == 80, "copied in 16-byte pieces");

// Dimensions sorted by group.
struct HeadOrder {
  uint8_t pos[HD];                   // position of a dimension
  uint8_t start[32];                 // first position of group g; 64 from group G on
};
static_assert(sizeof(HeadOrder) == 96, "copied in 16-byte pieces");

// What the query side of the backward reads of the groups and coefficients of a head (HeadFactor::e, mask, order), by
// threads tid of nthreads; `pos` and `group` of every dimension are known, b_of(g) = B_g, c_of(g, g2) = C_gg2 + C_g2g.
template <class BOf, class COf>
__device__ __forceinline__ void write_head_groups(float (&e)[RMAX_ALL][HD], uint32_t (&mask)[GMAX][HD / 2], HeadOrder& order,
                                                  const int* group, const int32_t* dim_perm, const int32_t* group_start, int G,
                                                  float scale, BOf b_of, COf c_of, int tid, int nthreads) {
  for (int x = tid; x < (G + 1) * HD; x += nthreads) {
    const int r = x / HD, g = group[x % HD];
    e[r][x % HD] = r == 0 ? scale * b_of(g) : scale * scale * c_of(r - 1, g);
  }
  for (int x = tid; x < G * (HD / 2); x += nthreads) {
    const int g = x / (HD / 2), wd = x % (HD / 2);
    mask[g][wd] = (group[2 * wd] == g ? 0x0000FFFFu : 0u) | (group[2 * wd + 1] == g ? 0xFFFF0000u : 0u);
  }
  for (int p = tid; p < HD; p += nthreads) order.pos[dim_perm[p]] = (uint8_t)p;
  for (int g = tid; g < 32; g += nthreads) order.start[g] = (uint8_t)(g < G ? group_start[g] : HD);
}

// Per-head factor table in global memory (written by the prologue or head_factor_kernel).
struct alignas(16) HeadFactor {
  HeadScalars s;
  float l[RMAX_ALL][HD];             // l_r[d], original dimension order
  float e[RMAX_ALL][HD];             // of the dimension's group g: e_0 = scale B_g, e_r = scale^2 (C_rg + C_gr)
  uint32_t mask[GMAX][HD / 2];       // the dimensions of a group, as words of two bf16
  HeadOrder order;
  float t[RMAX_ALL][T_PITCH];        // t[a][r] = V[a][r] / lambda_r  (v = t u)
};
static_assert(offsetof(HeadFactor, t) % 16 == 0 && sizeof(HeadFactor::t) % 16 == 0, "copied in 16-byte pieces");

// Chunks 8 and 9 of the image of [v | 1 | 0]: one in the first element of rows below `valid`, zeros elsewhere.
__device__ __forceinline__ void augment_rows(unsigned char* img, int valid, int tid, int nthreads) {
  for (int x = tid; x < 2 * CT; x += nthreads) {
    const int r = x & 127;
    *reinterpret_cast<uint4*>(img + (8 + (x >> 7)) * CP + r * 16) = make_uint4((x < CT && r < valid) ? 0x00003F80u : 0u, 0u, 0u, 0u);
  }
}
// A head's l (rank rows) and scalars, by threads tid of nthreads.
__device__ __forceinline__ void load_head(float* l, HeadScalars* sc, const HeadFactor* f, int rank, int tid, int nthreads) {
  for (int x = tid; x < rank * (HD / 4) + 5; x += nthreads) {
    const int y = x - 5;
    if (y < 0) async_copy16(reinterpret_cast<unsigned char*>(sc) + x * 16, reinterpret_cast<const unsigned char*>(&f->s) + x * 16, true);
    else async_copy16(l + 4 * y, &f->l[0][0] + 4 * y, true);
  }
}

// Term r of this thread's row as the MMA's A operand in tensor memory: bf16(l_r[d] x[d]) for 16 dimensions from d0
// (columns d0 / 2 ..) and, 32 columns further, the rounding remainders: the scaled side enters u_r with about 16
// bits.  xrow points at the thread's row in chunk 0 of an image.
constexpr uint32_t TERM_COLS = 64;
template <int PITCH = CP>
__device__ __forceinline__ void build_term16(uint32_t slot, const unsigned char* xrow, const float* l, int d0) {
  uint32_t hw[8], lw[8];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint4 raw = *reinterpret_cast<const uint4*>(xrow + (d0 / 8 + k) * PITCH);
    const ulonglong2 la = *reinterpret_cast<const ulonglong2*>(l + d0 + 8 * k);
    const ulonglong2 lb = *reinterpret_cast<const ulonglong2*>(l + d0 + 8 * k + 4);
    const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
    const f32x2 lv[4] = {la.x, la.y, lb.x, lb.y};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a, b;
      f2_unpack(f2_mul(f2_pack(bf16_lo(rw[j]), bf16_hi(rw[j])), lv[j]), a, b);
      const uint32_t h = umma::pack_bf16(a, b);
      hw[4 * k + j] = h;
      lw[4 * k + j] = umma::pack_bf16(a - bf16_lo(h), b - bf16_hi(h));
    }
  }
  umma::tmem_st8(slot + d0 / 2, hw);
  umma::tmem_st8(slot + 32 + d0 / 2, lw);
}

// term . rows^T into 128 x n columns, K = 64 for the value and 64 for the remainder operand: `b_addr` is the first of
// the n rows in an image.  (The kernels add c_r themselves, in fp32.)
template <int PITCH = CP>
__device__ __forceinline__ void issue_term(uint32_t tmem_u, uint32_t slot, uint32_t b_addr, int n) {
  const uint32_t idesc = umma::instr_desc_bf16(128, n, 0, 0);
  const uint64_t db = umma::smem_desc(b_addr, PITCH, 128);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
    umma::mma_bf16_ts(tmem_u, slot + 8 * ks, umma::desc_advance(db, (ks & 3) * 2 * PITCH), idesc, ks > 0);
}

// Query-side tiles.  The 128 rows of a CTA are four blocks of 32 query rows, one per tensor-memory lane quadrant,
// that share a key / value chunk but not necessarily a head: the 4 rep row blocks of the rep query heads of a KV
// head are taken in the order of how many keys they see (block 3 of every head, then block 2, ...), four at a time.
// Tile t then needs keys 0 .. 32 (4 - 4 t / rep) - 1 only, and its four quadrants see about the same number of them:
// with the rows of one head in a tile, the quadrant of rows 96..127 works on all 128 keys while that of rows 0..31
// is masked out of 96, and its scheduler is what the kernel waits for.  For rep = 7: 608 key columns per chunk
// and KV head instead of 896.
// Grid: (chunk, batch row x KV head, tile); tiles with the most keys are launched first, so the last wave is made of
// short ones.
struct QueryTile {
  int b, kvh, c, t, rep, nc;          // nc: tokens of the chunk
  __device__ __forceinline__ QueryTile(int Hkv, int N, int rep_) {
    c = blockIdx.x;
    b = blockIdx.y / Hkv;
    kvh = blockIdx.y - b * Hkv;
    t = blockIdx.z;
    rep = rep_;
    nc = min(CT, N - c * CT);
  }
  __device__ __forceinline__ int rb(int quadrant) const { return 3 - (4 * t + quadrant) / rep; }
  __device__ __forceinline__ int head(int quadrant) const { return kvh * rep + (4 * t + quadrant) % rep; }
  __device__ __forceinline__ int columns() const { return min(32 * (rb(0) + 1), (nc + 31) & ~31); }
  __device__ __forceinline__ bool empty() const { return 32 * rb(3) >= nc; }
};

}  // namespace oal
