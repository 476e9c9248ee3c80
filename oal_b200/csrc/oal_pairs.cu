// Token-pair kernels (fp32 CUDA-core arithmetic).
//
// They evaluate the kernel weight of a (query i, key j) pair directly from the
// per-group dot products
//     s_g(i,j) = sum_{d in g} (scale q_i[d]) k_j[d]
//     w(i,j)   = A + sum_g B_g s_g + sum_{g,g'} C_gg' s_g s_g'
// and accumulate  num_i, den_i = sum_{j<=i} w(i,j) [v_j, 1]  together with the
// first-order gradients, over the whole causal prefix of every query: the exact fp32 mode of the operator
// (reference semantics: oal_attention/grouped_reference.py:102-178, dense statement
// tests/operators/test_grouped_quadratic.py:31-84).
//
// What bounds them is the FMA pipe (about 170 FMA per pair forward, 280 / 320 in the two backward kernels at 8
// groups) and, next to it, shared-memory wavefronts: an SM retires four warp-FMAs per clock but one 128-byte
// wavefront.  So every phase works on register tiles fed by 16-byte loads:
//   * tiles are stored transposed, [dimension in group order][token], row pitch 68: a warp of 8 x 4 threads reads
//     four owner tokens per thread and JP others in one wavefront each, JP x 4 FMAs per dimension; threads that
//     walk tokens of one dimension (lanes over dimensions) read four tokens per conflict-free load;
//   * a thread keeps all group scores of its 4 x JP pairs in registers, 64 or 128 of them;
//   * per-group weight gradients go through shared memory once, and a thread then owns 16 tokens of ONE
//     dimension, so that the group of its dimension is fixed.
// Clusters of up to 8 CTAs share an owner tile when there are too few tiles to fill the chip: each takes every
// S-th tile of the other side, and the partial sums meet through distributed shared memory in rank order.
//
// Measured against one pair per (thread, key slot) with scalar shared-memory reads, us: 14 / 2 heads, N = 2048,
// 8 groups: forward 955 -> 398, query side 2500 -> 681, key/value side 8124 -> 867 with its reduction; 2 heads,
// N = 256, 4 groups: 76 -> 22, 119 -> 21, 126 -> 25.
// Dimensions of a head are visited in group-sorted order (dim_perm), so a group is
// a contiguous range and s_g needs no gather.
#include <cooperative_groups.h>

#include "oal_common.cuh"
#include "oal_kernels.h"

namespace oal {

namespace {

namespace cg = cooperative_groups;

constexpr int TP = 64;       // pair tile edge
constexpr int PT = 68;       // row pitch of a transposed tile: 16-byte rows, 8 consecutive rows cover all banks
constexpr int TT = HD * PT;  // floats of a transposed tile
constexpr int THREADS = 256;

__device__ __forceinline__ int tri_index(int g, int g2) {   // g <= g2 < GMAX
  return g * GMAX - (g * (g - 1)) / 2 + (g2 - g);
}

// JP by group capacity.  At 8 groups the query side takes 4 (128 scores, 255 registers: 681 us at N = 2048, 14 heads,
// against 750 with 2); the forward is faster with 2 and two CTAs per SM (398 us against 451 with 4 and one), the
// key/value side spills with 4.
constexpr int jp(int gcap) { return gcap <= 4 ? 4 : gcap <= 8 ? 2 : 1; }
constexpr int jp_q(int gcap) { return gcap <= 8 ? 4 : 1; }
template <int GCAP, int JPT>
struct PairCfg {
  static constexpr int JP = JPT;     // 4 x JP pairs per thread
  static constexpr int SUB = 16 * JP;                              // tokens of the other side per pass
  static constexpr int GS = SUB * TP + 4;                          // group stride of the weight gradients
};

// Head description and coefficients in shared memory; C2 = C + C^T (the gradients use 2 C of a symmetric C).
template <int GCAP>
struct HeadInfo {
  HeadGroups hg;
  int inv[HD];
  float A;
  alignas(16) float B[GCAP];
  alignas(16) float C2[GCAP * GCAP];
};

template <int GCAP>
__device__ __forceinline__ void load_head(HeadInfo<GCAP>& hi, const PairArgs& a, int h, bool twice, int tid) {
  load_head_groups(hi.hg, a.dim_perm, a.group_start, h, tid, THREADS);
  if (tid == 0) hi.A = a.A[h];
  for (int x = tid; x < GCAP; x += THREADS) hi.B[x] = x < a.G ? a.Bc[h * a.G + x] : 0.f;
  for (int x = tid; x < GCAP * GCAP; x += THREADS) {
    const int g = x / GCAP, g2 = x % GCAP;
    float c = 0.f;
    if (g < a.G && g2 < a.G) {
      c = a.Cc[(h * a.G + g) * a.G + g2];
      c = twice ? 2.f * c : g == g2 ? c : c + a.Cc[(h * a.G + g2) * a.G + g];
    }
    hi.C2[x] = c;
  }
  for (int x = tid; x < HD; x += THREADS) hi.inv[hi.hg.perm[x]] = x;      // perm was staged before load_head_groups' barrier
  __syncthreads();
}

// Four consecutive elements; `vec`: the tensor starts on a boundary of four elements.
__device__ __forceinline__ void load_quad(const void* src, size_t at, int dt, bool vec, float (&o)[4]) {
  if (vec) {
    load4(src, at, dt, o);
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) o[c] = load_elem(src, at + c, dt);
  }
}

// Rows [row0, row0 + 64) of a [.., N, pitch] tensor, columns 0..63 -> dst[place(column)][row], pitch PT; rows past N
// are zero.  Eight lanes read 128 contiguous bytes of a row; a lane stores its four columns in an order rotated by its
// column block, so that the 32 stores of an instruction fall into 32 banks when place() is the identity.
template <class Place>
__device__ __forceinline__ void load_transposed(float* dst, const void* src, size_t base, int pitch, int row0, int N, int dt, bool vec,
                                                float mul, Place place, int tid) {
  const int cb = tid & 7, r = tid >> 3;
  const int rot = (cb >> 1) & 3;
  float v[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int row = r + 32 * (x >> 1), col = 4 * cb + 32 * (x & 1);
#pragma unroll
    for (int c = 0; c < 4; ++c) v[x][c] = 0.f;
    if (row0 + row < N) load_quad(src, base + (size_t)(row0 + row) * pitch + col, dt, vec, v[x]);
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int row = r + 32 * (x >> 1), col = 4 * cb + 32 * (x & 1);
    const float a0 = rot & 1 ? v[x][1] : v[x][0], a1 = rot & 1 ? v[x][2] : v[x][1];
    const float a2 = rot & 1 ? v[x][3] : v[x][2], a3 = rot & 1 ? v[x][0] : v[x][3];
    const float w[4] = {rot & 2 ? a2 : a0, rot & 2 ? a3 : a1, rot & 2 ? a0 : a2, rot & 2 ? a1 : a3};
#pragma unroll
    for (int s = 0; s < 4; ++s) dst[place(col + ((s + rot) & 3)) * PT + row] = mul * w[s];
  }
}

// The same rows in natural order: dst[row][64].
__device__ __forceinline__ void load_rows(float* dst, const void* src, size_t base, int pitch, int row0, int N, int dt, bool vec, int tid) {
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int row = (tid >> 4) + 16 * x, col = 4 * (tid & 15);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (row0 + row < N) load_quad(src, base + (size_t)(row0 + row) * pitch + col, dt, vec, v);
    *reinterpret_cast<float4*>(dst + row * TP + col) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

struct Ident {
  __device__ __forceinline__ int operator()(int c) const { return c; }
};
struct ByGroup {
  const int* inv;
  __device__ __forceinline__ int operator()(int c) const { return inv[c]; }
};

template <int JP>
__device__ __forceinline__ void load_jp(const float* p, float (&o)[JP]) {
  if constexpr (JP == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
  } else if constexpr (JP == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    o[0] = t.x; o[1] = t.y;
  } else {
    o[0] = *p;
  }
}

// acc[r][m] += sum_e own[e][r] other[e][m] over 64 rows of two transposed tiles
template <int JP>
__device__ __forceinline__ void outer64(const float* own, const float* other, float (&acc)[4][JP]) {
#pragma unroll 4
  for (int e = 0; e < HD; ++e) {
    const float4 a = *reinterpret_cast<const float4*>(own + e * PT);
    float b[JP];
    load_jp<JP>(other + e * PT, b);
#pragma unroll
    for (int m = 0; m < JP; ++m) {
      acc[0][m] = fmaf(a.x, b[m], acc[0][m]);
      acc[1][m] = fmaf(a.y, b[m], acc[1][m]);
      acc[2][m] = fmaf(a.z, b[m], acc[2][m]);
      acc[3][m] = fmaf(a.w, b[m], acc[3][m]);
    }
  }
}

// s[g][r][m] = dot product of group g between owner token r and other token m
template <int GCAP, int JP>
__device__ __forceinline__ void group_scores(const HeadGroups& hg, const float* own, const float* other, float (&s)[GCAP][4][JP]) {
#pragma unroll
  for (int g = 0; g < GCAP; ++g) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int m = 0; m < JP; ++m) s[g][r][m] = 0.f;
    const int d1 = hg.start[g + 1];
#pragma unroll 4
    for (int d = hg.start[g]; d < d1; ++d) {
      const float4 a = *reinterpret_cast<const float4*>(own + d * PT);
      float b[JP];
      load_jp<JP>(other + d * PT, b);
#pragma unroll
      for (int m = 0; m < JP; ++m) {
        s[g][0][m] = fmaf(a.x, b[m], s[g][0][m]);
        s[g][1][m] = fmaf(a.y, b[m], s[g][1][m]);
        s[g][2][m] = fmaf(a.z, b[m], s[g][2][m]);
        s[g][3][m] = fmaf(a.w, b[m], s[g][3][m]);
      }
    }
  }
}

// acc[x] += sum over the pass's tokens of ds[group of the dimension][token][16 owner tokens] other[token]
// ds: first of the 16 owner tokens of the thread's group; other: the thread's dimension in a transposed tile
template <int SUB>
__device__ __forceinline__ void token_sums(const float* ds, const float* other, float (&acc)[16]) {
#pragma unroll 1
  for (int t = 0; t < SUB; t += 4) {
    const float4 o = *reinterpret_cast<const float4*>(other + t);
    const float ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float4 d = *reinterpret_cast<const float4*>(ds + (t + u) * TP + 4 * x);
        acc[4 * x + 0] = fmaf(d.x, ov[u], acc[4 * x + 0]);
        acc[4 * x + 1] = fmaf(d.y, ov[u], acc[4 * x + 1]);
        acc[4 * x + 2] = fmaf(d.z, ov[u], acc[4 * x + 2]);
        acc[4 * x + 3] = fmaf(d.w, ov[u], acc[4 * x + 3]);
      }
  }
}

// acc[r][c] += sum over `count` tokens of own[token][4] other[token][4], natural tiles of pitch 64
__device__ __forceinline__ void row_products(const float* own, const float* other, int count, float (&acc)[4][4]) {
#pragma unroll 4
  for (int t = 0; t < count; ++t) {
    const float4 a = *reinterpret_cast<const float4*>(own + t * TP), b = *reinterpret_cast<const float4*>(other + t * TP);
    const float ar[4] = {a.x, a.y, a.z, a.w}, br[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(ar[r], br[c], acc[r][c]);
  }
}

// Place of a block: `split` ranks (one cluster) of an owner tile of (batch row, query head).
struct PairBlock {
  int rank, tile, h, b;
  __device__ __forceinline__ PairBlock(const PairArgs& a, bool heavy_last) {
    const int heads = a.B * a.Hq;
    const int x = blockIdx.x;
    rank = x % a.split;
    const int rest = x / a.split, bh = rest % heads;
    tile = rest / heads;                                 // tiles with the longest walk are started first
    if (heavy_last) tile = (int)(gridDim.x / a.split) / heads - 1 - tile;
    h = bh % a.Hq;
    b = bh / a.Hq;
  }
};

// Sum over the ranks of a cluster of the value at the same place of their shared memory, in rank order.
__device__ __forceinline__ float sum_ranks(float* p, int split) {
  if (split == 1) return *p;
  cg::cluster_group c = cg::this_cluster();
  float t = 0.f;
  for (int r = 0; r < split; ++r) t += *c.map_shared_rank(p, r);
  return t;
}
__device__ __forceinline__ void sync_ranks(int split) {
  if (split == 1) __syncthreads();
  else cg::this_cluster().sync();
}

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------
template <int GCAP>
__global__ void __launch_bounds__(THREADS, 2) fwd_pairs_kernel(const PairArgs a) {
  using Cfg = PairCfg<GCAP, jp(GCAP)>;
  constexpr int JP = Cfg::JP;
  extern __shared__ __align__(16) float sm[];
  float* Qt = sm;                 // [64 d][68]  scaled, group order
  float* Kt = Qt + TT;            // [64 d][68]
  float* Us = Kt + TT;            // [64 j][64]
  float* WT = Us + TP * TP;       // [64 j][64 i]; at the end the sums [64 i][64]
  float* den_part = Us;           // at the end: [64 i][17]
  __shared__ HeadInfo<GCAP> hi;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const PairBlock pb(a, true);
  const int N = a.N, it = pb.tile, i0 = it * TP, kvh = pb.h / (a.Hq / a.Hkv);
  load_head<GCAP>(hi, a, pb.h, false, tid);
  const size_t qbase = (size_t)(pb.b * a.Hq + pb.h) * N * HD;
  const size_t kbase = (size_t)(pb.b * a.Hkv + kvh) * N * HD;
  load_transposed(Qt, a.q, qbase, HD, i0, N, a.io_dt, a.vec & 1, a.scale, ByGroup{hi.inv}, tid);

  const int ti = (warp & 1) * 8 + (lane & 7), tj = (warp >> 1) * 4 + (lane >> 3);
  float acc[4][4], den[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    den[r] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
  }
  for (int jt = pb.rank; jt <= it; jt += a.split) {
    const int j0 = jt * TP;
    load_transposed(Kt, a.k, kbase, HD, j0, N, a.io_dt, a.vec & 2, 1.f, ByGroup{hi.inv}, tid);
    load_rows(Us, a.v, kbase, HD, j0, N, a.io_dt, a.vec & 4, tid);
    __syncthreads();
#pragma unroll 1
    for (int j1 = JP * tj; j1 < TP; j1 += Cfg::SUB) {
      float s[GCAP][4][JP];
      group_scores<GCAP, JP>(hi.hg, Qt + 4 * ti, Kt + j1, s);
#pragma unroll
      for (int m = 0; m < JP; ++m) {
        float w[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) w[r] = hi.A;
#pragma unroll
        for (int g = 0; g < GCAP; ++g)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            float t = hi.B[g];
#pragma unroll
            for (int g2 = 0; g2 <= g; ++g2) t = fmaf(hi.C2[g * GCAP + g2], s[g2][r][m], t);
            w[r] = fmaf(s[g][r][m], t, w[r]);
          }
        const int gj = j0 + j1 + m;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int gi = i0 + 4 * ti + r;
          w[r] = (gj <= gi && gi < N) ? w[r] : 0.f;
          den[r] += w[r];
        }
        *reinterpret_cast<float4*>(WT + (j1 + m) * TP + 4 * ti) = make_float4(w[0], w[1], w[2], w[3]);
      }
    }
    __syncthreads();
    row_products(WT + 4 * ti, Us + 4 * tj, TP, acc);
    __syncthreads();
  }
  // sums and shares of the denominator to shared memory; every rank of the cluster then finishes a share of the rows
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    *reinterpret_cast<float4*>(WT + (4 * ti + r) * TP + 4 * tj) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    den_part[(4 * ti + r) * 17 + tj] = den[r];
  }
  __syncthreads();
  if (tid < TP) {
    float t = 0.f;
#pragma unroll
    for (int x = 0; x < 16; ++x) t += den_part[tid * 17 + x];
    den_part[tid * 17 + 16] = t;
  }
  sync_ranks(a.split);
  int flags = 0;
  const int share = TP / a.split;
  for (int x = tid; x < share * 16; x += THREADS) {
    const int r = pb.rank * share + (x >> 4), c4 = (x & 15) * 4, i = i0 + r;
    if (i >= N) continue;
    const size_t row = (size_t)(pb.b * a.Hq + pb.h) * N + i;
    const float dsum = sum_ranks(den_part + r * 17 + 16, a.split);
    float nv[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) nv[c] = sum_ranks(WT + r * TP + c4 + c, a.split);
    if (a.vec & 8) *reinterpret_cast<float4*>(a.num + row * VD + c4) = make_float4(nv[0], nv[1], nv[2], nv[3]);
    const float dn = fmaxf(dsum, a.floor);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (!(a.vec & 8)) a.num[row * VD + c4 + c] = nv[c];
      if (!finite_f(nv[c])) flags |= OAL_STATUS_NONFINITE;
      store_elem(a.out, row * VD + c4 + c, a.out_dt, nv[c] / dn);
    }
    if (c4 == 0) {
      a.den[row] = dsum;
      if (!finite_f(dsum)) flags |= OAL_STATUS_NONFINITE;
      else if (!(dsum > 0.f)) flags |= OAL_STATUS_DENOMINATOR;
    }
  }
  if (flags) atomicOr(a.status, flags);
  sync_ranks(a.split);      // no rank leaves while another one still reads its sums
  if (tid == 0) sink_status(a.status, a.sink);
}

// ---------------------------------------------------------------------------
// backward, query side: dq and the coefficient partial sums
// ---------------------------------------------------------------------------
template <int GCAP>
__device__ __forceinline__ void block_reduce_coefs(float cA, const float (&cB)[GCAP],
                                                   const float (&cC)[GCAP * (GCAP + 1) / 2],
                                                   float* red /* [8][NCOEF] smem */, float* dst,
                                                   int tid) {
  const int warp = tid >> 5, lane = tid & 31;
  auto wsum = [](float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  for (int x = lane; x < NCOEF; x += 32) red[warp * NCOEF + x] = 0.f;
  __syncwarp();
  float v = wsum(cA);
  if (lane == 0) red[warp * NCOEF + 0] = v;
#pragma unroll
  for (int g = 0; g < GCAP; ++g) {
    v = wsum(cB[g]);
    if (lane == 0) red[warp * NCOEF + 1 + g] = v;
  }
  int idx = 0;
#pragma unroll
  for (int g = 0; g < GCAP; ++g)
#pragma unroll
    for (int g2 = g; g2 < GCAP; ++g2) {
      v = wsum(cC[idx]);
      if (lane == 0) red[warp * NCOEF + 1 + GMAX + tri_index(g, g2)] = v;
      ++idx;
    }
  __syncthreads();
  for (int x = tid; x < NCOEF; x += THREADS) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[w * NCOEF + x];
    dst[x] = t;
  }
}

template <int GCAP>
__global__ void __launch_bounds__(THREADS, 1) bwd_q_pairs_kernel(const PairArgs a) {
  using Cfg = PairCfg<GCAP, jp_q(GCAP)>;
  constexpr int JP = Cfg::JP, SUB = Cfg::SUB, GS = Cfg::GS;
  extern __shared__ __align__(16) float sm[];
  float* Qt = sm;                     // [64 d][68]  scaled, group order; at the end the sums [64 i][64 d]
  float* Kt = Qt + TT;                // [64 d][68]
  float* gT = Kt + TT;                // [64 e][68 i]
  float* UT = gT + TT;                // [64 e][68 j]
  float* gden = UT + TT;              // [64 i] gradient of the denominator
  float* DS = gden + TP;              // [GCAP][SUB j][64 i] (also reduction scratch at the end)
  __shared__ HeadInfo<GCAP> hi;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const PairBlock pb(a, true);
  const int N = a.N, it = pb.tile, i0 = it * TP, kvh = pb.h / (a.Hq / a.Hkv);
  load_head<GCAP>(hi, a, pb.h, true, tid);
  const size_t qbase = (size_t)(pb.b * a.Hq + pb.h) * N * HD;
  const size_t kbase = (size_t)(pb.b * a.Hkv + kvh) * N * HD;
  const size_t gbase = (size_t)(pb.b * a.Hq + pb.h) * N * EP;
  load_transposed(Qt, a.q, qbase, HD, i0, N, a.io_dt, a.vec & 1, a.scale, ByGroup{hi.inv}, tid);
  load_transposed(gT, a.g, gbase, EP, i0, N, OAL_DTYPE_F32, true, 1.f, Ident{}, tid);
  if (tid < TP) gden[tid] = i0 + tid < N ? a.g[gbase + (size_t)(i0 + tid) * EP + VD] : 0.f;

  const int ti = (warp & 1) * 8 + (lane & 7), tj = (warp >> 1) * 4 + (lane >> 3);
  const int pd = (warp & 1) * 32 + lane, ib = (warp >> 1) * 16;       // dimension and owner tokens in the dq sums
  const float* ds_own = DS + hi.hg.group_of[pd] * GS + ib;
  float acc[16];
#pragma unroll
  for (int x = 0; x < 16; ++x) acc[x] = 0.f;
  float cA = 0.f, cB[GCAP], cC[GCAP * (GCAP + 1) / 2];
#pragma unroll
  for (int g = 0; g < GCAP; ++g) cB[g] = 0.f;
#pragma unroll
  for (int x = 0; x < GCAP * (GCAP + 1) / 2; ++x) cC[x] = 0.f;

  for (int jt = pb.rank; jt <= it; jt += a.split) {
    const int j0 = jt * TP;
    load_transposed(Kt, a.k, kbase, HD, j0, N, a.io_dt, a.vec & 2, 1.f, ByGroup{hi.inv}, tid);
    load_transposed(UT, a.v, kbase, HD, j0, N, a.io_dt, a.vec & 4, 1.f, Ident{}, tid);
    __syncthreads();
#pragma unroll 1
    for (int js = 0; js < TP; js += SUB) {
      {
        const int j1 = js + JP * tj;
        float dw[4][JP];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int m = 0; m < JP; ++m) dw[r][m] = gden[4 * ti + r];
        outer64<JP>(gT + 4 * ti, UT + j1, dw);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int m = 0; m < JP; ++m) {
            const int gi = i0 + 4 * ti + r, gj = j0 + j1 + m;
            dw[r][m] = (gj <= gi && gi < N) ? dw[r][m] : 0.f;
            cA += dw[r][m];
          }
        float s[GCAP][4][JP];
        group_scores<GCAP, JP>(hi.hg, Qt + 4 * ti, Kt + j1, s);
        int idx = 0;
#pragma unroll
        for (int g = 0; g < GCAP; ++g) {
          float t[4][JP];
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int m = 0; m < JP; ++m) t[r][m] = hi.B[g];
#pragma unroll
          for (int g2 = 0; g2 < GCAP; ++g2) {
            const float c = hi.C2[g * GCAP + g2];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
              for (int m = 0; m < JP; ++m) t[r][m] = fmaf(c, s[g2][r][m], t[r][m]);
          }
#pragma unroll
          for (int m = 0; m < JP; ++m)
            *reinterpret_cast<float4*>(DS + g * GS + (JP * tj + m) * TP + 4 * ti) =
                make_float4(dw[0][m] * t[0][m], dw[1][m] * t[1][m], dw[2][m] * t[2][m], dw[3][m] * t[3][m]);
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int m = 0; m < JP; ++m) {
              t[r][m] = dw[r][m] * s[g][r][m];
              cB[g] += t[r][m];
            }
#pragma unroll
          for (int g2 = g; g2 < GCAP; ++g2) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
              for (int m = 0; m < JP; ++m) cC[idx] = fmaf(t[r][m], s[g2][r][m], cC[idx]);
            ++idx;
          }
        }
      }
      __syncthreads();
      // dq~[i][p] += sum_j ds_{g(p)}(i,j) k[j][p]
      token_sums<SUB>(ds_own, Kt + pd * PT + js, acc);
      __syncthreads();
    }
  }
  __syncthreads();      // a rank without tiles comes here straight from its loads
  if (a.dq) {
    float* sums = Qt;
#pragma unroll
    for (int x = 0; x < 16; ++x) sums[(ib + x) * TP + pd] = acc[x];
    sync_ranks(a.split);
    const int share = TP / a.split;
    for (int x = tid; x < share * HD; x += THREADS) {
      const int r = pb.rank * share + (x >> 6), d = x & 63, i = i0 + r;
      if (i >= N) continue;
      store_elem(a.dq, qbase + (size_t)i * HD + d, a.io_dt, a.scale * sum_ranks(sums + r * TP + hi.inv[d], a.split));
    }
    sync_ranks(a.split);
  }
  if (a.coef_partial) {
    float* dst = a.coef_partial + ((size_t)((pb.b * a.Hq + pb.h) * a.tiles + it) * a.split + pb.rank) * NCOEF;
    block_reduce_coefs<GCAP>(cA, cB, cC, DS, dst, tid);
  }
}

// ---------------------------------------------------------------------------
// backward, key/value side: dk and dv of one query head, to the gradients themselves where a KV head has one query
// head, else to fp32 shares that head_sum_kernel adds up
// ---------------------------------------------------------------------------
template <int GCAP>
__global__ void __launch_bounds__(THREADS, 1) bwd_kv_pairs_kernel(const PairArgs a) {
  using Cfg = PairCfg<GCAP, jp(GCAP)>;
  constexpr int IP = Cfg::JP, SUB = Cfg::SUB, GS = Cfg::GS;
  extern __shared__ __align__(16) float sm[];
  float* Kt = sm;                     // [64 d][68]  group order; at the end the sums of dk [64 j][64 d]
  float* Qt = Kt + TT;                // [64 d][68]  scaled; at the end the sums of dv [64 j][64 e]
  float* UT = Qt + TT;                // [64 e][68 j]
  float* gT = UT + TT;                // [64 e][68 i]
  float* gs = gT + TT;                // [64 i][64 e]
  float* gden = gs + TP * TP;         // [64 i]
  float* Ws = gden + TP;              // [SUB i][64 j]
  float* DS = Ws + SUB * TP;          // [GCAP][SUB i][64 j]
  __shared__ HeadInfo<GCAP> hi;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const PairBlock pb(a, false);
  const int rep = a.Hq / a.Hkv, kvh = pb.h / rep;
  const int N = a.N, j0 = pb.tile * TP;
  load_head<GCAP>(hi, a, pb.h, true, tid);
  const size_t kbase = (size_t)(pb.b * a.Hkv + kvh) * N * HD;
  const size_t qbase = (size_t)(pb.b * a.Hq + pb.h) * N * HD;
  const size_t gbase = (size_t)(pb.b * a.Hq + pb.h) * N * EP;
  load_transposed(Kt, a.k, kbase, HD, j0, N, a.io_dt, a.vec & 2, 1.f, ByGroup{hi.inv}, tid);
  load_transposed(UT, a.v, kbase, HD, j0, N, a.io_dt, a.vec & 4, 1.f, Ident{}, tid);

  const int tj = (warp & 1) * 8 + (lane & 7), ti = (warp >> 1) * 4 + (lane >> 3);
  const int pd = (warp & 1) * 32 + lane, jb = (warp >> 1) * 16;
  const float* ds_own = DS + hi.hg.group_of[pd] * GS + jb;
  float adk[16], adv[4][4];
#pragma unroll
  for (int x = 0; x < 16; ++x) adk[x] = 0.f;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) adv[r][c] = 0.f;

  for (int it = pb.tile + pb.rank; it < a.tiles; it += a.split) {
    const int i0 = it * TP;
    load_transposed(Qt, a.q, qbase, HD, i0, N, a.io_dt, a.vec & 1, a.scale, ByGroup{hi.inv}, tid);
    load_transposed(gT, a.g, gbase, EP, i0, N, OAL_DTYPE_F32, true, 1.f, Ident{}, tid);
    load_rows(gs, a.g, gbase, EP, i0, N, OAL_DTYPE_F32, true, tid);
    if (tid < TP) gden[tid] = i0 + tid < N ? a.g[gbase + (size_t)(i0 + tid) * EP + VD] : 0.f;
    __syncthreads();
#pragma unroll 1
    for (int is = 0; is < TP; is += SUB) {
      {
        const int i1 = is + IP * ti;
        float dw[4][IP];
#pragma unroll
        for (int m = 0; m < IP; ++m)
#pragma unroll
          for (int r = 0; r < 4; ++r) dw[r][m] = gden[i1 + m];
        outer64<IP>(UT + 4 * tj, gT + i1, dw);
        float s[GCAP][4][IP], w[4][IP];
        group_scores<GCAP, IP>(hi.hg, Kt + 4 * tj, Qt + i1, s);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int m = 0; m < IP; ++m) {
            const int gi = i0 + i1 + m, gj = j0 + 4 * tj + r;
            dw[r][m] = (gj <= gi && gi < N) ? dw[r][m] : 0.f;
            w[r][m] = 0.f;
          }
#pragma unroll
        for (int g = 0; g < GCAP; ++g) {
          float t[4][IP];
          const float bg = hi.B[g];
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int m = 0; m < IP; ++m) t[r][m] = bg;
#pragma unroll
          for (int g2 = 0; g2 < GCAP; ++g2) {
            const float c = hi.C2[g * GCAP + g2];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
              for (int m = 0; m < IP; ++m) t[r][m] = fmaf(c, s[g2][r][m], t[r][m]);
          }
          // t = B_g + 2 sum C s: the weight takes s_g (B_g + t) / 2
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int m = 0; m < IP; ++m) w[r][m] = fmaf(s[g][r][m], bg + t[r][m], w[r][m]);
#pragma unroll
          for (int m = 0; m < IP; ++m)
            *reinterpret_cast<float4*>(DS + g * GS + (IP * ti + m) * TP + 4 * tj) =
                make_float4(dw[0][m] * t[0][m], dw[1][m] * t[1][m], dw[2][m] * t[2][m], dw[3][m] * t[3][m]);
        }
#pragma unroll
        for (int m = 0; m < IP; ++m) {
          float wm[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int gi = i0 + i1 + m, gj = j0 + 4 * tj + r;
            wm[r] = (gj <= gi && gi < N) ? fmaf(0.5f, w[r][m], hi.A) : 0.f;
          }
          *reinterpret_cast<float4*>(Ws + (IP * ti + m) * TP + 4 * tj) = make_float4(wm[0], wm[1], wm[2], wm[3]);
        }
      }
      __syncthreads();
      token_sums<SUB>(ds_own, Qt + pd * PT + is, adk);
      row_products(Ws + 4 * tj, gs + is * TP + 4 * ti, SUB, adv);
      __syncthreads();
    }
  }
  __syncthreads();      // a rank without tiles comes here straight from its loads
  float *sdk = Kt, *sdv = Qt;
#pragma unroll
  for (int x = 0; x < 16; ++x) sdk[(jb + x) * TP + pd] = adk[x];
#pragma unroll
  for (int r = 0; r < 4; ++r)
    *reinterpret_cast<float4*>(sdv + (4 * tj + r) * TP + 4 * ti) = make_float4(adv[r][0], adv[r][1], adv[r][2], adv[r][3]);
  sync_ranks(a.split);
  const int share = TP / a.split;
  for (int x = tid; x < share * HD; x += THREADS) {
    const int r = pb.rank * share + (x >> 6), d = x & 63, j = j0 + r;
    if (j >= N) continue;
    const float vk = sum_ranks(sdk + r * TP + hi.inv[d], a.split), vv = sum_ranks(sdv + r * TP + d, a.split);
    if (rep > 1) {
      a.dk_part[qbase + (size_t)j * HD + d] = vk;
      a.dv_part[qbase + (size_t)j * HD + d] = vv;
    } else {
      if (a.dk) store_elem(a.dk, kbase + (size_t)j * HD + d, a.io_dt, vk);
      if (a.dv) store_elem(a.dv, kbase + (size_t)j * HD + d, a.io_dt, vv);
    }
  }
  sync_ranks(a.split);
}

// dk (blockIdx.y = 0) and dv (1): sums of the query heads' shares in head order.
__global__ void __launch_bounds__(THREADS) head_sum_kernel(const PairArgs a) {
  const size_t row = (size_t)a.N * HD, total = (size_t)a.B * a.Hkv * row;
  const size_t x = (size_t)blockIdx.x * THREADS + threadIdx.x;
  void* out = blockIdx.y ? a.dv : a.dk;
  if (x >= total || !out) return;
  const int rep = a.Hq / a.Hkv;
  const float* src = (blockIdx.y ? a.dv_part : a.dk_part) + (x / row) * rep * row + x % row;
  float t = 0.f;
#pragma unroll 8
  for (int r = 0; r < rep; ++r) t += src[r * row];
  store_elem(out, x, a.io_dt, t);
}

// ---------------------------------------------------------------------------
// normalisation VJP: g_i = [dnum_i, dden_i]
//   den' = max(den, floor); dnum = dout/den' + grad_num;
//   dden = -(dout . num)/den'^2 [den >= floor] + grad_den
// (oal_attention/hd_block_gemm_backward.py:272-307)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) norm_vjp_kernel(const void* grad_out, int out_dt,
                                                       const float* grad_num, const float* grad_den,
                                                       const float* num, const float* den,
                                                       float floor_v, float* g, size_t rows, int32_t* clear_status) {
  if (clear_status && blockIdx.x == 0 && threadIdx.x == 0) *clear_status = 0;     // first kernel of the backward
  const size_t row = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float dn = den[row];
  const float dw = fmaxf(dn, floor_v);
  float gv[2] = {0.f, 0.f}, dot = 0.f;
  if (grad_out) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float go = load_elem(grad_out, row * VD + lane + 32 * c, out_dt);
      dot = fmaf(go, num[row * VD + lane + 32 * c], dot);
      gv[c] = go / dw;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (grad_num) gv[c] += grad_num[row * VD + lane + 32 * c];
    g[row * EP + lane + 32 * c] = gv[c];
  }
  if (lane < EP - VD) {
    float v = 0.f;
    if (lane == 0) {
      if (grad_out) v = (dn >= floor_v) ? -(dot / dw) / dw : 0.f;
      if (grad_den) v += grad_den[row];
    }
    g[row * EP + VD + lane] = v;
  }
}

// Fixed-order reduction of the per-tile coefficient partial sums.
//   partial [B][Hq][tiles][NCOEF]; extra [Hq][NCOEF] (already summed over the batch) or null
__global__ void reduce_coefs_kernel(const float* p0, int tiles0, const float* extra, int B, int Hq, int G,
                                    float* dA, float* dB, float* dC) {
  const int h = blockIdx.x;
  for (int x = threadIdx.x; x < 1 + G + G * G; x += blockDim.x) {
    int slot;
    if (x == 0) slot = 0;
    else if (x <= G) slot = x;            // 1 + g
    else {
      int g = (x - 1 - G) / G, g2 = (x - 1 - G) % G;
      slot = 1 + GMAX + (g <= g2 ? tri_index(g, g2) : tri_index(g2, g));
    }
    float t = extra ? extra[(size_t)h * NCOEF + slot] : 0.f;
    for (int b = 0; b < B; ++b)
      for (int i = 0; i < tiles0; ++i) t += p0[((size_t)(b * Hq + h) * tiles0 + i) * NCOEF + slot];
    if (x == 0) dA[h] = t;
    else if (x <= G) dB[h * G + x - 1] = t;
    else dC[(size_t)h * G * G + (x - 1 - G)] = t;
  }
}

template <int GCAP>
constexpr size_t fwd_smem() { return sizeof(float) * (2 * TT + 2 * TP * TP); }
template <int GCAP>
constexpr size_t bwd_q_smem() { return sizeof(float) * (4 * TT + TP + GCAP * PairCfg<GCAP, jp_q(GCAP)>::GS); }
template <int GCAP>
constexpr size_t bwd_kv_smem() {
  return sizeof(float) * (4 * TT + TP * TP + TP + PairCfg<GCAP, jp(GCAP)>::SUB * TP + GCAP * PairCfg<GCAP, jp(GCAP)>::GS);
}

// Launch with clusters of a.split CTAs.
template <auto Kernel>
cudaError_t launch_clusters(const PairArgs& a, size_t smem, cudaStream_t st) {
  cudaError_t e = allow_smem<Kernel>((int)smem);
  if (e != cudaSuccess) return e;
  const size_t blocks = (size_t)a.tiles * a.split * a.Hq * a.B;
  if (blocks > 0x7fffffffu) return cudaErrorInvalidConfiguration;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)a.split;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = a.split > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, Kernel, a);
}

template <int GCAP>
cudaError_t launch_pairs(const PairArgs& a, int which, cudaStream_t st) {
  if (which == 0) return launch_clusters<fwd_pairs_kernel<GCAP>>(a, fwd_smem<GCAP>(), st);
  if (which == 1) return launch_clusters<bwd_q_pairs_kernel<GCAP>>(a, bwd_q_smem<GCAP>(), st);
  return launch_clusters<bwd_kv_pairs_kernel<GCAP>>(a, bwd_kv_smem<GCAP>(), st);
}

cudaError_t dispatch_pairs(const PairArgs& args, int which, cudaStream_t st) {
  PairArgs a = args;
  const size_t quad = a.io_dt == OAL_DTYPE_F32 ? 16 : 8;      // bytes of four elements
  const void* in[3] = {a.q, a.k, a.v};
  a.vec = 0;
  for (int x = 0; x < 3; ++x) a.vec |= reinterpret_cast<uintptr_t>(in[x]) % quad == 0 ? 1 << x : 0;
  a.vec |= reinterpret_cast<uintptr_t>(a.num) % 16 == 0 ? 8 : 0;
  a.tiles = pairs_tiles(a.N);
  a.split = pairs_split(a.B, a.Hq, a.N);
  if (a.G <= 4) return launch_pairs<4>(a, which, st);
  if (a.G <= 8) return launch_pairs<8>(a, which, st);
  return launch_pairs<16>(a, which, st);
}

}  // namespace

cudaError_t pairs_forward(const PairArgs& a, cudaStream_t st) { return dispatch_pairs(a, 0, st); }
cudaError_t pairs_backward_q(const PairArgs& a, cudaStream_t st) { return dispatch_pairs(a, 1, st); }
cudaError_t pairs_backward_kv(const PairArgs& a, cudaStream_t st) {
  cudaError_t e = dispatch_pairs(a, 2, st);
  if (e != cudaSuccess || a.Hq == a.Hkv) return e;
  const size_t total = (size_t)a.B * a.Hkv * a.N * HD;
  head_sum_kernel<<<dim3((unsigned)((total + THREADS - 1) / THREADS), 2), THREADS, 0, st>>>(a);
  return cudaGetLastError();
}
int pairs_tiles(int n) { return (n + TP - 1) / TP; }
// CTAs that share an owner tile: doubled while the chip's SMs would not get two blocks each, up to the number of
// tiles there are to share and the portable cluster size.  The number of SMs is a constant here: workspace sizes follow
// the split, and they are asked for without a device too.
constexpr int B200_SMS = 148;
int pairs_split(int B, int Hq, int N) {
  const long long tiles = pairs_tiles(N), blocks = tiles * Hq * B;
  int s = 1;
  while (s < 8 && 2 * s <= tiles && blocks * s < 2 * B200_SMS) s *= 2;
  return s;
}

cudaError_t norm_vjp(const void* grad_out, int out_dt, const float* grad_num, const float* grad_den,
                     const float* num, const float* den, float floor_v, float* g, size_t rows,
                     int32_t* clear_status, cudaStream_t st) {
  norm_vjp_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(grad_out, out_dt, grad_num, grad_den, num,
                                                             den, floor_v, g, rows, clear_status);
  return cudaGetLastError();
}

cudaError_t reduce_coefs(const float* p0, int tiles0, const float* extra, int B, int Hq, int G,
                         float* dA, float* dB, float* dC, cudaStream_t st) {
  reduce_coefs_kernel<<<Hq, 128, 0, st>>>(p0, tiles0, extra, B, Hq, G, dA, dB, dC);
  return cudaGetLastError();
}

}  // namespace oal
