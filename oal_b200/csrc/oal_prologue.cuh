// Per-head prologue of a forward call, one block per query head, in one launch or in two (coefficients and their table
// beside the row images' blocks, the factor table on a side stream): packed factor row L (lower triangular,
// M = L L^T + eps e0 e0^T) -> coefficients A, B, C, the coefficient table of the state kernels and the
// factor table of the intra-chunk kernels.
//
// The eigenvectors of L L^T come from one-sided Jacobi rotations of the columns of L^T: with Y = L^T J
// orthogonal by columns, J holds the eigenvectors V and the column norms are lambda_r = sqrt(sigma_r).
// One warp holds a column of Y and a column of J per lane, in registers; a round of the round-robin
// tournament is 2 n shuffles and 7 n multiply-adds, so the whole factorisation is one short register
// chain (the two-sided rotations of the matrix in shared memory, which explicit and possibly indefinite
// A, B, C still take, need 50 us at n = 9).  eps never enters the rotations: it is added to every pair
// weight as the constant w0.
#pragma once

#include "oal_intra.cuh"

namespace oal {

struct PrologueArgs {
  const float* factor;               // [factor_rows (1 or Hq), (G+1)(G+2)/2]
  int factor_rows, G;
  float eps, scale;
  const int32_t *dim_perm, *group_start;
  float *A, *B, *C;                  // outputs [Hq], [Hq,G], [Hq,G,G], or all null
  float* coef_table;                 // output [Hq, F_ROWS], or null (no state kernels follow)
  HeadFactor* factors;               // output, or null (no tensor-core intra-chunk kernels follow)
  int32_t *status, *counter;         // cleared by block 0 (each may be null)
};

struct PrologueSmem {
  float L[RMAX_ALL][RMAX_ALL + 1];   // lower triangle, zero above
  float M[RMAX_ALL][RMAX_ALL + 1];   // L L^T (without eps)
  float V[RMAX_ALL][RMAX_ALL + 1];   // V[a][r]
  float lam[RMAX_ALL + 3];
  int gdim[HD];
};

// Eigenvectors (columns of V) and lambda of L L^T by one warp; NM >= n is the register extent.
template <int NM>
__device__ __forceinline__ void one_sided_jacobi(PrologueSmem& s, int n, int lane) {
  float y[NM], v[NM];
#pragma unroll
  for (int i = 0; i < NM; ++i) {
    y[i] = (lane < n && i < n) ? s.L[lane][i] : 0.f;        // column `lane` of L^T = row `lane` of L
    v[i] = (lane < n && i == lane) ? 1.f : 0.f;
  }
  const int m = (n + 1) & ~1;                                // players; an odd n gets a zero column as bye
  for (int sweep = 0; sweep < 14; ++sweep) {
    bool rotated = false;
    for (int t = 0; t < m - 1; ++t) {
      int q = lane;
      if (lane < m - 1) {
        q = 2 * t - lane;
        if (q < 0) q += m - 1;
        if (q >= m - 1) q -= m - 1;
        if (q == lane) q = m - 1;
      } else if (lane == m - 1) {
        q = t;
      }
      float z[NM], own = 0.f, other = 0.f, cross = 0.f;
#pragma unroll
      for (int i = 0; i < NM; ++i) z[i] = __shfl_sync(0xffffffffu, y[i], q);
#pragma unroll
      for (int i = 0; i < NM; ++i) {
        own = fmaf(y[i], y[i], own);
        other = fmaf(z[i], z[i], other);
        cross = fmaf(y[i], z[i], cross);
      }
      const bool low = lane < q;
      const float alpha = low ? own : other, beta = low ? other : own;
      float c = 1.f, sn = 0.f;
      // columns orthogonal to fp32 precision (or zero) are left alone; both lanes of a pair see the same numbers
      const bool turn = cross * cross > 1e-12f * alpha * beta && fabsf(cross) > 1e-36f;
      if (turn) {
        const float zeta = (beta - alpha) / (2.f * cross);
        const float tt = (zeta >= 0.f ? 1.f : -1.f) / (fabsf(zeta) + sqrtf(fmaf(zeta, zeta, 1.f)));
        c = rsqrtf(fmaf(tt, tt, 1.f));
        sn = tt * c;
        if (low) sn = -sn;                                   // low column: c x - s y; high column: s x + c y
      }
      rotated |= turn;
#pragma unroll
      for (int i = 0; i < NM; ++i) y[i] = fmaf(c, y[i], sn * z[i]);
#pragma unroll
      for (int i = 0; i < NM; ++i) {
        const float w = __shfl_sync(0xffffffffu, v[i], q);
        v[i] = fmaf(c, v[i], sn * w);
      }
    }
    if (!__any_sync(0xffffffffu, rotated)) break;
  }
  float norm = 0.f;
#pragma unroll
  for (int i = 0; i < NM; ++i) norm = fmaf(y[i], y[i], norm);
  float top = norm;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  if (lane < n) {
    // a vanishing term keeps its direction at a negligible weight, so that the coefficient gradient of a
    // singular factor can be rotated back; a NaN (which fmaxf would drop) stays one and reaches weights and status
    const float least = fmaxf(1e-12f * top, 1e-30f);
    s.lam[lane] = sqrtf(norm < least ? least : norm);
#pragma unroll
    for (int i = 0; i < NM; ++i)
      if (i < n) s.V[i][lane] = v[i];
  }
}

// Its own function: inlined beside the group tables the rotations of 17 columns took 59.1 us, alone 56.6 (of 9 columns 21.8 inlined,
// 22.6 alone).
static __device__ __noinline__ void one_sided_jacobi_wide(PrologueSmem& s, int n, int lane) { one_sided_jacobi<RMAX_ALL>(s, n, lane); }

// All threads of the block; blockDim.x a multiple of 32, at least 64.
__device__ __forceinline__ void head_prologue(const PrologueArgs& a, int h, PrologueSmem& s, int tid, int nthreads) {
  const int n = a.G + 1;
  const float* f = a.factor + (size_t)(a.factor_rows == 1 ? 0 : h) * (n * (n + 1) / 2);
  if (h == 0 && tid == 0) {
    if (a.status) *a.status = 0;
    if (a.counter) *a.counter = 0;
  }
  for (int x = tid; x < RMAX_ALL * RMAX_ALL; x += nthreads) {
    const int r = x / RMAX_ALL, c = x % RMAX_ALL;
    s.L[r][c] = (r < n && c <= r) ? f[r * (r + 1) / 2 + c] : 0.f;
  }
  if (tid < HD) {
    const int32_t* gs = a.group_start + h * (GMAX + 1);
    int g = 0;
    while (g < GMAX - 1 && tid >= gs[g + 1]) ++g;
    s.gdim[a.dim_perm[h * HD + tid]] = min(g, a.G - 1);
  }
  __syncthreads();
  for (int x = tid; x < n * n; x += nthreads) {
    const int i = x / n, j = x % n;
    float m = 0.f;
    for (int k = 0; k <= min(i, j); ++k) m = fmaf(s.L[i][k], s.L[j][k], m);
    s.M[i][j] = m;
    if (!a.A) continue;
    if (i == 0 && j == 0) a.A[h] = m + a.eps;
    else if (i == 0) a.B[(size_t)h * a.G + j - 1] = 2.f * m;
    else if (j > 0) a.C[((size_t)h * a.G + i - 1) * a.G + j - 1] = m;
  }
  __syncthreads();
  if (tid < 32) {
    if (a.factors) {
      if (n <= 9) one_sided_jacobi<9>(s, n, tid);
      else one_sided_jacobi_wide(s, n, tid);
    }
  } else {
    // beside the rotations, which the other warps would only wait for (after them: 22.2 instead of 21.8 us at 8 groups)
    if (a.factors) {
      HeadFactor& out = a.factors[h];
      const float (*M)[RMAX_ALL + 1] = s.M;
      write_head_groups(out.e, out.mask, out.order, s.gdim, a.dim_perm + h * HD, a.group_start + h * (GMAX + 1), a.G, a.scale,
                        [&](int g) { return 2.f * M[0][1 + g]; }, [&](int g, int g2) { return 2.f * M[1 + g][1 + g2]; }, tid - 32, nthreads - 32);
    }
    for (int fr = tid - 32; a.coef_table && fr < F_ROWS; fr += nthreads - 32) {
      float v = 0.f;
      const FeatureId id = feature_id(fr);
      if (id.kind == 0 && id.live) v = (id.r == id.c ? 1.f : 2.f) * s.M[1 + s.gdim[id.r]][1 + s.gdim[id.c]];
      else if (id.kind == 1) v = 2.f * s.M[0][1 + s.gdim[id.r]];
      else if (id.kind == 2) v = s.M[0][0] + a.eps;
      a.coef_table[(size_t)h * F_ROWS + fr] = v * feature_scale_factor(fr, a.scale);
    }
  }
  if (!a.factors) return;
  __syncthreads();
  HeadFactor& out = a.factors[h];
  for (int x = tid; x < RMAX_ALL * HD; x += nthreads) {
    const int r = x / HD, d = x % HD;
    out.l[r][d] = r < n ? a.scale * s.lam[r] * s.V[1 + s.gdim[d]][r] : 0.f;
  }
  for (int x = tid; x < RMAX_ALL * RMAX_ALL; x += nthreads) {
    const int i = x / RMAX_ALL, r = x % RMAX_ALL;
    if (i < n && r < n) out.t[i][r] = s.V[i][r] / s.lam[r];
  }
  if (tid < RMAX_ALL) out.s.c[tid] = tid < n ? s.lam[tid] * s.V[0][tid] : 0.f;
  if (tid == 0) {
    out.s.rank = n;
    out.s.rpos = n;
    out.s.w0 = a.eps;
  }
}

}  // namespace oal
