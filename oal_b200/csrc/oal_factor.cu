// Per-head factorisation of the kernel's quadratic form, and the way back for its gradient.
//
// head_factor_kernel: M = [[A, B/2], [B/2, C]] (symmetric, (G+1) x (G+1), any signature) is
// diagonalised by cyclic Jacobi rotations (fp32; the eigenvalues are re-evaluated as Rayleigh quotients
// of the untouched matrix), one warp per query head, the rotations of a round (disjoint index pairs of
// a round-robin tournament) applied together.  The result is stored as the
// table the intra-chunk kernels read (oal_intra.cuh): c_r, l_r[d], the back-transform t and the count of positive terms.  Replaces nothing in the reference, which evaluates the direct form
// (oal_attention/grouped_reference.py:61-99); the values of w are the same.
//
// intra_coef_finish_kernel: sums the per-(batch row, row block) partial sums of the query-side backward in
// fixed order, adds the cross-chunk coefficient gradient of the state kernels and writes dA, dB, dC
// (oal_attention/hd_block_gemm_feature_backward.py:59-131 coefficient partials).
#include "oal_intra.cuh"
#include "oal_kernels.h"
#include "oal_prologue.cuh"

namespace oal {
namespace {

constexpr int JN = RMAX_ALL;          // 17
constexpr int JP = JN + 1;            // row pitch
constexpr int JH = (JN + 1) / 2;      // index pairs per round (9)

// One warp per head.  Lane = (pair index i = lane & 15, row parity lane >> 4): the two lanes of a pair
// compute the same rotation from the untouched matrix and then update every other row (column) of
// the two columns (rows) of their pair, so no index arithmetic needs a division.
__global__ void __launch_bounds__(32) head_factor_kernel(const int32_t* dim_perm, const int32_t* group_start,
                                                         const float* A, const float* Bc, const float* Cc, int G,
                                                         float scale, HeadFactor* table) {
  __shared__ float M[JN][JP], V[JN][JP], M0[JN][JP];
  __shared__ int gdim[HD];
  __shared__ int order[JN];
  __shared__ float lam[JN], sig[JN];
  __shared__ int gstart[GMAX + 1];
  __shared__ float coefC[GMAX * GMAX], coefB[GMAX];
  const int h = blockIdx.x, lane = threadIdx.x;
  const int n = G + 1;
  // one coalesced pass over the head's tables (the loops below would otherwise chain global latencies)
  if (lane <= GMAX) gstart[lane] = group_start[h * (GMAX + 1) + lane];
  if (lane < G) coefB[lane] = Bc[h * G + lane];
  for (int x = lane; x < G * G; x += 32) coefC[x] = Cc[(size_t)h * G * G + x];
  const float coefA = A[h];
  const int perm0 = dim_perm[h * HD + lane], perm1 = dim_perm[h * HD + lane + 32];
  __syncwarp();
  for (int half_i = 0; half_i < 2; ++half_i) {
    const int p = lane + 32 * half_i;
    int g = 0;
    while (g < GMAX - 1 && p >= gstart[g + 1]) ++g;
    gdim[half_i ? perm1 : perm0] = min(g, G - 1);
  }
  if (lane < n) {
    const int a = lane;
    for (int b = 0; b < n; ++b) {
      float v;
      if (a == 0 && b == 0) v = coefA;
      else if (a == 0) v = 0.5f * coefB[b - 1];
      else if (b == 0) v = 0.5f * coefB[a - 1];
      else v = 0.5f * (coefC[(a - 1) * G + b - 1] + coefC[(b - 1) * G + a - 1]);
      M[a][b] = v;
      M0[a][b] = v;
      V[a][b] = a == b ? 1.f : 0.f;
    }
  }
  __syncwarp();
  const int m = (n & 1) ? n + 1 : n;          // players of the tournament; index n (if any) is a bye
  const int half = m / 2;
  const int pi = lane & 15, lg = lane >> 4;
  for (int sweep = 0; sweep < 12; ++sweep) {
    float off = 0.f, all = 0.f;
    if (lane < n)
      for (int b = 0; b < n; ++b) {
        const float v = M[lane][b];
        all = fmaf(v, v, all);
        if (b != lane) off = fmaf(v, v, off);
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (off <= 1e-11f * all) break;     // off-diagonal norm below 3e-6 of the whole: the Rayleigh quotients finish the job
    for (int t = 0; t < m - 1; ++t) {
      int p = 0, q = -1;
      float c = 1.f, s = 0.f;
      if (pi < half) {
        if (pi == 0) { p = m - 1; q = t; }
        else { p = t + pi; if (p >= m - 1) p -= m - 1; q = t - pi; if (q < 0) q += m - 1; }
        if (p > q) { const int x = p; p = q; q = x; }
        if (q < n) {
          const float apq = M[p][q];
          if (fabsf(apq) > 1e-30f) {
            const float tau = (M[q][q] - M[p][p]) / (2.f * apq);
            const float tt = (tau >= 0.f ? 1.f : -1.f) / (fabsf(tau) + sqrtf(1.f + tau * tau));
            c = rsqrtf(1.f + tt * tt);
            s = tt * c;
          }
        } else {
          q = -1;
        }
      }
      __syncwarp();
      // all loads of a phase are issued before its first store (the compiler cannot reorder them itself:
      // same array), so a phase costs one shared-memory latency instead of one per row
      if (q >= 0) {
        float xm[JH], ym[JH], xv[JH], yv[JH];
#pragma unroll
        for (int it = 0; it < JH; ++it) {           // columns p, q of M and V, rows l = lg, lg + 2, ...
          const int l = min(lg + 2 * it, n - 1);
          xm[it] = M[l][p]; ym[it] = M[l][q];
          xv[it] = V[l][p]; yv[it] = V[l][q];
        }
#pragma unroll
        for (int it = 0; it < JH; ++it) {
          const int l = lg + 2 * it;
          if (l < n) {
            M[l][p] = c * xm[it] - s * ym[it]; M[l][q] = s * xm[it] + c * ym[it];
            V[l][p] = c * xv[it] - s * yv[it]; V[l][q] = s * xv[it] + c * yv[it];
          }
        }
      }
      __syncwarp();
      if (q >= 0) {
        float xm[JH], ym[JH];
#pragma unroll
        for (int it = 0; it < JH; ++it) {           // rows p, q of M
          const int l = min(lg + 2 * it, n - 1);
          xm[it] = M[p][l]; ym[it] = M[q][l];
        }
#pragma unroll
        for (int it = 0; it < JH; ++it) {
          const int l = lg + 2 * it;
          if (l < n) { M[p][l] = c * xm[it] - s * ym[it]; M[q][l] = s * xm[it] + c * ym[it]; }
        }
      }
      __syncwarp();
    }
  }
  // eigenvalues as Rayleigh quotients of the untouched matrix (second-order accurate in the
  // remaining rotation error)
  if (lane < n) {
    float acc = 0.f;
    for (int a = 0; a < n; ++a) {
      float row = 0.f;
      for (int b = 0; b < n; ++b) row = fmaf(M0[a][b], V[b][lane], row);
      acc = fmaf(V[a][lane], row, acc);
    }
    sig[lane] = acc;
  }
  __syncwarp();
  // order: positive eigenvalues first; lambda_r = sqrt(max(|sigma_r|, tiny relative floor))
  if (lane == 0) {
    float smax = 0.f;
    for (int r = 0; r < n; ++r) smax = fmaxf(smax, fabsf(sig[r]));
    const float floor_v = fmaxf(1e-12f * smax, 1e-30f);
    int k = 0;
    for (int r = 0; r < n; ++r) if (sig[r] >= 0.f) order[k++] = r;
    const int rpos = k;
    for (int r = 0; r < n; ++r) if (!(sig[r] >= 0.f)) order[k++] = r;      // negative or not a number: all n entries are indices
    for (int r = 0; r < n; ++r) {
      const float size = fabsf(sig[order[r]]);
      lam[r] = sqrtf(size < floor_v ? floor_v : size);                     // a NaN stays one and reaches the status word
    }
    table[h].s.rank = n;
    table[h].s.rpos = rpos;
    table[h].s.w0 = 0.f;
  }
  __syncwarp();
  HeadFactor& out = table[h];
  write_head_groups(out.e, out.mask, out.order, gdim, dim_perm + h * HD, group_start + h * (GMAX + 1), G, scale,
                    [&](int g) { return coefB[g]; }, [&](int g, int g2) { return coefC[g * G + g2] + coefC[g2 * G + g]; }, lane, 32);
  if (lane < RMAX_ALL) out.s.c[lane] = lane < n ? lam[lane] * V[0][order[lane]] : 0.f;
  for (int r = 0; r < RMAX_ALL; ++r) {
    const bool live = r < n;
    const float sl = live ? scale * lam[r] : 0.f;
    const int col = live ? order[r] : 0;
    out.l[r][lane] = live ? sl * V[1 + gdim[lane]][col] : 0.f;
    out.l[r][lane + 32] = live ? sl * V[1 + gdim[lane + 32]][col] : 0.f;
    if (lane < RMAX_ALL) out.t[lane][r] = (live && lane < n) ? V[lane][col] / lam[r] : 0.f;
  }
}

__device__ __forceinline__ int tri_all(int g, int g2) { return g * GMAX - (g * (g - 1)) / 2 + (g2 - g); }

// The prologue on its own: on a side stream, or for calls without row images (rows_prologue_kernel shares its launch with it).
__global__ void __launch_bounds__(256) head_prologue_kernel(const PrologueArgs a) {
  __shared__ PrologueSmem s;
  head_prologue(a, blockIdx.x, s, threadIdx.x, 256);
}

__global__ void deliver_status_kernel(const int32_t* status, StatusSink sink) {
  *sink.host = *status | STATUS_DELIVERED;
  __threadfence_system();
}

// partial: [B][Hq][tiles][1 + G + G (G + 1) / 2]: dA, dB, upper triangle of dC in row-major order.  One block per head;
// FINISH_SEGS threads share the tiles of a sum (a serial walk over 512 tiles is 60 us of dependent loads), their parts are
// added in fixed order.  With `factor` the block goes on from dM to the gradient of its own packed factor row:
// dL = (S + S^T) L, see expand_factor_grad_kernel.
constexpr int FINISH_THREADS = 1024, FINISH_SEGS = 16, FINISH_SUMS = 1 + GMAX + GMAX * (GMAX + 1) / 2;
__global__ void __launch_bounds__(FINISH_THREADS) intra_coef_finish_kernel(const float* partial, int tiles, const float* extra, int B,
                                                                int Hq, int G, float* dA, float* dB, float* dC,
                                                                const float* factor, float* dfactor) {
  __shared__ float S[RMAX_ALL][RMAX_ALL];       // S[0][0] = dA, S[0][b] = 2 dB, S[a][0] = 0, S[a][b] = dC
  __shared__ float seg_sum[FINISH_SEGS][FINISH_SUMS];
  const int h = blockIdx.x, tid = threadIdx.x;
  const int n = G + 1, nv = 1 + G + G * (G + 1) / 2;
  const int outer = B * tiles, per = (outer + FINISH_SEGS - 1) / FINISH_SEGS;
  for (int x = tid; x < nv * FINISH_SEGS; x += FINISH_THREADS) {
    const int v = x % nv, seg = x / nv, o0 = seg * per, o1 = min(outer, o0 + per);
    float t = 0.f;
#pragma unroll 8
    for (int o = o0; o < o1; ++o) {
      const int b = o / tiles, i = o - b * tiles;
      t += partial[((size_t)(b * Hq + h) * tiles + i) * nv + v];
    }
    seg_sum[seg][v] = t;
  }
  __syncthreads();
  for (int v = tid; v < nv; v += FINISH_THREADS) {
    float t = 0.f;
#pragma unroll
    for (int seg = 0; seg < FINISH_SEGS; ++seg) t += seg_sum[seg][v];
    if (v <= G) {
      if (extra) t += extra[(size_t)h * NCOEF + v];
      if (v == 0) dA[h] = t;
      else dB[h * G + v - 1] = t;
      S[0][v] = v ? 2.f * t : t;
      if (v) S[v][0] = 0.f;
    } else {
      int g = 0, rest = v - 1 - G;
      while (rest >= G - g) { rest -= G - g; ++g; }
      const int g2 = g + rest;
      if (extra) t += extra[(size_t)h * NCOEF + 1 + GMAX + tri_all(g, g2)];
      dC[((size_t)h * G + g) * G + g2] = dC[((size_t)h * G + g2) * G + g] = t;
      S[1 + g][1 + g2] = S[1 + g2][1 + g] = t;
    }
  }
  if (!factor) return;
  __syncthreads();
  const int P = n * (n + 1) / 2;
  for (int x = tid; x < P; x += FINISH_THREADS) {
    int i = 0, rest = x;
    while (rest > i) { rest -= i + 1; ++i; }
    const int k = rest;
    float t = 0.f;
    for (int j = k; j < n; ++j) t = fmaf(S[i][j] + S[j][i], factor[(size_t)h * P + j * (j + 1) / 2 + k], t);
    dfactor[(size_t)h * P + x] = t;
  }
}


// ---------------------------------------------------------------------------
// Packed factor -> coefficients and back.  L is the lower-triangular matrix whose packed rows
// (row-major over (row, col <= row), the order of torch.tril_indices) are `factor`; M = L L^T;
// A = M00 + eps, B = 2 M[0, 1:], C = M[1:, 1:].  One block per query head, thread = (i, j).
// Replaces the tensor-op sequence of oal_attention/grouped_quadratic.py (_expand_factor_coefficients there)
// and its autograd graph: two launches per step instead of about forty.
// ---------------------------------------------------------------------------
constexpr int XS = GMAX + 1;     // largest side of L

__device__ __forceinline__ float packed_l(const float* f, int r, int c) { return c <= r ? f[r * (r + 1) / 2 + c] : 0.f; }

__global__ void __launch_bounds__(XS * XS) expand_factor_kernel(const float* factor, int factor_rows, int G, float eps,
                                                                float* A, float* B, float* C) {
  const int h = blockIdx.x, side = G + 1;
  const float* f = factor + (size_t)(factor_rows == 1 ? 0 : h) * (side * (side + 1) / 2);
  const int i = threadIdx.x / side, j = threadIdx.x % side;
  if (i >= side) return;
  float m = 0.f;
  for (int k = 0; k <= min(i, j); ++k) m = fmaf(packed_l(f, i, k), packed_l(f, j, k), m);
  if (i == 0 && j == 0) A[h] = m + eps;
  else if (i == 0) B[(size_t)h * G + j - 1] = 2.f * m;
  else if (j > 0) C[((size_t)h * G + i - 1) * G + j - 1] = m;
}

// dL = (S + S^T) L on the lower triangle, S[0][0] = dA, S[0][j] = 2 dB[j-1], S[i][j] = dC[i-1][j-1] (i, j >= 1),
// S[i][0] = 0.  With one shared factor row (factor_rows == 1) a single block walks the heads in order.
__global__ void __launch_bounds__(XS * XS) expand_factor_grad_kernel(const float* factor, int factor_rows, int Hq, int G,
                                                                     const float* dA, const float* dB, const float* dC,
                                                                     float* dfactor) {
  const int side = G + 1, P = side * (side + 1) / 2;
  const int i = threadIdx.x / side, k = threadIdx.x % side;
  const bool mine = i < side && k <= i;
  const int h0 = factor_rows == 1 ? 0 : blockIdx.x, h1 = factor_rows == 1 ? Hq : h0 + 1;
  const float* f = factor + (size_t)(factor_rows == 1 ? 0 : h0) * P;
  float acc = 0.f;
  for (int h = h0; h < h1 && mine; ++h) {
    auto S = [&](int r, int c) -> float {
      if (r == 0) return c == 0 ? dA[h] : 2.f * dB[(size_t)h * G + c - 1];
      return c == 0 ? 0.f : dC[((size_t)h * G + r - 1) * G + c - 1];
    };
    for (int j = k; j < side; ++j) acc = fmaf(S(i, j) + S(j, i), packed_l(f, j, k), acc);
  }
  if (mine) dfactor[(size_t)(factor_rows == 1 ? 0 : h0) * P + i * (i + 1) / 2 + k] = acc;
}

}  // namespace

size_t head_factor_bytes(int Hq) { return (size_t)Hq * sizeof(HeadFactor); }

cudaError_t build_head_factors(const int32_t* dim_perm, const int32_t* group_start, const float* A, const float* Bc,
                               const float* Cc, int Hq, int G, float scale, void* table, cudaStream_t st) {
  head_factor_kernel<<<Hq, 32, 0, st>>>(dim_perm, group_start, A, Bc, Cc, G, scale, static_cast<HeadFactor*>(table));
  return cudaGetLastError();
}

cudaError_t launch_head_prologue(const PrologueArgs& a, int Hq, cudaStream_t st) {
  head_prologue_kernel<<<Hq, 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t deliver_status(const int32_t* status, StatusSink sink, cudaStream_t st) {
  deliver_status_kernel<<<1, 1, 0, st>>>(status, sink);
  return cudaGetLastError();
}

cudaError_t intra_coef_finish(const float* partial, int tiles, const float* extra, int B, int Hq, int G, float* dA, float* dB,
                              float* dC, const float* factor, float* dfactor, cudaStream_t st) {
  intra_coef_finish_kernel<<<Hq, FINISH_THREADS, 0, st>>>(partial, tiles, extra, B, Hq, G, dA, dB, dC, factor, dfactor);
  return cudaGetLastError();
}

cudaError_t expand_factor(const float* factor, int factor_rows, int Hq, int G, float eps, float* A, float* B, float* C,
                          cudaStream_t st) {
  expand_factor_kernel<<<Hq, (GMAX + 1) * (GMAX + 1), 0, st>>>(factor, factor_rows, G, eps, A, B, C);
  return cudaGetLastError();
}

cudaError_t expand_factor_grad(const float* factor, int factor_rows, int Hq, int G, const float* dA, const float* dB,
                               const float* dC, float* dfactor, cudaStream_t st) {
  expand_factor_grad_kernel<<<factor_rows == 1 ? 1 : Hq, (GMAX + 1) * (GMAX + 1), 0, st>>>(factor, factor_rows, Hq, G, dA,
                                                                                           dB, dC, dfactor);
  return cudaGetLastError();
}

}  // namespace oal
