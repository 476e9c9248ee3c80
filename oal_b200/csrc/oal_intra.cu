// Intra-chunk term of the chunked scan on the tensor cores (tcgen05 / TMEM), forward.
//
// One CTA = one query tile (oal_intra.cuh: four blocks of 32 query rows that share a key / value chunk).  For every
// term r of the factored weight:
//   the compute warps scale their query rows by l_r into the A operand in tensor memory (two slots),
//   U_r = term . K^T     one MMA chain per half of the keys (64 columns each, so that one half is read
//                        while the other is computed),
//   w += sgn_r u_r^2     in registers, 64 keys per thread.
// Then the causal mask, the weight tile W into tensor memory (bf16 value + remainder), Y = W [v | 1] (one MMA chain), and the epilogue
// adds the cross-chunk part left in num / den by cross_read, normalises and writes out / num / den and the status
// flags.  Eight compute warps (quadrant x 2), one warp issues the MMAs; two CTAs share an SM.  Replaces, per chunk,
// the reference's F-wide local score GEMM, tril, bf16 cast, score x U GEMM, merge and normalise stages
// (oal_attention/hd_block_gemm_runtime.py:530-597, hd_block_gemm_normalization_ops.py:113).
//
// What bounds it: instruction latency and barriers, not the tensor pipe.  Over 448 tiles of 8 groups the issue slots are 37 %
// busy, the tensor pipe 12 %; a warp waits for the CTA's hand-over of terms (2.0 of 11 warp-cycles per instruction),
// tensor-memory loads (1.4) and fixed latencies (1.6).  B = 4, N = 4096, 8 groups: 146 -> 134 us.
#include "oal_intra.cuh"
#include "oal_kernels.h"

namespace oal {
namespace {

using namespace umma;

struct IntraFwdArgs {
  const __nv_bfloat16 *q, *k, *v;
  const HeadFactor* factors;
  void* out;
  float *num, *den;
  int32_t* status;
  int N, Hq, Hkv, rep, rank, out_dt;      // rank = groups + 1, the same for every head of a call
  float floor;
  int out_token_major;      // out is [B, N, Hq, 64] instead of [B, Hq, N, 64]
  int cross_from;           // first chunk that has a cross-chunk part in num / den
  StatusSink sink;
};

// Warps 0..7 compute, warp 8 issues; 9..11 only fill the issuer's warpgroup, whose registers the compute warps take:
// 384 threads x 80 at launch = 256 x 104 + 128 x 24 and 1024 to spare.
constexpr int FW_COMPUTE = 8, FW_ISSUER = FW_COMPUTE, FW_THREADS = (FW_COMPUTE + 4) * 32;
// tensor memory: U (two halves of 64 columns), later Y (80) | two term slots (64 each), later the weight tile (64)
constexpr uint32_t FW_U = 0, FW_TERM = 128;
constexpr int FW_L_FLOATS = 4 * RMAX_ALL * HD;
constexpr int FW_SMEM = 2 * X_BYTES + XA_BYTES + FW_L_FLOATS * 4;
static_assert(CT * 65 * 4 <= 2 * X_BYTES + XA_BYTES, "output staging tile must fit in the operand images");

__global__ void __launch_bounds__(FW_THREADS, 2) intra_fwd_kernel(const IntraFwdArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* Qimg = smem;
  unsigned char* Kimg = Qimg + X_BYTES;
  unsigned char* Uimg = Kimg + X_BYTES;
  float* lq = reinterpret_cast<float*>(Uimg + XA_BYTES);      // [quadrant][term][64]
  __shared__ __align__(16) HeadScalars sc[4];
  __shared__ uint64_t u_full[2], u_free[2], term_full[2], w_full, y_full;
  __shared__ uint32_t tmem_base;
  __shared__ int dead;
  __shared__ float den_s[CT];
  struct Unit {
    size_t row, token_row;      // of its first query in num / den, and in a token-major out
    int rows;                   // rows that exist
  };
  __shared__ Unit unit[4];
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const QueryTile tile(a.Hkv, a.N, a.rep);
  if (tile.empty()) {
    if (tid == 0) sink_status(a.status, a.sink);
    return;
  }
  const int qd = warp & 3, sub = (warp >> 2) & 1, row = 32 * qd + lane;
  const int tok0 = tile.c * CT, cols = tile.columns(), rank = a.rank;
  const int my_rb = tile.rb(qd), my_head = tile.head(qd);
  {
    const size_t koff = ((size_t)tile.b * a.Hkv + tile.kvh) * a.N + tok0;
    const size_t qoff = ((size_t)tile.b * a.Hq + my_head) * a.N + tok0 + min(32 * my_rb, tile.nc - 1);
    const int third = (warp >> 2) * 32 + lane;                  // three warps load a quadrant's rows and table
    load_rows(Qimg, 32 * qd, a.q + qoff * HD, 32, max(tile.nc - 32 * my_rb, 0), third, 96);
    load_head(lq + qd * RMAX_ALL * HD, &sc[qd], a.factors + my_head, rank, third, 96);
    load_rows(Kimg, 0, a.k + koff * HD, cols, tile.nc, tid, FW_THREADS);
    load_rows(Uimg, 0, a.v + koff * VD, cols, tile.nc, tid, FW_THREADS);
  }
  augment_rows(Uimg, tile.nc, tid, FW_THREADS);
  if (warp < 4 && lane == 0) {
    const size_t tok = tok0 + 32 * my_rb;
    unit[qd] = Unit{((size_t)tile.b * a.Hq + my_head) * a.N + tok, ((size_t)tile.b * a.N + tok) * a.Hq + my_head,
                    min(max(tile.nc - 32 * my_rb, 0), 32)};
  }
  if (warp == 0) tmem_alloc(&tmem_base, 256);
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&u_full[s], 1);
      mbar_init(&u_free[s], FW_COMPUTE);
      mbar_init(&term_full[s], FW_COMPUTE);
    }
    mbar_init(&w_full, FW_COMPUTE);
    mbar_init(&y_full, 1);
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
  int flags = 0;

  if (warp >= FW_ISSUER) {
    registers_down_to<24>();
    if (warp == FW_ISSUER) {
      const uint32_t k_addr = smem_u32(Kimg), u_addr = smem_u32(Uimg);
      if (elect_one()) {
        for (int r = 0; r < rank; ++r) {
          const uint32_t slot = tmem + FW_TERM + (r & 1) * TERM_COLS;
          w.wait(&term_full[r & 1], (r >> 1) & 1, 0x11);
          if (r > 0) w.wait(&u_free[0], (r - 1) & 1, 0x12);
          fence_after_sync();
          issue_term(tmem + FW_U, slot, k_addr, na);
          mma_commit(&u_full[0]);
          if (r > 0) w.wait(&u_free[1], (r - 1) & 1, 0x13);      // also without a second half: no barrier runs two phases ahead
          if (nb2) {
            fence_after_sync();
            issue_term(tmem + FW_U + 64, slot, k_addr + 64 * 16, nb2);
          }
          mma_commit(&u_full[1]);            // also: the term's slot has been read
        }
        w.wait(&w_full, 0, 0x14);
        fence_after_sync();
        const uint64_t du = smem_desc(u_addr, 128, CP);
        for (int part = 0; part < 2; ++part)                    // the weights' bf16 values, then their remainders
          for (int ks = 0; ks < cols / 16; ++ks)
            mma_bf16_ts(tmem + FW_U, tmem + FW_TERM + part * TERM_COLS + 8 * ks, desc_advance(du, ks * 256),
                        instr_desc_bf16(128, EP, 0, 1), part + ks > 0);
        mma_commit(&y_full);
      }
      __syncwarp();
    }
  } else {
    registers_up_to<104>();
    const unsigned char* xrow = Qimg + row * 16;
    const float* l = lq + qd * RMAX_ALL * HD;
    const int rpos = uniform(sc[qd].rpos);
    const int last_key = 32 * my_rb + 31;                     // of the quadrant
    const auto build = [&](int r) {
      const uint32_t slot = tmem + FW_TERM + (r & 1) * TERM_COLS + lane_off;
      build_term16(slot, xrow, l + r * HD, 32 * sub);
      build_term16(slot, xrow, l + r * HD, 32 * sub + 16);
      tmem_st_wait();
      fence_before_sync();
      warp_arrive(&term_full[r & 1], lane);
    };
    // this warp's keys: of every half, the first or second half of its columns, in blocks of 16
    f32x2 acc[2][2][8];
    const f32x2 w0 = f2_bcast(sc[qd].w0);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[hf][x][j] = w0;
    const auto key_of = [&](int hf, int x) { return 64 * hf + sub * ((hf ? nb2 : na) / 2) + 16 * x; };
    const auto on = [&](int hf, int x) { return 32 * x < (hf ? nb2 : na) && key_of(hf, x) <= last_key; };
    build(0);
    for (int r = 0; r < rank; ++r) {
      // the next term is built while the MMAs of this one run; its slot's last reader was term r - 1, complete
      // since u_full[1](r - 1)
      if (r + 1 < rank) build(r + 1);
      const f32x2 c2 = f2_bcast(sc[qd].c[r]);
      const auto add = [&](const float (&u)[16], f32x2 (&s)[8]) {
        if (r < rpos) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const f32x2 t = f2_add(f2_pack(u[2 * j], u[2 * j + 1]), c2);
            s[j] = f2_fma(t, t, s[j]);
          }
        } else {
          const f32x2 minus = f2_bcast(-1.f);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const f32x2 t = f2_add(f2_pack(u[2 * j], u[2 * j + 1]), c2);
            s[j] = f2_fma(f2_mul(t, minus), t, s[j]);
          }
        }
      };
      float u[16];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        w.wait(&u_full[hf], r & 1, 0x15 + hf);
        fence_after_sync();
        if (on(hf, 0)) tmem_ld16(tmem + FW_U + lane_off + key_of(hf, 0), u);
        tmem_ld_wait();
        if (on(hf, 0)) add(u, acc[hf][0]);
        if (on(hf, 1)) {                       // implies on(hf, 0)
          tmem_ld16(tmem + FW_U + lane_off + key_of(hf, 1), u);
          tmem_ld_wait();
        }
        fence_before_sync();
        warp_arrive(&u_free[hf], lane);
        if (on(hf, 1)) add(u, acc[hf][1]);
      }
    }
    // weight tile over the term slots (every MMA that read them is complete): masked, 16 keys = 8 columns, bf16 values
    // over the first slot and their rounding remainders over the second.  Without the remainders a numerator is off by
    // 2^-9 of its largest weight, which the first rows of a sequence, where few weights are summed and gradients are
    // large, turn into errors of a third of dq's rms (B = 4, N = 4096, 8 groups, gains of 20; with them
    // under a tenth).
    const int my_key = 32 * my_rb + lane;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (32 * x < (hf ? nb2 : na)) {
          const int key = key_of(hf, x);
          uint32_t o[8], rest[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float w_a, w_b;
            f2_unpack(acc[hf][x][j], w_a, w_b);
            if (key + 2 * j > my_key) w_a = 0.f;
            if (key + 2 * j + 1 > my_key) w_b = 0.f;
            o[j] = pack_bf16(w_a, w_b);
            rest[j] = pack_bf16(w_a - bf16_lo(o[j]), w_b - bf16_hi(o[j]));
          }
          tmem_st8(tmem + FW_TERM + lane_off + key / 2, o);
          tmem_st8(tmem + FW_TERM + TERM_COLS + lane_off + key / 2, rest);
        }
    tmem_st_wait();
    fence_before_sync();
    warp_arrive(&w_full, lane);
    // The epilogue's rows: 128 rows x 8 segments of 8 columns, 4 per compute thread (a warp instruction touches four
    // whole rows).  The cross-chunk numerators are on their way while Y is computed.
    constexpr int T = FW_COMPUTE * 32, PER = CT * 8 / T;
    const bool cross = tile.c >= a.cross_from;
    float4 o0[PER], o1[PER];
    static_assert(T / 8 == 32, "pass `it` of the row-major loops covers quadrant `it`");
    const int er = tid >> 3, seg = tid & 7;
    float den_cross = 0.f;
    const bool my_live = lane < unit[qd].rows;
    const size_t my_orow = unit[qd].row + lane;
    {
#pragma unroll
      for (int it = 0; it < PER; ++it) {
        o0[it] = o1[it] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (er < unit[it].rows && cross) {
          const float* np = a.num + (unit[it].row + er) * VD + seg * 8;
          o0[it] = *reinterpret_cast<const float4*>(np);
          o1[it] = *reinterpret_cast<const float4*>(np + 4);
        }
      }
      if (sub == 1 && my_live && cross) den_cross = a.den[my_orow];
    }
    w.wait(&y_full, 0, 0x17);
    fence_after_sync();
    // Every MMA has completed (or the CTA is dead): the operand images are free.  The intra-chunk numerators go
    // through a row-major staging tile in shared memory so that the global accesses are full 16- and 32-byte vectors.
    float* stage_out = reinterpret_cast<float*>(smem);        // [128][65] fp32
    asm volatile("bar.sync 1, %0;" ::"n"(FW_COMPUTE * 32) : "memory");
    {
      const int col0 = sub == 0 ? 0 : 48, ncol = sub == 0 ? 48 : 32;
#pragma unroll
      for (int cc = 0; cc < 48; cc += 16) {
        if (cc < ncol) {
          float vv[16];
          tmem_ld16(tmem + FW_U + lane_off + col0 + cc, vv);
          tmem_ld_wait();
          if (col0 + cc < VD) {
#pragma unroll
            for (int x = 0; x < 16; ++x) stage_out[row * 65 + col0 + cc + x] = vv[x];
          } else {
            const float den = vv[0] + den_cross;      // column 64
            if (my_live && !dead) {
              a.den[my_orow] = den;
              if (!finite_f(den)) flags |= OAL_STATUS_NONFINITE;
              else if (!(den > 0.f)) flags |= OAL_STATUS_DENOMINATOR;
            }
            den_s[row] = den;
          }
        }
      }
    }
    fence_before_sync();
    asm volatile("bar.sync 1, %0;" ::"n"(FW_COMPUTE * 32) : "memory");
    if (!dead) {
#pragma unroll
      for (int it = 0; it < PER; ++it) {
        if (er >= unit[it].rows) continue;
        const float inv = 1.f / fmaxf(den_s[32 * it + er], a.floor);
        const size_t oo = (unit[it].row + er) * VD + seg * 8;
        const size_t ot = a.out_token_major ? (unit[it].token_row + (size_t)er * a.Hq) * VD + seg * 8 : oo;
        float* np = a.num + oo;
        const float* sp = stage_out + (32 * it + er) * 65 + seg * 8;
        const float n[8] = {sp[0] + o0[it].x, sp[1] + o0[it].y, sp[2] + o0[it].z, sp[3] + o0[it].w,
                            sp[4] + o1[it].x, sp[5] + o1[it].y, sp[6] + o1[it].z, sp[7] + o1[it].w};
        *reinterpret_cast<float4*>(np) = make_float4(n[0], n[1], n[2], n[3]);
        *reinterpret_cast<float4*>(np + 4) = make_float4(n[4], n[5], n[6], n[7]);
        bool fin = true;
#pragma unroll
        for (int j = 0; j < 8; ++j) fin = fin && finite_f(n[j]);
        if (!fin) flags |= OAL_STATUS_NONFINITE;
        if (a.out_dt == OAL_DTYPE_BF16) {
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + ot) =
              make_uint4(pack_bf16(n[0] * inv, n[1] * inv), pack_bf16(n[2] * inv, n[3] * inv),
                         pack_bf16(n[4] * inv, n[5] * inv), pack_bf16(n[6] * inv, n[7] * inv));
        } else if (a.out_dt == OAL_DTYPE_F32) {
          float* op = reinterpret_cast<float*>(a.out) + ot;
          *reinterpret_cast<float4*>(op) = make_float4(n[0] * inv, n[1] * inv, n[2] * inv, n[3] * inv);
          *reinterpret_cast<float4*>(op + 4) = make_float4(n[4] * inv, n[5] * inv, n[6] * inv, n[7] * inv);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) store_elem(a.out, ot + j, a.out_dt, n[j] * inv);
        }
      }
    }
  }
  if (flags) atomicOr(a.status, flags);
  __syncthreads();
  w.settle();
  if (warp == 0) tmem_dealloc(tmem_base, 256);
  if (tid == 0) {
    if (dead) atomicOr(a.status, w.status_bits());
    sink_status(a.status, a.sink);
  }
}

}  // namespace

cudaError_t intra_forward(const void* q, const void* k, const void* v, const void* factors, void* out,
                          float* num, float* den, int32_t* status, int B, int Hq, int Hkv, int N, int NB, int groups,
                          int out_dt, float floor_v, bool out_token_major, int cross_from, StatusSink sink,
                          cudaStream_t st) {
  cudaError_t e = allow_smem<intra_fwd_kernel>(FW_SMEM);
  if (e != cudaSuccess) return e;
  IntraFwdArgs a{static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k),
                 static_cast<const __nv_bfloat16*>(v), static_cast<const HeadFactor*>(factors), out, num, den, status,
                 N, Hq, Hkv, Hq / Hkv, groups + 1, out_dt, floor_v, out_token_major ? 1 : 0, cross_from, sink};
  intra_fwd_kernel<<<dim3(NB, B * Hkv, Hq / Hkv), FW_THREADS, FW_SMEM, st>>>(a);
  return cudaGetLastError();
}

}  // namespace oal
