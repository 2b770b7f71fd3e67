// The gated delta rule of linear_attn.cu on prompts, in chunks of 16 tokens on the tensor cores.
//
// With alpha_t the decay, beta_t the write gate, k^, q^ the normalised keys and queries and S the state [key][value],
//   delta_t = beta_t (v_t - alpha_t S_{t-1}^T k^_t),   S_t = alpha_t S_{t-1} + k^_t delta_t^T,   y_t = S_t^T q^_t.
// Inside a chunk, with Gamma(t, j) = alpha_{j+1} .. alpha_t, g_t = alpha_1 .. alpha_t and S the state in front of the chunk,
//   (I + A) Delta = diag(beta) V - diag(beta g) K^ S,   A_tj = beta_t Gamma(t, j) k^_t . k^_j  (j < t)
//   Y = diag(g) Q^ S + M Delta,                         M_tj = Gamma(t, j) q^_t . k^_j         (j <= t)
//   S' = g_C S + K^T diag(Gamma(C, .)) Delta,
// so a chunk costs three products with the state's size and two of 16 x 16; T = (I + A)^-1 and M do not depend on S.
//
//   zb_gdn_prep   one warp per (chunk, key head): norms, K K^T, Q K^T, decays (products, never quotients), T by forward substitution,
//                 M; a record of 3.3 KB per (chunk, value head)
//   zb_gdn_scan   one CTA per (sequence, value head, 64 value columns); a warp keeps S^T of 16 value columns in registers as fp32
//                 accumulators and is independent of the others: S^T in accumulator layout is, split into bf16 pieces, the A operand
//                 of K S and Q S; chunks come through a ring of cp.async stages
//   zb_gdn_norm   the gated RMSNorm over a head's values
//
// Precision: everything that is fp32 in the token-by-token kernel stays fp32.  The bf16 inputs k, q and v enter products as they are
// (norms are factors of rows behind the product); an fp32 operand is three bf16 pieces, 24 bits, and a product of two such operands six
// products of pieces.  The large products have an accumulator apart from the small ones, and the state is updated by one fused
// multiply-add per chunk outside the tensor core, whose additions truncate.
//
// The products run over all 16 tokens of a chunk, and zero times a NaN is one.  So that a token whose inputs are not finite reaches no token
// in front of it (as token by token), a value's row with such a number is multiplied again with zeros from there on, and is NaN from there on
// (`cut_rows`; the test, behind the product, costs nothing that could be measured; in front of it 5 - 9 %).
//
// What bounds it: mma.sync: a chunk of a warp is 168 of them and about 900 other instructions, 1.6 us (3100 clocks) with a quarter of an
// SM to itself, and the next chunk waits for it.  (Q S on the FMA pipes instead: twice as long.)  32 heads of 128: 4096 tokens of one sequence 0.48 ms
// (the walk token by token: 8.1), 8192 tokens of 7 sequences of 128 .. 2048 0.55 (4.3), 8 x 512 0.24 (1.23).  Against 64 bits the
// outputs are off as before (the bf16 rounding, 2.2e-3), the state by 0.4 - 1.3 times the walk's 7e-8 .. 1.5e-6.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "host_api.h"

namespace {
constexpr uint32_t kKernelGdnScan = 25;
constexpr int kC = 16;                               // tokens of a chunk
constexpr int kRecT = 0, kRecM = 1536, kRecCoef = 3072, kRecBytes = 3344;      // T and M in pieces, [beta | c1 | c2 | c3][16], g_C
constexpr int kStages = 3;

struct GdnChunkParams {
  const __nv_bfloat16* mix;    // [T, ld_mix]: q heads | k heads | v heads
  long long ld_mix;
  const __nv_bfloat16* z;      // [T, ld_z]
  long long ld_z;
  const __nv_bfloat16* a;      // [T, ld_ab]
  const __nv_bfloat16* b;
  long long ld_ab;
  const float* a_log;          // [hv]
  const float* dt_bias;        // [hv]
  const __nv_bfloat16* norm_w; // [dv]
  float eps;
  float* state;                // [slots, hv, dk, dv]
  __nv_bfloat16* out;          // [T, ld_out]
  long long ld_out;
  const int32_t* q_start;
  const int32_t* seq_lens;
  const int32_t* slots;
  uint8_t* rec;                // [T / 16 + seqs][hv][kRecBytes]
  __nv_bfloat16* y;            // [T, hv * dv]
  int num_seqs, tokens;
  int hk, hv, dv;
};

// Records of sequence s begin here: the number of chunks in front of it is at most this.
ZB_DEVICE int chunk_base(const int32_t* q_start, int s) { return q_start[s] / kC + s; }

ZB_DEVICE void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
ZB_DEVICE void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
ZB_DEVICE void stsm4_t(uint32_t addr, const uint32_t (&r)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
ZB_DEVICE void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
ZB_DEVICE void cp16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
ZB_DEVICE float lo_of(uint32_t u) { return __uint_as_float(u << 16); }
ZB_DEVICE float hi_of(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// Two fp32 as three bf16 pieces each: x = p[0] + p[1] + p[2] up to 2^-24 of x.
ZB_DEVICE void split3(float x0, float x1, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = zb_pack_bf16x2(x0, x1);
  x0 -= lo_of(p0);
  x1 -= hi_of(p0);
  p1 = zb_pack_bf16x2(x0, x1);
  x0 -= lo_of(p1);
  x1 -= hi_of(p1);
  p2 = zb_pack_bf16x2(x0, x1);
}
// A 16 x 16 A operand from two accumulator tiles.
ZB_DEVICE void split_a(const float (&u)[4], const float (&v)[4], uint32_t (&a)[3][4]) {
  split3(u[0], u[1], a[0][0], a[1][0], a[2][0]);
  split3(u[2], u[3], a[0][1], a[1][1], a[2][1]);
  split3(v[0], v[1], a[0][2], a[1][2], a[2][2]);
  split3(v[2], v[3], a[0][3], a[1][3], a[2][3]);
}
// cut: the first token (column) of either row of X^T [2 tiles of 8 tokens] that is not finite, 16 where there is none; zeros from there on.
// The whole warp; true where a row may be cut.
ZB_DEVICE bool cut_rows(float (&x)[2][4], int (&cut)[2]) {
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) sum += fabsf(x[0][i]) + fabsf(x[1][i]);
  cut[0] = cut[1] = kC;
  if (__all_sync(0xffffffffu, sum < INFINITY)) return false;
  const int t0 = 2 * (threadIdx.x & 3);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (!(fabsf(x[i >> 2][i & 3]) < INFINITY)) cut[(i >> 1) & 1] = min(cut[(i >> 1) & 1], (i >> 2) * 8 + t0 + (i & 1));
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    cut[h] = min(cut[h], __shfl_xor_sync(0xffffffffu, cut[h], 1));
    cut[h] = min(cut[h], __shfl_xor_sync(0xffffffffu, cut[h], 2));
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((i >> 2) * 8 + t0 + (i & 1) >= cut[(i >> 1) & 1]) x[i >> 2][i & 3] = 0.f;
  return true;
}
// hi += a b over the leading pieces, lo += the other products that matter; b as a record keeps it (two n-tiles per piece).
ZB_DEVICE void mma_pieces(float (&hi)[2][4], float (&lo)[2][4], const uint32_t (&a)[3][4], const uint4* b) {
  const uint4 b0 = b[0], b1 = b[32], b2 = b[64];
  mma(lo[0], a[2], b0.x, b0.y);
  mma(lo[1], a[2], b0.z, b0.w);
  mma(hi[0], a[0], b0.x, b0.y);
  mma(hi[1], a[0], b0.z, b0.w);
  mma(lo[0], a[0], b2.x, b2.y);
  mma(lo[1], a[0], b2.z, b2.w);
  mma(lo[0], a[1], b1.x, b1.y);
  mma(lo[1], a[1], b1.z, b1.w);
  mma(lo[0], a[1], b0.x, b0.y);
  mma(lo[1], a[1], b0.z, b0.w);
  mma(lo[0], a[0], b1.x, b1.y);
  mma(lo[1], a[0], b1.z, b1.w);
}

ZB_DEVICE void add_tiles(float (&x)[2][4], const float (&y)[2][4]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i >> 2][i & 3] += y[i >> 2][i & 3];
}
// d = x b^T anew for rows that are cut, with NaN from the cut on.
ZB_DEVICE void again_from(float (&d)[2][4], const float (&x)[2][4], const int (&cut)[2], const uint4* b) {
  uint32_t a[3][4];
  float lo[2][4] = {};
#pragma unroll
  for (int i = 0; i < 8; ++i) d[i >> 2][i & 3] = 0.f;
  split_a(x[0], x[1], a);
  mma_pieces(d, lo, a, b);
  add_tiles(d, lo);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((i >> 2) * 8 + 2 * static_cast<int>(threadIdx.x & 3) + (i & 1) >= cut[(i >> 1) & 1]) d[i >> 2][i & 3] = __int_as_float(0x7fffffff);
}

// ------------------------------------------------------------------------------------------
constexpr int kPrepWarps = 4;
template <int DK>
struct PrepShared {
  __nv_bfloat16 k[kC][DK + 8], q[kC][DK + 8];
  float kk[kC][kC + 1], qk[kC][kC + 1], gam[kC][kC + 1], t[kC][kC + 1];
  float ck[kC], cq[kC], al[kC], be[kC], g[kC];
};

template <int DK>
__global__ void __launch_bounds__(32 * kPrepWarps) zb_gdn_prep_kernel(const GdnChunkParams p) {
  zb_pdl_launch();
  zb_pdl_wait();
  extern __shared__ __align__(16) uint8_t raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  PrepShared<DK>& sh = reinterpret_cast<PrepShared<DK>*>(raw)[warp];
  const int item = blockIdx.x * kPrepWarps + warp, cid = item / p.hk, kh = item - cid * p.hk;
  if (cid >= p.tokens / kC + p.num_seqs) return;
  int s = 0;                                         // the last sequence whose records begin at or in front of cid
  for (int hi = p.num_seqs; hi - s > 1;) {
    const int mid = (s + hi) >> 1;
    if (chunk_base(p.q_start, mid) <= cid) s = mid; else hi = mid;
  }
  const int t0 = p.q_start[s] + (cid - chunk_base(p.q_start, s)) * kC, n = min(kC, p.q_start[s + 1] - t0);
  if (n <= 0 || t0 < p.q_start[s]) return;           // the whole warp; no block barrier below.  (In front of the first sequence: nobody's rows.)

  constexpr int kPieces = DK / 8;                    // 16-byte pieces of a row
#pragma unroll
  for (int i = lane; i < kC * kPieces; i += 32) {
    const int row = i / kPieces, c = (i - row * kPieces) * 8;
    uint4 kv = make_uint4(0, 0, 0, 0), qv = kv;
    if (row < n) {
      const __nv_bfloat16* src = p.mix + static_cast<long long>(t0 + row) * p.ld_mix + kh * DK + c;
      qv = *reinterpret_cast<const uint4*>(src);
      kv = *reinterpret_cast<const uint4*>(src + p.hk * DK);
    }
    *reinterpret_cast<uint4*>(&sh.k[row][c]) = kv;
    *reinterpret_cast<uint4*>(&sh.q[row][c]) = qv;
  }
  __syncwarp();
  {
    const int row = lane >> 1, c0 = (lane & 1) * (DK / 2);
    float sk = 0.f, sq = 0.f;
#pragma unroll 8
    for (int c = 0; c < DK / 2; c += 2) {
      const uint32_t ku = *reinterpret_cast<const uint32_t*>(&sh.k[row][c0 + c]), qu = *reinterpret_cast<const uint32_t*>(&sh.q[row][c0 + c]);
      sk = fmaf(lo_of(ku), lo_of(ku), fmaf(hi_of(ku), hi_of(ku), sk));
      sq = fmaf(lo_of(qu), lo_of(qu), fmaf(hi_of(qu), hi_of(qu), sq));
    }
    sk += __shfl_xor_sync(0xffffffffu, sk, 1);
    sq += __shfl_xor_sync(0xffffffffu, sq, 1);
    if ((lane & 1) == 0) {
      sh.ck[row] = row < n ? rsqrtf(sk + 1e-6f) : 0.f;
      sh.cq[row] = row < n ? rsqrtf(sq + 1e-6f) * rsqrtf(static_cast<float>(DK)) : 0.f;
    }
  }
  float kk[2][4] = {}, qk[2][4] = {};
  {
    const int mi = lane >> 3, r = lane & 7;
    const uint32_t a_k = zb_smem_u32(&sh.k[(mi & 1) * 8 + r][(mi >> 1) * 8]), a_q = zb_smem_u32(&sh.q[(mi & 1) * 8 + r][(mi >> 1) * 8]);
    const uint32_t b_k = zb_smem_u32(&sh.k[(mi >> 1) * 8 + r][(mi & 1) * 8]);
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
      uint32_t ak[4], aq[4], bk[4];
      ldsm4(ak, a_k + ks * 32);
      ldsm4(aq, a_q + ks * 32);
      ldsm4(bk, b_k + ks * 32);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        mma(kk[nt], ak, bk[2 * nt], bk[2 * nt + 1]);
        mma(qk[nt], aq, bk[2 * nt], bk[2 * nt + 1]);
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = g + 8 * (i >> 1), j = nt * 8 + 2 * tq + (i & 1);
      sh.kk[t][j] = kk[nt][i] * sh.ck[t] * sh.ck[j];
      sh.qk[t][j] = qk[nt][i] * sh.cq[t] * sh.ck[j];
    }

  const int rep = p.hv / p.hk;
  for (int v = 0; v < rep; ++v) {
    const int h = kh * rep + v;
    __syncwarp();
    if (lane < kC) {
      float alpha = 1.f, beta = 0.f;
      if (lane < n) {
        const long long at = static_cast<long long>(t0 + lane) * p.ld_ab + h;
        const float x = __bfloat162float(p.a[at]) + p.dt_bias[h];
        alpha = expf(-expf(p.a_log[h]) * (x > 20.f ? x : log1pf(expf(x))));
        beta = 1.f / (1.f + expf(-__bfloat162float(p.b[at])));
      }
      sh.al[lane] = alpha;
      sh.be[lane] = beta;
    }
    __syncwarp();
    if (lane <= kC) {                                // column `lane` of Gamma; the last lane has the decay from the chunk's start
      float r = 1.f;
#pragma unroll
      for (int t = 0; t < kC; ++t) {
        if (lane == kC) {
          r *= sh.al[t];
          sh.g[t] = r;
        } else if (t >= lane) {
          if (t > lane) r *= sh.al[t];
          sh.gam[t][lane] = r;
        } else {
          sh.gam[t][lane] = 0.f;
        }
      }
    }
    __syncwarp();
    if (lane < kC) {                                 // column `lane` of T
      float x[kC];
#pragma unroll
      for (int t = 0; t < kC; ++t) {
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < t; ++i) acc = fmaf(sh.gam[t][i] * sh.kk[t][i], x[i], acc);
        x[t] = (t == lane ? 1.f : 0.f) - sh.be[t] * acc;
      }
#pragma unroll
      for (int t = 0; t < kC; ++t) sh.t[t][lane] = x[t];
    }
    __syncwarp();
    uint8_t* rec = p.rec + (static_cast<size_t>(cid) * p.hv + h) * kRecBytes;
    uint32_t ft[3][4], fm[3][4];                     // [piece][n-tile and half]: the B operands T^T and M^T
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = nt * 8 + g, j = 2 * tq + 8 * half, at = 2 * nt + half;
        split3(sh.t[t][j], sh.t[t][j + 1], ft[0][at], ft[1][at], ft[2][at]);
        split3(j <= t ? sh.gam[t][j] * sh.qk[t][j] : 0.f, j < t ? sh.gam[t][j + 1] * sh.qk[t][j + 1] : 0.f, fm[0][at], fm[1][at], fm[2][at]);
      }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      reinterpret_cast<uint4*>(rec + kRecT)[q * 32 + lane] = make_uint4(ft[q][0], ft[q][1], ft[q][2], ft[q][3]);
      reinterpret_cast<uint4*>(rec + kRecM)[q * 32 + lane] = make_uint4(fm[q][0], fm[q][1], fm[q][2], fm[q][3]);
    }
    float* coef = reinterpret_cast<float*>(rec + kRecCoef);
    if (lane < kC) {
      coef[lane] = sh.be[lane];
      coef[kC + lane] = sh.be[lane] * sh.g[lane] * sh.ck[lane];
      coef[2 * kC + lane] = sh.g[lane] * sh.cq[lane];
      coef[3 * kC + lane] = sh.gam[kC - 1][lane] * sh.ck[lane];
    } else if (lane == kC) {
      coef[4 * kC] = sh.g[kC - 1];
    }
  }
}

// ------------------------------------------------------------------------------------------
template <int DK, int DVP>
struct ScanStage {
  __nv_bfloat16 k[kC][DK + 8], q[kC][DK + 8], v[kC][DVP + 8];
  uint8_t rec[kRecBytes];
};

template <int DK, int DVP>
__global__ void __launch_bounds__(2 * DVP) zb_gdn_scan_kernel(const GdnChunkParams p) {
  zb_pdl_launch();
  zb_pdl_wait();
  using Stage = ScanStage<DK, DVP>;
  static_assert(sizeof(Stage) % 16 == 0, "stages start on 16 bytes");
  extern __shared__ __align__(16) uint8_t raw[];
  Stage* stages = reinterpret_cast<Stage*>(raw);
  constexpr int kThreads = 2 * DVP, kPitch = 24;     // staged outputs: 16 values and 8 of padding per token
  __nv_bfloat16* y_s = reinterpret_cast<__nv_bfloat16*>(raw + kStages * sizeof(Stage));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3, mi = lane >> 3, r8 = lane & 7;
  const int parts = p.dv / DVP, h = blockIdx.x / parts, part = blockIdx.x - h * parts, s = blockIdx.y;
  const int t0 = p.q_start[s], n = p.q_start[s + 1] - t0;
  if (n <= 0) return;
  if (!ZB_BC_OK(p.slots[s], ZB_BC_STATE_SLOTS, kKernelGdnScan, 1)) return;      // uniform over the block
  const int chunks = (n + kC - 1) / kC, kh = h / (p.hv / p.hk), key_dim = p.hk * DK;
  const uint8_t* rec = p.rec + (static_cast<size_t>(chunk_base(p.q_start, s)) * p.hv + h) * kRecBytes;
  const __nv_bfloat16* qcol = p.mix + kh * DK;
  const __nv_bfloat16* vcol = p.mix + 2 * key_dim + h * p.dv + part * DVP;

  auto load = [&](int c) {
    if (c < chunks) {
      Stage& st = stages[c % kStages];
      constexpr int kKp = DK / 8, kVp = DVP / 8;
#pragma unroll
      for (int i = threadIdx.x; i < kC * kKp; i += kThreads) {
        const int row = i / kKp, col = (i - row * kKp) * 8, tok = c * kC + row;
        const __nv_bfloat16* src = qcol + static_cast<long long>(t0 + min(tok, n - 1)) * p.ld_mix + col;
        const uint32_t bytes = tok < n ? 16u : 0u;
        cp16(zb_smem_u32(&st.q[row][col]), src, bytes);
        cp16(zb_smem_u32(&st.k[row][col]), src + key_dim, bytes);
      }
#pragma unroll
      for (int i = threadIdx.x; i < kC * kVp; i += kThreads) {
        const int row = i / kVp, col = (i - row * kVp) * 8, tok = c * kC + row;
        cp16(zb_smem_u32(&st.v[row][col]), vcol + static_cast<long long>(t0 + min(tok, n - 1)) * p.ld_mix + col, tok < n ? 16u : 0u);
      }
      const uint8_t* from = rec + static_cast<size_t>(c) * p.hv * kRecBytes;
      for (int i = threadIdx.x; i < kRecBytes / 16; i += kThreads) cp16(zb_smem_u32(st.rec + i * 16), from + i * 16, 16u);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // S^T: rows are this warp's value columns (g, g + 8), columns keys (8 j + 2 tq, + 1)
  float S[DK / 8][4];
  float* st = p.state + (static_cast<size_t>(p.slots[s]) * p.hv + h) * DK * p.dv + part * DVP + warp * 16 + g;
  const bool fresh = p.seq_lens[s] - n <= 0;
  load(0);
  load(1);
#pragma unroll
  for (int j = 0; j < DK / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) S[j][i] = fresh ? 0.f : st[static_cast<size_t>(8 * j + 2 * tq + (i & 1)) * p.dv + 8 * (i >> 1)];

  __nv_bfloat16* y_w = y_s + warp * kC * kPitch;
  const uint32_t y_at = zb_smem_u32(y_w + ((mi >> 1) * 8 + r8) * kPitch + (mi & 1) * 8);
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                 // this chunk's stage is complete, and the previous one's readers are done
    load(c + 2);
    const Stage& sg = stages[c % kStages];
    const uint32_t k_at = zb_smem_u32(&sg.k[(mi >> 1) * 8 + r8][(mi & 1) * 8]), q_at = zb_smem_u32(&sg.q[(mi >> 1) * 8 + r8][(mi & 1) * 8]);
    const uint32_t kt_at = zb_smem_u32(&sg.k[(mi & 1) * 8 + r8][(mi >> 1) * 8]);
    const float* coef = reinterpret_cast<const float*>(sg.rec + kRecCoef);

    // (K S)^T and (Q S)^T: [16 values x 16 tokens]
    float rh[2][4] = {}, rl[2][4] = {}, yh[2][4] = {}, yl[2][4] = {};
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
      uint32_t a[3][4], kf[4], qf[4];
      ldsm4(kf, k_at + ks * 32);
      ldsm4(qf, q_at + ks * 32);
      split_a(S[2 * ks], S[2 * ks + 1], a);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        mma(rh[nt], a[0], kf[2 * nt], kf[2 * nt + 1]);
        mma(yh[nt], a[0], qf[2 * nt], qf[2 * nt + 1]);
        mma(rl[nt], a[1], kf[2 * nt], kf[2 * nt + 1]);
        mma(yl[nt], a[1], qf[2 * nt], qf[2 * nt + 1]);
        mma(rl[nt], a[2], kf[2 * nt], kf[2 * nt + 1]);
        mma(yl[nt], a[2], qf[2 * nt], qf[2 * nt + 1]);
      }
    }
    // right-hand side, then Delta^T
    uint32_t vf[4], a[3][4];
    ldsm4_t(vf, zb_smem_u32(&sg.v[(mi >> 1) * 8 + r8][warp * 16 + (mi & 1) * 8]));
    float x[2][4], d[2][4] = {}, dl[2][4] = {};
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const float2 be = *reinterpret_cast<const float2*>(coef + nt * 8 + 2 * tq), c1 = *reinterpret_cast<const float2*>(coef + kC + nt * 8 + 2 * tq);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float v = (i & 1) ? hi_of(vf[2 * nt + (i >> 1)]) : lo_of(vf[2 * nt + (i >> 1)]);
        x[nt][i] = fmaf(-((i & 1) ? c1.y : c1.x), rh[nt][i] + rl[nt][i], ((i & 1) ? be.y : be.x) * v);
      }
    }
    split_a(x[0], x[1], a);
    mma_pieces(d, dl, a, reinterpret_cast<const uint4*>(sg.rec + kRecT) + lane);
    add_tiles(d, dl);
    int cut[2];
    const bool odd = cut_rows(x, cut);               // whatever T and M hold beside x: a key or gate that is not finite makes x so
    if (odd) again_from(d, x, cut, reinterpret_cast<const uint4*>(sg.rec + kRecT) + lane);
    // S' = g S + K^T diag(c3) Delta
    {
      const float gc = coef[4 * kC];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float2 c3 = *reinterpret_cast<const float2*>(coef + 3 * kC + nt * 8 + 2 * tq);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[nt][i] = d[nt][i] * ((i & 1) ? c3.y : c3.x);
      }
      split_a(x[0], x[1], a);
#pragma unroll
      for (int j = 0; j < DK / 8; j += 2) {
        uint32_t kf[4];
        ldsm4_t(kf, kt_at + j * 16);
        float u[2][4] = {};
#pragma unroll
        for (int q = 2; q >= 0; --q) {
          mma(u[0], a[q], kf[0], kf[1]);
          mma(u[1], a[q], kf[2], kf[3]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          S[j][i] = fmaf(gc, S[j][i], u[0][i]);
          S[j + 1][i] = fmaf(gc, S[j + 1][i], u[1][i]);
        }
      }
    }
    // Y^T = diag(c2) (Q S)^T + Delta^T M^T
    {
      float e[2][4] = {}, el[2][4] = {};
      split_a(d[0], d[1], a);
      mma_pieces(e, el, a, reinterpret_cast<const uint4*>(sg.rec + kRecM) + lane);
      add_tiles(e, el);
      if (odd && cut_rows(d, cut)) again_from(e, d, cut, reinterpret_cast<const uint4*>(sg.rec + kRecM) + lane);
      uint32_t yo[4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float2 c2 = *reinterpret_cast<const float2*>(coef + 2 * kC + nt * 8 + 2 * tq);
#pragma unroll
        for (int i = 0; i < 4; ++i) e[nt][i] = fmaf((i & 1) ? c2.y : c2.x, yh[nt][i] + yl[nt][i], e[nt][i]);
        yo[2 * nt] = zb_pack_bf16x2(e[nt][0], e[nt][1]);
        yo[2 * nt + 1] = zb_pack_bf16x2(e[nt][2], e[nt][3]);
      }
      __syncwarp();
      stsm4_t(y_at, yo);
      __syncwarp();
      const int tok = c * kC + (lane >> 1);
      if (tok < n)
        *reinterpret_cast<uint4*>(p.y + static_cast<size_t>(t0 + tok) * p.hv * p.dv + h * p.dv + part * DVP + warp * 16 + (lane & 1) * 8) =
            *reinterpret_cast<const uint4*>(y_w + (lane >> 1) * kPitch + (lane & 1) * 8);
    }
  }
#pragma unroll
  for (int j = 0; j < DK / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) st[static_cast<size_t>(8 * j + 2 * tq + (i & 1)) * p.dv + 8 * (i >> 1)] = S[j][i];
}

// ------------------------------------------------------------------------------------------
// weight * y / rms(y) * silu(z): G lanes per (token, head), 16 bytes a lane, two of them on their way at once.  It should move three times
// the outputs' bytes: 8192 tokens of 32 heads of 128, 201 MB, 30 us at the copy bandwidth; 60 us (86 with a warp per head, 8 bytes a
// lane, one at a time and a division for every one).
template <int G>
__global__ void __launch_bounds__(256) zb_gdn_norm_kernel(const GdnChunkParams p) {
  zb_pdl_launch();
  zb_pdl_wait();
  const int at = (threadIdx.x & (G - 1)) * 8;
  const bool mine = at < p.dv;
  float w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = mine ? __bfloat162float(p.norm_w[at + i]) : 0.f;
  const long long first = (blockIdx.x * 256ll + threadIdx.x) / G, stride = gridDim.x * (256ll / G), items = static_cast<long long>(p.tokens) * p.hv;
  const long long t_step = stride / p.hv;
  const int h_step = static_cast<int>(stride - t_step * p.hv);
  const int t_first = p.q_start[0], t_last = min(p.q_start[p.num_seqs], p.tokens);      // rows of no sequence stay as they are
  long long t = first / p.hv;
  int h = static_cast<int>(first - t * p.hv);
  const long long warp_first = (blockIdx.x * 256ll + (threadIdx.x & ~31)) / G;
  for (long long base = warp_first; base < items; base += 2 * stride) {      // a warp goes through the loop as a whole
    uint4 y[2], z[2];
    long long to[2];
    bool in[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      in[k] = mine && t >= t_first && t < t_last;
      y[k] = z[k] = make_uint4(0u, 0u, 0u, 0u);
      const long long col = static_cast<long long>(h) * p.dv + at;
      if (in[k]) {
        y[k] = *reinterpret_cast<const uint4*>(p.y + t * p.hv * p.dv + col);
        z[k] = *reinterpret_cast<const uint4*>(p.z + t * p.ld_z + col);
      }
      to[k] = t * p.ld_out + col;
      t += t_step;
      h += h_step;
      if (h >= p.hv) {
        h -= p.hv;
        ++t;
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t yu[4] = {y[k].x, y[k].y, y[k].z, y[k].w}, zu[4] = {z[k].x, z[k].y, z[k].z, z[k].w};
      float f[8], ss = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        f[2 * i] = lo_of(yu[i]);
        f[2 * i + 1] = hi_of(yu[i]);
        ss = fmaf(f[2 * i], f[2 * i], fmaf(f[2 * i + 1], f[2 * i + 1], ss));
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float inv = rsqrtf(ss / static_cast<float>(p.dv) + p.eps);
      uint32_t o4[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float z0 = lo_of(zu[i]), z1 = hi_of(zu[i]);
        o4[i] = zb_pack_bf16x2(f[2 * i] * inv * w[2 * i] * (z0 / (1.f + __expf(-z0))), f[2 * i + 1] * inv * w[2 * i + 1] * (z1 / (1.f + __expf(-z1))));
      }
      if (in[k]) *reinterpret_cast<uint4*>(p.out + to[k]) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
    }
  }
}

template <int DK, int DVP>
int launch_scan(const GdnChunkParams& p, cudaStream_t s) {
  constexpr int kSmem = kStages * sizeof(ScanStage<DK, DVP>) + (DVP / 16) * kC * 24 * 2;
  static bool configured[16] = {};
  constexpr int kShare = 227 * 1024, kMost = kShare / 2 + 1024;
  if (const int rc = zb_config_smem_once(zb_gdn_scan_kernel<DK, DVP>, std::max(kSmem, kMost), configured)) return rc;
  // A CTA asks for so much shared memory that an SM holds no more of them than its part: those that start while zb_gdn_prep still holds
  // most SMs would otherwise crowd on the others, where they share a tensor core for as long as they run: one sequence of 4096 tokens (64 CTAs)
  // 0.72 - 0.80 ms so, 0.48 on an SM each; eight of 512 (512 CTAs) 0.234 either way.
  const long long ctas = static_cast<long long>(p.hv) * (p.dv / DVP) * p.num_seqs, sms = std::max(1, zb_num_sms()), per_sm = (ctas + sms - 1) / sms;
  const int smem = std::max(kSmem, static_cast<int>(kShare / (per_sm + 1)) / 16 * 16 + 1024);
  zb_launch(zb_gdn_scan_kernel<DK, DVP>, dim3(p.hv * (p.dv / DVP), p.num_seqs), dim3(2 * DVP), smem, s, p);
  return static_cast<int>(cudaGetLastError());
}

template <int DK>
int launch_chunked(const GdnChunkParams& p, cudaStream_t s) {
  constexpr int kSmem = kPrepWarps * sizeof(PrepShared<DK>);
  static bool configured[16] = {};
  if (const int rc = zb_config_smem_once(zb_gdn_prep_kernel<DK>, kSmem, configured)) return rc;
  const long long items = (static_cast<long long>(p.tokens) / kC + p.num_seqs) * p.hk;
  zb_launch(zb_gdn_prep_kernel<DK>, dim3(static_cast<unsigned>((items + kPrepWarps - 1) / kPrepWarps)), dim3(32 * kPrepWarps), kSmem, s, p);
  if (const int rc = static_cast<int>(cudaGetLastError())) return rc;
  if (const int rc = p.dv % 64 == 0 ? launch_scan<DK, 64>(p, s) : launch_scan<DK, 32>(p, s)) return rc;
  const int lanes = p.dv <= 32 ? 4 : (p.dv <= 64 ? 8 : (p.dv <= 128 ? 16 : 32));
  const auto norm = lanes == 4 ? zb_gdn_norm_kernel<4> : (lanes == 8 ? zb_gdn_norm_kernel<8> : (lanes == 16 ? zb_gdn_norm_kernel<16> : zb_gdn_norm_kernel<32>));
  const long long blocks = (static_cast<long long>(p.tokens) * p.hv * lanes + 255) / 256;
  zb_launch(norm, dim3(static_cast<unsigned>(std::min(zb_num_sms() * 8ll, blocks))), dim3(256), 0, s, p);
  zb_count_launch(3);
  return static_cast<int>(cudaGetLastError());
}
}  // namespace

extern "C" {

// Bytes of `rec` for a batch.
size_t zb_gated_delta_rec_bytes(int tokens, int num_seqs, int hv) { return (static_cast<size_t>(tokens) / kC + num_seqs) * hv * kRecBytes; }

// zb_gated_delta_scan over chunks, for batches with prompts.  dk in {64, 128}; dv a multiple of 32, <= 256.  mix, z and out start on 16
// bytes and their row strides are multiples of 8 elements.  `rec` (zb_gated_delta_rec_bytes, 16-byte aligned) and `y` (bf16
// [tokens, hv * dv]) are scratch; y may be out.
int zb_gated_delta_chunked(const void* mix, long long ld_mix, const void* z, long long ld_z, const void* a, const void* b, long long ld_ab,
                           const float* a_log, const float* dt_bias, const void* norm_w, float eps, float* state, void* out, long long ld_out,
                           const int32_t* q_start, const int32_t* seq_lens, const int32_t* slots, int num_seqs, int tokens, int hk, int hv, int dk,
                           int dv, void* rec, void* y, void* stream) {
  if (num_seqs <= 0 || tokens <= 0) return 0;
  if (hk <= 0 || hv % hk != 0 || dv % 32 != 0 || dv > 256) return -71;
  if (((reinterpret_cast<uintptr_t>(mix) | reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(rec) |
        reinterpret_cast<uintptr_t>(y)) & 15) != 0 || ((ld_mix | ld_z | ld_out) & 7) != 0)
    return -74;
  GdnChunkParams p;
  p.mix = reinterpret_cast<const __nv_bfloat16*>(mix);
  p.ld_mix = ld_mix;
  p.z = reinterpret_cast<const __nv_bfloat16*>(z);
  p.ld_z = ld_z;
  p.a = reinterpret_cast<const __nv_bfloat16*>(a);
  p.b = reinterpret_cast<const __nv_bfloat16*>(b);
  p.ld_ab = ld_ab;
  p.a_log = a_log;
  p.dt_bias = dt_bias;
  p.norm_w = reinterpret_cast<const __nv_bfloat16*>(norm_w);
  p.eps = eps;
  p.state = state;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.ld_out = ld_out;
  p.q_start = q_start;
  p.seq_lens = seq_lens;
  p.slots = slots;
  p.rec = reinterpret_cast<uint8_t*>(rec);
  p.y = reinterpret_cast<__nv_bfloat16*>(y);
  p.num_seqs = num_seqs;
  p.tokens = tokens;
  p.hk = hk;
  p.hv = hv;
  p.dv = dv;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dk == 64) return launch_chunked<64>(p, s);
  if (dk == 128) return launch_chunked<128>(p, s);
  return -72;
}

}  // extern "C"
