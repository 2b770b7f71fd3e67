// Bandwidth-bound layer glue for sm_100a: RMSNorm(+residual), RoPE fused with the
// paged KV-cache write (and optional per-head q/k RMSNorm), SwiGLU, embedding
// gather, argmax and top-k + Gumbel-max sampling.
//
// These replace XLA's elementwise / reduction fusions of the reference:
// rmsNorm zml/nn.zig:486-493, rope zml/nn.zig:687-716, KvCache.update
// zml/attention/paged_attention.zig:218-254, swiglu
// examples/llm/models/llama/model.zig:491-496, TokenEmbedding zml/nn.zig:432-436,
// sampleTokens zml/nn.zig:1999-2033.
#include <algorithm>

#include "common.cuh"
#include "host_api.h"

namespace {
constexpr uint32_t kKernelRopeKvWrite = 20;
constexpr uint32_t kKernelEmbedding = 21;
constexpr uint32_t kKernelDecodeAdvance = 22;

// ---------------------------------------------------------------- RMSNorm
// y = x_total * rsqrt(mean(x_total^2) + eps) * (w or 1 + w), x_total = x (+ residual).
// When residual_out != null the summed row is written back (pre-norm residual stream).
template <int VEC_PER_THREAD>
__global__ void __launch_bounds__(256) zb_rmsnorm_kernel(
    const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
    const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out,
    __nv_bfloat16* __restrict__ residual_out, int rows, int d, long long x_stride,
    long long out_stride, float eps, int unit_offset) {
  zb_pdl_launch();
  zb_pdl_wait();
  const int row = blockIdx.x;
  if (row >= rows) return;
  const int nvec = d >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * x_stride);
  const uint4* rr = residual ? reinterpret_cast<const uint4*>(residual + static_cast<size_t>(row) * d) : nullptr;
  uint4* ro = residual_out ? reinterpret_cast<uint4*>(residual_out + static_cast<size_t>(row) * d) : nullptr;
  float vals[VEC_PER_THREAD][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < VEC_PER_THREAD; ++i) {
    const int v = threadIdx.x + i * 256;
    if (v < nvec) {
      uint4 a = xr[v];
      const uint32_t au[4] = {a.x, a.y, a.z, a.w};
      uint32_t bu[4] = {0, 0, 0, 0};
      if (rr) {
        uint4 b = rr[v];
        bu[0] = b.x; bu[1] = b.y; bu[2] = b.z; bu[3] = b.w;
      }
      uint32_t su[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f = zb_unpack_bf16x2(au[j]);
        if (rr) {
          float2 g = zb_unpack_bf16x2(bu[j]);
          f.x += g.x;
          f.y += g.y;
          // the residual stream is stored in bf16: normalise what is stored
          su[j] = zb_pack_bf16x2(f.x, f.y);
          f = zb_unpack_bf16x2(su[j]);
        }
        vals[i][2 * j] = f.x;
        vals[i][2 * j + 1] = f.y;
        ss += f.x * f.x + f.y * f.y;
      }
      if (ro) ro[v] = rr ? make_uint4(su[0], su[1], su[2], su[3]) : a;
    }
  }
  __shared__ float red[8];
  ss = zb_warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float inv = rsqrtf(tot / static_cast<float>(d) + eps);
  uint4* orow = reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * out_stride);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
#pragma unroll
  for (int i = 0; i < VEC_PER_THREAD; ++i) {
    const int v = threadIdx.x + i * 256;
    if (v < nvec) {
      uint32_t wu[4] = {0, 0, 0, 0};
      if (w) {
        uint4 ww = wr[v];
        wu[0] = ww.x; wu[1] = ww.y; wu[2] = ww.z; wu[3] = ww.w;
      }
      uint32_t ou[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 g = w ? zb_unpack_bf16x2(wu[j]) : make_float2(1.f, 1.f);
        if (unit_offset) {
          g.x += 1.f;
          g.y += 1.f;
        }
        ou[j] = zb_pack_bf16x2(vals[i][2 * j] * inv * g.x, vals[i][2 * j + 1] * inv * g.y);
      }
      orow[v] = make_uint4(ou[0], ou[1], ou[2], ou[3]);
    }
  }
}

// ---------------------------------------------------------------- RoPE + KV write
// One warp per (token, head) of the fused qkv activation [T, (Hq + 2*Hkv) * hd].
//   q heads : optional RMSNorm over hd, rotate, write to q_out [T, Hq, hd]
//   k heads : optional RMSNorm, rotate, write into the paged K cache at slot_mapping[t]
//   v heads : copy into the paged V cache
// rope layout 0 (real_im_pass, HF rotate_half): pairs (i, i + rot/2), pass-through after rot;
//             1 (interleaved): pairs (2i, 2i + 1);
//             2 (real_pass_im_pass): pairs (i, hd/2 + i) for i < rot/2.
struct RopeParams {
  const __nv_bfloat16* qkv;
  __nv_bfloat16* q_out;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  const int32_t* positions;
  const int32_t* slot_mapping;
  const float* inv_freq;        // [rot_dim / 2]
  const __nv_bfloat16* q_norm_w;  // [hd] or null
  const __nv_bfloat16* k_norm_w;
  long long qkv_stride;
  int tokens, hq, hkv, hd, rot_dim, layout, page_size;
  float attn_factor;            // yarn magnitude scaling applied to cos/sin
  float norm_eps;
  int norm_unit_offset;
  long long num_slots;          // bounds for slot_mapping; slots < 0 are skipped (padding)
  int share;                    // pieces of a token that one CTA takes (zb_rope_rows_kernel)
};

// One warp takes `heads_per_warp` consecutive heads (q, then k, then v) of one token: the rotation angles
// depend on the token only, so sin / cos are computed once per warp and reused for its heads (with one head
// per warp the accurate sincosf on position x frequency dominated prefill: 128 us for 8 192 tokens x 36 heads).
__global__ void __launch_bounds__(128) zb_rope_kvwrite_kernel(const RopeParams p, int heads_per_warp) {
  zb_pdl_launch();
  zb_pdl_wait();
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int heads = p.hq + 2 * p.hkv;
  const int groups = (heads + heads_per_warp - 1) / heads_per_warp;
  if (warp_global >= p.tokens * groups) return;
  const int tok = warp_global / groups;
  const int h_begin = (warp_global - tok * groups) * heads_per_warp;
  const int h_end = min(heads, h_begin + heads_per_warp);
  const int half = p.rot_dim >> 1;
  const int hh = p.hd >> 1;
  constexpr int kMaxAngles = 4;                // half <= 128
  float sn_r[kMaxAngles], cs_r[kMaxAngles];
  // Fast path (head_dim 128, whole head rotated, halves layout): a lane holds 4 consecutive elements of the
  // head (one 8-byte load and store per head), its rotation partner sits 16 lanes away.
  const bool fast = p.layout == 0 && p.rot_dim == p.hd && p.hd == 128;
  if (h_begin < p.hq + p.hkv) {
    const float pos = static_cast<float>(p.positions[tok]);
#pragma unroll
    for (int a = 0; a < kMaxAngles; ++a) {
      const int i = fast ? 4 * (lane & 15) + a : lane + 32 * a;
      sn_r[a] = 0.f;
      cs_r[a] = 1.f;
      if (i < half) {
        sincosf(pos * p.inv_freq[i], &sn_r[a], &cs_r[a]);
        sn_r[a] *= p.attn_factor;
        cs_r[a] *= p.attn_factor;
      }
    }
  }
  const long long slot = p.slot_mapping[tok];
  // negative = padding row (no KV write); the checking build reports a slot past the cache instead of dropping it
  if (slot >= p.num_slots) (void)ZB_BC_OK(slot, p.num_slots, kKernelRopeKvWrite, 1);
  const bool slot_ok = slot >= 0 && slot < p.num_slots;
  for (int h = h_begin; h < h_end; ++h) {
    const __nv_bfloat16* __restrict__ src = p.qkv + static_cast<size_t>(tok) * p.qkv_stride + static_cast<size_t>(h) * p.hd;
    const bool is_q = h < p.hq;
    const bool is_k = !is_q && h < p.hq + p.hkv;
    __nv_bfloat16* __restrict__ dst;
    if (is_q) {
      dst = p.q_out + (static_cast<size_t>(tok) * p.hq + h) * p.hd;
    } else {
      if (!slot_ok) continue;
      const int kvh = is_k ? h - p.hq : h - p.hq - p.hkv;
      __nv_bfloat16* cache = is_k ? p.k_cache : p.v_cache;
      dst = cache + (static_cast<size_t>(slot) * p.hkv + kvh) * p.hd;
    }
    if (!is_q && !is_k) {
      // V: plain copy, 16 bytes per lane per step
      const uint4* s4 = reinterpret_cast<const uint4*>(src);
      uint4* d4 = reinterpret_cast<uint4*>(dst);
      for (int i = lane; i < p.hd / 8; i += 32) d4[i] = s4[i];
      continue;
    }
    const __nv_bfloat16* nw = is_q ? p.q_norm_w : p.k_norm_w;
    if (fast) {
      const uint2 raw = reinterpret_cast<const uint2*>(src)[lane];
      const float2 lo = zb_unpack_bf16x2(raw.x), hi = zb_unpack_bf16x2(raw.y);
      float v[4] = {lo.x, lo.y, hi.x, hi.y};
      if (nw) {
        const float ss = zb_warp_sum(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3]);
        const float inv = rsqrtf(ss / 128.f + p.norm_eps);
        const uint2 graw = reinterpret_cast<const uint2*>(nw)[lane];
        const float2 g0 = zb_unpack_bf16x2(graw.x), g1 = zb_unpack_bf16x2(graw.y);
        const float g[4] = {g0.x, g0.y, g1.x, g1.y};
#pragma unroll
        for (int j = 0; j < 4; ++j)      // normalised in f32, rounded to the activation dtype before rotating (as the reference does)
          v[j] = __bfloat162float(__float2bfloat16(v[j] * inv * (g[j] + (p.norm_unit_offset ? 1.f : 0.f))));
      }
      float o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float partner = __shfl_xor_sync(0xffffffffu, v[j], 16);
        o[j] = lane < 16 ? v[j] * cs_r[j] - partner * sn_r[j] : v[j] * cs_r[j] + partner * sn_r[j];
      }
      reinterpret_cast<uint2*>(dst)[lane] = make_uint2(zb_pack_bf16x2(o[0], o[1]), zb_pack_bf16x2(o[2], o[3]));
      continue;
    }
    float inv_rms = 1.f;
    if (nw) {
      float ss = 0.f;
      for (int i = lane; i < p.hd; i += 32) {
        const float v = __bfloat162float(src[i]);
        ss += v * v;
      }
      ss = zb_warp_sum(ss);
      inv_rms = rsqrtf(ss / static_cast<float>(p.hd) + p.norm_eps);
    }
    auto load = [&](int i) -> float {
      float v = __bfloat162float(src[i]);
      if (nw) {
        float g = __bfloat162float(nw[i]);
        if (p.norm_unit_offset) g += 1.f;
        // the reference normalises in f32 and rounds to the activation dtype before rotating
        v = __bfloat162float(__float2bfloat16(v * inv_rms * g));
      }
      return v;
    };
#pragma unroll
    for (int a = 0; a < kMaxAngles; ++a) {
      const int i = lane + 32 * a;
      if (i >= half) continue;
      const int i0 = p.layout == 1 ? 2 * i : i;
      const int i1 = p.layout == 0 ? i + half : (p.layout == 1 ? 2 * i + 1 : i + hh);
      const float x = load(i0), y = load(i1);
      dst[i0] = __float2bfloat16(x * cs_r[a] - y * sn_r[a]);
      dst[i1] = __float2bfloat16(y * cs_r[a] + x * sn_r[a]);
    }
    if (p.rot_dim < p.hd) {
      for (int i = lane; i < p.hd; i += 32) {
        const bool rotated = p.layout == 2 ? ((i < half) || (i >= hh && i < hh + half)) : (i < p.rot_dim);
        if (!rotated) dst[i] = __float2bfloat16(load(i));
      }
    }
  }
}

// The halves layout for heads of 64, 128 or 256 whose rows start on 16 bytes.  A CTA takes one token: its angles go to shared memory once,
// then every thread has two 16-byte pieces of one head - the two that rotate into each other, or two behind the rotated part, or two of
// a value head - so all loads of a token are in flight at once (the kernel above walks a warp's heads one after the other, each load
// behind the store before it).  A head's hd / 16 threads are neighbours in a warp and add up its sum of squares.
// 8192 tokens of 32 + 8 + 8 heads: 64 columns a head 23 us (85), 128 51 (78); 16 + 4 + 4 heads of 256, normalised, 64 columns turned 57
// (107); 32 tokens 2.2 (3.1).
ZB_DEVICE void rope_unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = zb_unpack_bf16x2(w[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
ZB_DEVICE uint4 rope_pack8(const float (&f)[8]) {
  return make_uint4(zb_pack_bf16x2(f[0], f[1]), zb_pack_bf16x2(f[2], f[3]), zb_pack_bf16x2(f[4], f[5]), zb_pack_bf16x2(f[6], f[7]));
}

template <int HD>
__global__ void __launch_bounds__(512) zb_rope_rows_kernel(const RopeParams p) {
  constexpr int kLanes = HD / 16;
  __shared__ __align__(16) float sn[HD / 2], cs[HD / 2];
  zb_pdl_launch();
  zb_pdl_wait();
  const int tok = blockIdx.x, half = p.rot_dim >> 1;
  const float pos = static_cast<float>(p.positions[tok]);
  const long long slot = p.slot_mapping[tok];
  // negative = padding row (no KV write); the checking build reports a slot past the cache instead of dropping it
  if (slot >= p.num_slots) (void)ZB_BC_OK(slot, p.num_slots, kKernelRopeKvWrite, 1);
  const bool slot_ok = slot >= 0 && slot < p.num_slots;
  const int from = static_cast<int>(blockIdx.y) * p.share, units = min(from + p.share, (p.hq + 2 * p.hkv) * kLanes);
  const int rounded = from + ((units - from + 31) & ~31);      // a warp goes through the loop as a whole
  bool first = true;
  for (int u0 = from + threadIdx.x; u0 < rounded; u0 += blockDim.x) {
    const bool in = u0 < units;
    const int u = in ? u0 : units - 1, h = u / kLanes, j = u - h * kLanes;
    const bool is_q = h < p.hq, is_k = !is_q && h < p.hq + p.hkv;
    const bool turns = (is_q || is_k) && j < half / 8;
    const int v0 = turns ? j : half / 4 + 2 * (j - half / 8), v1 = turns ? j + half / 8 : v0 + 1;      // 16-byte pieces of the head
    const int a0 = is_q || is_k ? v0 : 2 * j, a1 = is_q || is_k ? v1 : 2 * j + 1;
    const uint4* src = reinterpret_cast<const uint4*>(p.qkv + static_cast<size_t>(tok) * p.qkv_stride + static_cast<size_t>(h) * HD);
    uint4 x0 = src[a0], x1 = src[a1];
    if (first) {                                     // the angles, while the loads are on their way
      first = false;
      for (int i = threadIdx.x; i < half; i += blockDim.x) {
        float s_, c_;
        sincosf(pos * p.inv_freq[i], &s_, &c_);
        sn[i] = s_ * p.attn_factor;
        cs[i] = c_ * p.attn_factor;
      }
      __syncthreads();
    }
    if (is_q || is_k) {
      float f0[8], f1[8];
      rope_unpack8(x0, f0);
      rope_unpack8(x1, f1);
      const __nv_bfloat16* nw = is_q ? p.q_norm_w : p.k_norm_w;
      // q and k heads lie in front of the value heads: the lanes of one head agree, and a warp whose last lanes have values still adds
      // up groups of kLanes
      if (nw != nullptr) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += f0[i] * f0[i] + f1[i] * f1[i];
        const uint32_t group = ((1ull << kLanes) - 1ull) << ((threadIdx.x & 31) / kLanes * kLanes);
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(group, ss, o);
        const float inv = rsqrtf(ss / static_cast<float>(HD) + p.norm_eps), one = p.norm_unit_offset ? 1.f : 0.f;
        float g0[8], g1[8];
        rope_unpack8(reinterpret_cast<const uint4*>(nw)[a0], g0);
        rope_unpack8(reinterpret_cast<const uint4*>(nw)[a1], g1);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          // normalised in f32, rounded to the activation dtype before rotating (as the reference does)
          f0[i] = __bfloat162float(__float2bfloat16(f0[i] * inv * (g0[i] + one)));
          f1[i] = __bfloat162float(__float2bfloat16(f1[i] * inv * (g1[i] + one)));
        }
      }
      if (turns) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float c_ = cs[8 * j + i], s_ = sn[8 * j + i], x = f0[i], y = f1[i];
          f0[i] = x * c_ - y * s_;
          f1[i] = y * c_ + x * s_;
        }
      }
      x0 = rope_pack8(f0);
      x1 = rope_pack8(f1);
    }
    if (!in || (!is_q && !slot_ok)) continue;
    const int kvh = h - p.hq - (is_k ? 0 : p.hkv);
    __nv_bfloat16* dst = is_q ? p.q_out + (static_cast<size_t>(tok) * p.hq + h) * HD
                              : (is_k ? p.k_cache : p.v_cache) + (static_cast<size_t>(slot) * p.hkv + kvh) * HD;
    reinterpret_cast<uint4*>(dst)[a0] = x0;
    reinterpret_cast<uint4*>(dst)[a1] = x1;
  }
}

// ---------------------------------------------------------------- SwiGLU
// out[t, f] = silu(gu[t, f]) * gu[t, F + f]
__global__ void __launch_bounds__(256) zb_swiglu_kernel(const __nv_bfloat16* __restrict__ gu,
                                                        __nv_bfloat16* __restrict__ out,
                                                        long long total_vec, int f_vec) {
  zb_pdl_launch();
  zb_pdl_wait();
  for (long long idx = blockIdx.x * 256ll + threadIdx.x; idx < total_vec;
       idx += static_cast<long long>(gridDim.x) * 256) {
    const long long t = idx / f_vec;
    const int fv = static_cast<int>(idx % f_vec);
    const uint4* row = reinterpret_cast<const uint4*>(gu) + t * (2ll * f_vec);
    const uint4 g = row[fv];
    const uint4 u = row[f_vec + fv];
    const uint32_t gg[4] = {g.x, g.y, g.z, g.w}, uu[4] = {u.x, u.y, u.z, u.w};
    uint32_t oo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 a = zb_unpack_bf16x2(gg[j]);
      const float2 b = zb_unpack_bf16x2(uu[j]);
      const float s0 = a.x / (1.f + __expf(-a.x));
      const float s1 = a.y / (1.f + __expf(-a.y));
      oo[j] = zb_pack_bf16x2(s0 * b.x, s1 * b.y);
    }
    reinterpret_cast<uint4*>(out)[idx] = make_uint4(oo[0], oo[1], oo[2], oo[3]);
  }
}

// ---------------------------------------------------------------- embedding
__global__ void __launch_bounds__(128) zb_embedding_kernel(const int32_t* __restrict__ ids,
                                                           const __nv_bfloat16* __restrict__ table,
                                                           __nv_bfloat16* __restrict__ out, int tokens,
                                                           int d, int vocab) {
  zb_pdl_launch();
  zb_pdl_wait();
  const int t = blockIdx.x;
  if (t >= tokens) return;
  int id = ids[t];
  if (id < 0 || id >= vocab) {
    (void)ZB_BC_OK(id, vocab, kKernelEmbedding, 1);      // the checking build reports the id; both builds read row 0
    id = 0;
  }
  const uint4* src = reinterpret_cast<const uint4*>(table + static_cast<size_t>(id) * d);
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * d);
  for (int i = threadIdx.x; i < d / 8; i += 128) dst[i] = src[i];
}

// ---------------------------------------------------------------- argmax
ZB_DEVICE void st_cluster(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// CTAs of a cluster that share a row of `vocab` logits: as many as keep the chip full without a second wave (at most `ctas`; 1024 threads a
// CTA, two CTAs an SM), at least `least` logits each.  32 rows of 128256 by one CTA a row leave four fifths of the SMs idle.  As a power
// of two.
int row_cluster(int rows, int vocab, int ctas, int least) {
  int log2 = 3;
  while (log2 > 0 && ((static_cast<long long>(rows) << log2) > ctas || (vocab >> log2) < least)) --log2;
  return log2;
}

// First index of the row maximum (ties -> lowest index, NaN ignored), f32 logits.
__global__ void __launch_bounds__(1024) zb_argmax_f32_kernel(const float* __restrict__ logits,
                                                             int32_t* __restrict__ out, int vocab,
                                                             long long stride) {
  zb_pdl_launch();
  zb_pdl_wait();
  float best;
  int bi;
  zb_block_argmax_1024(logits + static_cast<size_t>(blockIdx.x) * stride, vocab, best, bi);
  if (threadIdx.x == 0) out[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;
}

// The same with a cluster per row, each CTA a slice of it.  One row of 128256: 4.0 us (one CTA: 8.1); 32 rows 5.7 (8.4).
__global__ void __launch_bounds__(1024) zb_argmax_cluster_kernel(const float* __restrict__ logits,
                                                                 int32_t* __restrict__ out, int vocab,
                                                                 long long stride, int log2_ctas) {
  __shared__ float all_v[8];
  __shared__ int all_i[8];
  const int ctas = 1 << log2_ctas, rank = blockIdx.x & (ctas - 1), row = blockIdx.x >> log2_ctas;
  zb_cluster_arrive();                               // every CTA runs before another one writes to its shared memory
  zb_pdl_launch();
  zb_pdl_wait();
  const int per = (vocab + ctas - 1) >> log2_ctas, from = min(rank * per, vocab), n = min(per, vocab - from);
  float best;
  int bi;
  zb_block_argmax_1024(logits + static_cast<size_t>(row) * stride + from, n, best, bi);
  if (bi != 0x7fffffff) bi += from;
  zb_cluster_wait();
  if (threadIdx.x == 0) {
    st_cluster(zb_mapa(zb_smem_u32(&all_v[rank]), 0), __float_as_uint(best));
    st_cluster(zb_mapa(zb_smem_u32(&all_i[rank]), 0), static_cast<uint32_t>(bi));
  }
  zb_cluster_arrive();
  zb_cluster_wait();
  if (rank != 0 || threadIdx.x != 0) return;
  for (int c = 1; c < ctas; ++c) zb_argmax_merge(best, bi, all_v[c], all_i[c]);
  out[row] = bi == 0x7fffffff ? 0 : bi;
}

// ---------------------------------------------------------------- top-k + Gumbel-max
// Per row: select the k largest logits (k <= 128) with a 4-pass radix select on the
// order-preserving integer image of the floats, then draw one of them with the
// Gumbel-max trick at the given temperature (sampleTokens, zml/nn.zig:2007-2033).
// Also writes the selected (value, index) pairs, sorted descending, when asked.
ZB_DEVICE uint32_t float_key(float f) {
  const uint32_t u = __float_as_uint(f + 0.f);       // one zero
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

ZB_DEVICE float uniform01(uint64_t seed, uint64_t idx) {
  // splitmix64 -> 23 mantissa bits -> [1, 2) - 1, as the reference's Rng.uniform does
  uint64_t z = seed + 0x9e3779b97f4a7c15ull * (idx + 1);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  const uint32_t mant = static_cast<uint32_t>(z >> 41);
  return __uint_as_float(0x3f800000u | mant) - 1.f;
}

constexpr int kMaxTopK = 128;
constexpr int kCands = 2048;

// A candidate as one number: the larger, the further in front.  Above, the order of the floats (one zero, NaN above infinity), below, the
// complement of the index in the row: among equal logits the lower index goes first.
ZB_DEVICE uint64_t cand_of(uint32_t key, int idx) { return static_cast<uint64_t>(key) << 32 | static_cast<uint32_t>(~idx); }
ZB_DEVICE int cand_index(uint64_t c) { return ~static_cast<int>(static_cast<uint32_t>(c)); }
ZB_DEVICE float cand_value(uint64_t c) {
  const uint32_t key = static_cast<uint32_t>(c >> 32);
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}
struct TopkShared {
  uint64_t cand[kCands];
  uint64_t merge[8 * kMaxTopK];                      // CTA 0: every CTA's best, sorted
  uint32_t hist[256];
  uint32_t top[160];                                 // the warps' largest maxima
  uint32_t prefix, remaining, n, bound;
};

// The k largest of row[0, len) into sh.cand (any order; equal ones: the lowest indices), sh.n of them.  4-pass radix select; for
// slices whose candidates do not fit the short way below (many equal logits).
ZB_DEVICE void radix_topk(TopkShared& sh, const float* __restrict__ row, int len, int base, int k) {
  if (threadIdx.x == 0) {
    sh.prefix = 0;
    sh.remaining = k;
    sh.n = 0;
  }
  __syncthreads();
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    for (int i = threadIdx.x; i < 256; i += 1024) sh.hist[i] = 0;
    __syncthreads();
    const uint32_t prefix = sh.prefix;
    const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
    for (int i = threadIdx.x; i < len; i += 1024) {
      const uint32_t key = float_key(row[i]);
      if ((key & mask) == prefix) atomicAdd(&sh.hist[(key >> shift) & 0xff], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t rem = sh.remaining;
      int b = 255;
      for (; b > 0; --b) {
        if (sh.hist[b] >= rem) break;
        rem -= sh.hist[b];
      }
      sh.prefix = prefix | (static_cast<uint32_t>(b) << shift);
      sh.remaining = rem;
    }
    __syncthreads();
  }
  const uint32_t kth = sh.prefix;                    // key of the k-th largest value
  const int ties = static_cast<int>(sh.remaining);   // how many elements equal to it belong to the k largest
  for (int i = threadIdx.x; i < len; i += 1024) {
    const uint32_t key = float_key(row[i]);
    if (key > kth) {
      sh.cand[atomicAdd(&sh.n, 1u)] = cand_of(key, base + i);
    }
  }
  __syncthreads();
  const int greater = static_cast<int>(sh.n), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int taken = 0;                                     // ties in the order of their indices
  for (int i0 = 0; i0 < len && taken < ties; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    const bool tie = i < len && float_key(row[i]) == kth;
    const uint32_t ballot = __ballot_sync(0xffffffffu, tie);
    if (lane == 0) sh.top[warp] = __popc(ballot);
    __syncthreads();
    int before = taken, all = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += sh.top[w];
      all += sh.top[w];
    }
    before += __popc(ballot & ((1u << lane) - 1u));
    if (tie && before < ties) sh.cand[greater + before] = cand_of(kth, base + i);
    taken += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) sh.n = greater + min(taken, ties);
  __syncthreads();
}

// A cluster per row, each CTA a slice of it.  `bound`, the k-th largest among the few largest of the maxima that each warp's threads saw,
// is at most the k-th largest of the slice, and little less.  So a slice is read twice (the second time from L2) instead of five times
// with a shared-memory atomic per element; its candidates - not many more than k - are ranked by counting, the best k go to CTA 0, which
// merges all CTAs' and draws.  128256 logits, k = 40: one row 10 us, 32 rows 17 (one CTA per row and radix select: 85), 128 rows 19.
__global__ void __launch_bounds__(1024) zb_topk_sample_kernel(
    const float* __restrict__ logits, int32_t* __restrict__ out_token, float* __restrict__ topk_vals,
    int32_t* __restrict__ topk_idx, int rows, int vocab, long long stride, int k, float temperature,
    uint64_t seed, uint64_t step, const unsigned long long* __restrict__ dev_rng, int log2_ctas) {
  __shared__ TopkShared sh;
  __shared__ int merge_n[8];
  const int ctas = 1 << log2_ctas, rank = blockIdx.x & (ctas - 1), row_i = blockIdx.x >> log2_ctas, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (ctas > 1) zb_cluster_arrive();                 // every CTA runs before another one writes to its shared memory
  zb_pdl_launch();
  zb_pdl_wait();
  if (dev_rng != nullptr) {
    // seed and draw counter live on the device: a captured CUDA graph then samples with fresh noise at every
    // replay (the counter is advanced by zb_decode_advance) and with whatever seed was copied in before it
    seed = dev_rng[0];
    step += dev_rng[1];
  }
  const float* row = logits + static_cast<size_t>(row_i) * stride;
  const int per = (((vocab + ctas - 1) >> log2_ctas) + 3) & ~3, from = min(rank * per, vocab), len = min(per, vocab - from);
  const float* part = row + from;
  const bool vec = len >= 4096 && (reinterpret_cast<uintptr_t>(part) & 15) == 0;
  auto each = [&](auto&& f) {                        // f(index in the slice, logit), every element once
    int done = 0;
    if (vec) {
      done = len & ~3;
#pragma unroll 4
      for (int i = 4 * threadIdx.x; i < done; i += 4096) {
        const float4 v = *reinterpret_cast<const float4*>(part + i);
        f(i, v.x);
        f(i + 1, v.y);
        f(i + 2, v.z);
        f(i + 3, v.w);
      }
    }
    for (int i = done + threadIdx.x; i < len; i += 1024) f(i, part[i]);
  };
  uint32_t left = 0;                                 // below the key of every number
  each([&](int, float v) { left = max(left, float_key(v)); });
  const int per_warp = (k + 31) / 32 + 1;            // 2 .. 5 of a warp's 32 maxima: at least k in all
  for (int i = 0; i < per_warp; ++i) {
    const uint32_t best = __reduce_max_sync(0xffffffffu, left);
    const uint32_t who = __ballot_sync(0xffffffffu, left == best);
    if (lane == __ffs(who) - 1) left = 0;
    if (lane == 0) sh.top[i * 32 + warp] = best;
  }
  if (threadIdx.x == 0) sh.n = 0;
  __syncthreads();
  if (threadIdx.x < 32 * per_warp) {
    const uint32_t mine = sh.top[threadIdx.x];
    int ahead = 0;
    for (int j = 0; j < 32 * per_warp; ++j) ahead += sh.top[j] > mine || (sh.top[j] == mine && j < static_cast<int>(threadIdx.x)) ? 1 : 0;
    if (ahead == k - 1) sh.bound = mine;
  }
  __syncthreads();
  const uint32_t bound = sh.bound;
  each([&](int i, float v) {
    const uint32_t key = float_key(v);
    if (key >= bound) {
      const uint32_t slot = atomicAdd(&sh.n, 1u);
      if (slot < kCands) sh.cand[slot] = cand_of(key, from + i);
    }
  });
  __syncthreads();
  if (sh.n > 1024u) {
    __syncthreads();                                 // all threads have read n
    radix_topk(sh, part, len, from, min(k, len));
  }
  const int n_c = static_cast<int>(sh.n);
  int place = kMaxTopK;
  uint64_t mine = 0;
  if (static_cast<int>(threadIdx.x) < n_c) {
    mine = sh.cand[threadIdx.x];
    place = 0;
#pragma unroll 4
    for (int j = 0; j < n_c; ++j) place += sh.cand[j] > mine ? 1 : 0;
  }
  if (ctas > 1) zb_cluster_wait();
  if (place < k) {
    if (ctas > 1) {
      const uint32_t to = zb_mapa(zb_smem_u32(&sh.merge[rank * k + place]), 0);
      st_cluster(to, static_cast<uint32_t>(mine));
      st_cluster(to + 4, static_cast<uint32_t>(mine >> 32));
    } else {
      sh.merge[place] = mine;
    }
  }
  if (threadIdx.x == 0) {
    if (ctas > 1) st_cluster(zb_mapa(zb_smem_u32(&merge_n[rank]), 0), static_cast<uint32_t>(min(n_c, k)));
    else merge_n[0] = min(n_c, k);
  }
  if (ctas > 1) {
    zb_cluster_arrive();
    zb_cluster_wait();
    if (rank != 0) return;
  } else {
    __syncthreads();
  }
  // the k best of all CTAs'
  __shared__ float sort_v[kMaxTopK];
  __shared__ int sort_i[kMaxTopK];
  int n = 0;
  for (int c = 0; c < ctas; ++c) n += merge_n[c];
  n = min(n, k);
  for (int t = threadIdx.x; t < ctas * k; t += 1024) {
    const int c0 = t / k;
    int at = t - c0 * k;
    if (at >= merge_n[c0]) continue;
    const uint64_t c1 = sh.merge[t];
    for (int c = 0; c < ctas; ++c) {
      if (c == c0) continue;
      int lo = 0, hi = merge_n[c];                   // how many of CTA c go before
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sh.merge[c * k + mid] > c1) lo = mid + 1; else hi = mid;
      }
      at += lo;
    }
    if (at < k) {
      sort_v[at] = cand_value(c1);
      sort_i[at] = cand_index(c1);
    }
  }
  __syncthreads();
  if (topk_vals && threadIdx.x < k) {
    topk_vals[static_cast<size_t>(row_i) * k + threadIdx.x] = threadIdx.x < n ? sort_v[threadIdx.x] : -INFINITY;
    topk_idx[static_cast<size_t>(row_i) * k + threadIdx.x] = threadIdx.x < n ? sort_i[threadIdx.x] : 0;
  }
  if (threadIdx.x < 32) {
    float best = -INFINITY;
    int bi = n > 0 ? sort_i[0] : 0;
    for (int j = threadIdx.x; j < n; j += 32) {
      float score = sort_v[j];
      if (temperature > 0.f && k > 1) {
        const float u = fmaxf(uniform01(seed, (step * rows + row_i) * kMaxTopK + j), 1e-20f);
        score = score / temperature - __logf(-__logf(u));
      }
      if (score > best) {
        best = score;
        bi = sort_i[j];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best) {
        best = ov;
        bi = oi;
      }
    }
    if (threadIdx.x == 0) out_token[row_i] = bi;
  }
}

// ---------------------------------------------------------------- decode bookkeeping
// After sampling: feed the sampled token back as the next input, advance position and
// length, compute the KV slot of the new position from the block table, and append the
// token to the on-device history so that the host can read tokens in batches.
__global__ void zb_decode_advance_kernel(const int32_t* __restrict__ sampled, int32_t* __restrict__ ids,
                                         int32_t* __restrict__ positions, int32_t* __restrict__ seq_lens,
                                         int32_t* __restrict__ slot_mapping,
                                         const int32_t* __restrict__ block_table, int32_t* __restrict__ history,
                                         int32_t* __restrict__ step_counter, int batch, int max_pages,
                                         int page_size, int history_stride, int history_rows) {
  zb_pdl_launch();
  zb_pdl_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  const int step = *step_counter;
  if (b < batch) {
    const int tok = sampled[b];
    ids[b] = tok;
    const int pos = positions[b] + 1;
    positions[b] = pos;
    seq_lens[b] = pos + 1;
    const int pg = pos / page_size;
    int page = pg < max_pages ? block_table[static_cast<size_t>(b) * max_pages + pg] : -1;
    if (page >= 0 && !ZB_BC_OK(page, ZB_BC_PAGES, kKernelDecodeAdvance, 1)) page = -1;
    slot_mapping[b] = page >= 0 ? page * page_size + pos % page_size : -1;
    if (step < history_rows) history[static_cast<size_t>(step) * history_stride + b] = tok;
  }
}

// Runs after the kernel above on the same stream, so every block has read the old value.
__global__ void zb_counter_inc_kernel(int32_t* c, unsigned long long* rng) {
  zb_pdl_launch();
  zb_pdl_wait();
  *c += 1;
  if (rng != nullptr) rng[1] += 1ull;      // one more draw of the sampler (see zb_topk_sample_rng)
}

__global__ void zb_u64_add_kernel(unsigned long long* p, unsigned long long n) {
  zb_pdl_launch();
  zb_pdl_wait();
  *p += n;
}

}  // namespace

extern "C" {

int zb_rmsnorm(const void* x, const void* residual, const void* w, void* out, void* residual_out,
               int rows, int d, long long x_stride, long long out_stride, float eps,
               int unit_offset, void* stream) {
  if (rows <= 0) return 0;
  if (d % 8 != 0 || x_stride % 8 != 0 || out_stride % 8 != 0) return -40;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int nvec = d / 8;
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto R = reinterpret_cast<const __nv_bfloat16*>(residual);
  auto W = reinterpret_cast<const __nv_bfloat16*>(w);
  auto O = reinterpret_cast<__nv_bfloat16*>(out);
  auto RO = reinterpret_cast<__nv_bfloat16*>(residual_out);
  if (nvec <= 256) zb_launch(zb_rmsnorm_kernel<1>, dim3(rows), dim3(256), 0, s, X, R, W, O, RO, rows, d, x_stride, out_stride, eps, unit_offset);
  else if (nvec <= 512) zb_launch(zb_rmsnorm_kernel<2>, dim3(rows), dim3(256), 0, s, X, R, W, O, RO, rows, d, x_stride, out_stride, eps, unit_offset);
  else if (nvec <= 1024) zb_launch(zb_rmsnorm_kernel<4>, dim3(rows), dim3(256), 0, s, X, R, W, O, RO, rows, d, x_stride, out_stride, eps, unit_offset);
  else if (nvec <= 2048) zb_launch(zb_rmsnorm_kernel<8>, dim3(rows), dim3(256), 0, s, X, R, W, O, RO, rows, d, x_stride, out_stride, eps, unit_offset);
  else return -41;
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}

int zb_rope_kvwrite(const void* qkv, void* q_out, void* k_cache, void* v_cache,
                    const int32_t* positions, const int32_t* slot_mapping, const float* inv_freq,
                    const void* q_norm_w, const void* k_norm_w, long long qkv_stride, int tokens,
                    int hq, int hkv, int hd, int rot_dim, int layout, int page_size,
                    long long num_slots, float attn_factor, float norm_eps, int norm_unit_offset,
                    void* stream) {
  if (tokens <= 0) return 0;
  if (hd % 8 != 0 || rot_dim % 2 != 0 || rot_dim > hd) return -42;
  RopeParams p;
  p.qkv = reinterpret_cast<const __nv_bfloat16*>(qkv);
  p.q_out = reinterpret_cast<__nv_bfloat16*>(q_out);
  p.k_cache = reinterpret_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = reinterpret_cast<__nv_bfloat16*>(v_cache);
  p.positions = positions;
  p.slot_mapping = slot_mapping;
  p.inv_freq = inv_freq;
  p.q_norm_w = reinterpret_cast<const __nv_bfloat16*>(q_norm_w);
  p.k_norm_w = reinterpret_cast<const __nv_bfloat16*>(k_norm_w);
  p.qkv_stride = qkv_stride;
  p.tokens = tokens;
  p.hq = hq;
  p.hkv = hkv;
  p.hd = hd;
  p.rot_dim = rot_dim;
  p.layout = layout;
  p.page_size = page_size;
  p.attn_factor = attn_factor;
  p.norm_eps = norm_eps;
  p.norm_unit_offset = norm_unit_offset;
  p.num_slots = num_slots;
  if (rot_dim / 2 > 128) return -46;
  const auto at16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (layout == 0 && rot_dim % 16 == 0 && (hd == 64 || hd == 128 || hd == 256) && qkv_stride % 8 == 0 && at16(qkv) && at16(q_out) && at16(k_cache) &&
      at16(v_cache) && at16(q_norm_w) && at16(k_norm_w)) {
    // Few tokens of more pieces than a CTA has threads: several CTAs a token, which a second turn of one makes wait (8 tokens of 64 + 8 + 8 heads
    // of 128: 3.7 us in two turns).
    const int units = (hq + 2 * hkv) * (hd / 16), parts = tokens <= 64 ? (units + 511) / 512 : 1;
    p.share = ((units + parts - 1) / parts + 31) / 32 * 32;
    const int threads = std::min(512, p.share);
    const auto kernel = hd == 64 ? zb_rope_rows_kernel<64> : (hd == 128 ? zb_rope_rows_kernel<128> : zb_rope_rows_kernel<256>);
    zb_launch(kernel, dim3(tokens, parts), dim3(threads), 0, reinterpret_cast<cudaStream_t>(stream), p);
    zb_count_launch(1);
    return static_cast<int>(cudaGetLastError());
  }
  // enough warps to fill the SMs a few times; beyond that, more heads per warp (shared sin / cos)
  const int heads = hq + 2 * hkv;
  int heads_per_warp = static_cast<int>(static_cast<long long>(tokens) * heads / 2368);
  heads_per_warp = heads_per_warp < 1 ? 1 : (heads_per_warp > 8 ? 8 : heads_per_warp);      // a warp's heads run one after the other
  const long long warps = static_cast<long long>(tokens) * ((heads + heads_per_warp - 1) / heads_per_warp);
  const int blocks = static_cast<int>((warps + 3) / 4);
  zb_launch(zb_rope_kvwrite_kernel, dim3(blocks), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream), p, heads_per_warp);
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}

int zb_swiglu(const void* gate_up, void* out, long long tokens, int f, void* stream) {
  if (tokens <= 0) return 0;
  if (f % 8 != 0) return -43;
  const long long total_vec = tokens * (f / 8);
  long long blocks = (total_vec + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  zb_launch(zb_swiglu_kernel, dim3(static_cast<int>(blocks)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), 
      reinterpret_cast<const __nv_bfloat16*>(gate_up), reinterpret_cast<__nv_bfloat16*>(out), total_vec,
      f / 8);
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}

int zb_embedding(const int32_t* ids, const void* table, void* out, int tokens, int d, int vocab,
                 void* stream) {
  if (tokens <= 0) return 0;
  if (d % 8 != 0) return -44;
  zb_launch(zb_embedding_kernel, dim3(tokens), dim3(128), 0, reinterpret_cast<cudaStream_t>(stream), 
      ids, reinterpret_cast<const __nv_bfloat16*>(table), reinterpret_cast<__nv_bfloat16*>(out), tokens, d,
      vocab);
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}

int zb_argmax_f32(const float* logits, int32_t* out, int rows, int vocab, long long stride,
                  void* stream) {
  if (rows <= 0) return 0;
  // A cluster's two barriers take 0.6 us, which short rows do not give back (1 CTA / cluster, us: a row of 16000 3.2 / 3.6, of 32000 3.8 / 3.4), nor
  // rows of medium length that fill the SMs by themselves (64 of 32000: 4.1 / 4.6).
  const int log2 = vocab < 32000 || (vocab < 65536 && 4 * static_cast<long long>(rows) > zb_num_sms()) ? 0 : row_cluster(rows, vocab, 2 * zb_num_sms(), 8000);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (log2 == 0) zb_launch(zb_argmax_f32_kernel, dim3(rows), dim3(1024), 0, s, logits, out, vocab, stride);
  else zb_launch_cluster(zb_argmax_cluster_kernel, dim3(rows << log2), dim3(1024), 0, s, 1 << log2, logits, out, vocab, stride, log2);
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}

// `dev_rng` (may be null): two u64 in device memory, {seed, draws so far}; when given, the seed comes from there
// and the draw counter is added to `step`.
int zb_topk_sample_rng(const float* logits, int32_t* out_token, float* topk_vals, int32_t* topk_idx,
                       int rows, int vocab, long long stride, int k, float temperature,
                       unsigned long long seed, unsigned long long step, const unsigned long long* dev_rng, void* stream) {
  if (rows <= 0) return 0;
  if (k < 1 || k > kMaxTopK) return -45;
  const int log2 = row_cluster(rows, vocab, 2 * zb_num_sms(), 4096);
  zb_launch_cluster(zb_topk_sample_kernel, dim3(rows << log2), dim3(1024), 0, reinterpret_cast<cudaStream_t>(stream), 1 << log2, logits, out_token, topk_vals,
                    topk_idx, rows, vocab, stride, k, temperature, static_cast<uint64_t>(seed), static_cast<uint64_t>(step), dev_rng, log2);
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}

int zb_topk_sample(const float* logits, int32_t* out_token, float* topk_vals, int32_t* topk_idx,
                   int rows, int vocab, long long stride, int k, float temperature,
                   unsigned long long seed, unsigned long long step, void* stream) {
  return zb_topk_sample_rng(logits, out_token, topk_vals, topk_idx, rows, vocab, stride, k, temperature, seed, step, nullptr,
                            stream);
}

// Adds `n` to a u64 in device memory, in stream order (the draw counter of the sampler).
int zb_u64_add(unsigned long long* p, unsigned long long n, void* stream) {
  zb_launch(zb_u64_add_kernel, dim3(1), dim3(1), 0, reinterpret_cast<cudaStream_t>(stream), p, n);
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}

// Feeds sampled tokens back for the next decode step (see the kernel's comment).
int zb_decode_advance_rng(const int32_t* sampled, int32_t* ids, int32_t* positions, int32_t* seq_lens,
                          int32_t* slot_mapping, const int32_t* block_table, int32_t* history,
                          int32_t* step_counter, int batch, int max_pages, int page_size,
                          int history_stride, int history_rows, unsigned long long* rng, void* stream);

int zb_decode_advance(const int32_t* sampled, int32_t* ids, int32_t* positions, int32_t* seq_lens,
                      int32_t* slot_mapping, const int32_t* block_table, int32_t* history,
                      int32_t* step_counter, int batch, int max_pages, int page_size,
                      int history_stride, int history_rows, void* stream) {
  return zb_decode_advance_rng(sampled, ids, positions, seq_lens, slot_mapping, block_table, history, step_counter, batch,
                               max_pages, page_size, history_stride, history_rows, nullptr, stream);
}

// The same, and the sampler's draw counter rng[1] (see zb_topk_sample_rng) goes up by one.
int zb_decode_advance_rng(const int32_t* sampled, int32_t* ids, int32_t* positions, int32_t* seq_lens,
                          int32_t* slot_mapping, const int32_t* block_table, int32_t* history,
                          int32_t* step_counter, int batch, int max_pages, int page_size,
                          int history_stride, int history_rows, unsigned long long* rng, void* stream) {
  if (batch <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  zb_launch(zb_decode_advance_kernel, dim3((batch + 127) / 128), dim3(128), 0, s, sampled, ids, positions, seq_lens,
                                                             slot_mapping, block_table, history,
                                                             step_counter, batch, max_pages, page_size,
                                                             history_stride, history_rows);
  zb_launch(zb_counter_inc_kernel, dim3(1), dim3(1), 0, s, step_counter, rng);
  zb_count_launch(2);
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
