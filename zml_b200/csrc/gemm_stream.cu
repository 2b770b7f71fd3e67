// out[M,N] = a[M,K] * w[N,K]^T for at most 8 tokens: the decode step of a few sequences.
//
// The work is to read the weights once.  The tcgen05 kernel (gemm_bf16.cu) streams them well once it runs, but each launch pays for
// barriers, tensor memory, descriptors, a ring of tiles through shared memory and a cluster reduction, about 8 us that a matrix of 8 MB
// (1.3 us at the copy bandwidth) does not have.  Here a CTA takes 16 weight rows at a time with 8 warps along K; weights go from
// global memory straight into the registers of mma.sync (m16n8k16, weights as A, the tokens as the 8 columns of B):
//   * K is summed in an order of our own.  A lane's 16-byte piece of a weight row is four pairs of consecutive columns, which are its
//     A operands of two MMAs; the same 16 bytes of a token's row are its B operands.  No shuffles, no shared memory.
//   * A warp owns 128 columns of every 1024 (256 bytes a row) and keeps two such groups of 16 rows on their way: 16 KB a warp.
//   * With static weights both groups are requested before the kernel in front has finished (programmatic dependent launch); only the
//     tokens wait for it.
// The warps' sums meet in shared memory, once per 16 rows.
// One token, us (tcgen05 kernel; weights at the copy bandwidth): 2048 x 2048 2.9 (7.3; 1.3), 3072 x 2048 3.2 (8.0; 1.9), 16384 x 2048 with
// SwiGLU 10.7 (17.1; 10.1), 2048 x 8192 9.1 (13.0; 5.0), 28672 x 4096 35.6 (43.0; 35.3); eight tokens 0.3 - 3 more.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "host_api.h"

namespace {
constexpr int kWarps = 8, kRowsTile = 16, kTokens = 8, kGroup = 4;       // 32-column blocks of a warp's group
constexpr int kSpan = kWarps * kGroup * 32;                              // columns that the CTA's groups cover

struct StreamParams {
  const __nv_bfloat16* w;
  const __nv_bfloat16* a;
  void* out;
  const __nv_bfloat16* residual;   // rows of ldo
  const __nv_bfloat16* bias;
  long long ldw, lda, ldo;
  int m, n, k, tiles, out_f32, static_w, act;
  const float* in_sumsq;           // see ZbGemmEpi
  float* out_sumsq;                // [gridDim.x][out_ld]
  int in_parts, in_ld, out_ld;
  float in_inv_d, in_eps;
};

ZB_DEVICE uint4 ld_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
ZB_DEVICE void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(32 * kWarps, 2) zb_gemm_stream_kernel(const StreamParams p) {
  __shared__ float part[2][kWarps][kTokens][kRowsTile + 1];
  __shared__ float scale[kTokens];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  zb_pdl_launch();
  const int groups = (p.k + kSpan - 1) / kSpan;
  const int mine = (p.tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int steps = mine * groups;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const int col0 = warp * (kGroup * 32) + tq * 8;
  // position of the next group to request
  int l_tile = blockIdx.x, l_group = 0;
  auto request = [&](uint4 (&lo)[kGroup], uint4 (&hi)[kGroup]) {
    const int r0 = l_tile * kRowsTile + g, c = l_group * kSpan + col0;
    const __nv_bfloat16* at = p.w + static_cast<long long>(r0) * p.ldw + c;
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      const bool in = c + 32 * u < p.k;
      lo[u] = in && r0 < p.n ? ld_stream(at + 32 * u) : zero;
      hi[u] = in && r0 + 8 < p.n ? ld_stream(at + 8 * p.ldw + 32 * u) : zero;
    }
    if (++l_group == groups) {
      l_group = 0;
      l_tile += gridDim.x;
    }
  };
  int x_group = 0;
  auto request_x = [&](uint4 (&x)[kGroup]) {
    const int c = x_group * kSpan + col0;
#pragma unroll
    for (int u = 0; u < kGroup; ++u)
      x[u] = g < p.m && c + 32 * u < p.k ? *reinterpret_cast<const uint4*>(p.a + static_cast<long long>(g) * p.lda + c + 32 * u) : zero;
    if (++x_group == groups) x_group = 0;
  };
  uint4 lo[2][kGroup], hi[2][kGroup], x[2][kGroup];
  if (p.static_w) {
    request(lo[0], hi[0]);
    if (steps > 1) request(lo[1], hi[1]);
    zb_pdl_wait();
  } else {
    zb_pdl_wait();
    request(lo[0], hi[0]);
    if (steps > 1) request(lo[1], hi[1]);
  }
  request_x(x[0]);
  if (steps > 1) request_x(x[1]);
  if (p.in_sumsq != nullptr) {                       // warp t: RMSNorm factor of token t
    float ss = 0.f;
    if (warp < p.m)
      for (int i = lane; i < p.in_parts; i += 32) ss += p.in_sumsq[static_cast<size_t>(i) * p.in_ld + warp];
    ss = zb_warp_sum(ss);
    if (lane == 0) scale[warp] = rsqrtf(ss * p.in_inv_d + p.in_eps);
  }

  float acc[2][4] = {};
  int tile = blockIdx.x, group = 0, buf = 0;
  const int tok = threadIdx.x >> 3, pair = threadIdx.x & 7;              // of the first 64 threads: outputs (tok, 2 pair .. 2 pair + 1)
  float ss_out = 0.f;
  auto step = [&](uint4 (&l)[kGroup], uint4 (&h)[kGroup], uint4 (&xx)[kGroup], int s) {
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      mma16816(acc[0], l[u].x, h[u].x, l[u].y, h[u].y, xx[u].x, xx[u].y);
      mma16816(acc[1], l[u].z, h[u].z, l[u].w, h[u].w, xx[u].z, xx[u].w);
    }
    if (s + 2 < steps) {
      request(l, h);
      request_x(xx);
    }
    if (++group < groups) return;
    group = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      part[buf][warp][2 * tq + (i & 1)][g + 8 * (i >> 1)] = acc[0][i] + acc[1][i];
      acc[0][i] = acc[1][i] = 0.f;
    }
    __syncthreads();                                 // the other buffer is read by nobody any more once all warps are here
    if (threadIdx.x < 64 && tok < p.m) {
      const int row = tile * kRowsTile + 2 * pair;
      float v[2] = {0.f, 0.f};
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        v[0] += part[buf][w][tok][2 * pair];
        v[1] += part[buf][w][tok][2 * pair + 1];
      }
      const bool in[2] = {row < p.n, row + 1 < p.n};
      if (p.in_sumsq != nullptr) {
        v[0] *= scale[tok];
        v[1] *= scale[tok];
      }
      if (p.act == ZB_ACT_SWIGLU) {
        if (in[1]) reinterpret_cast<__nv_bfloat16*>(p.out)[static_cast<size_t>(tok) * p.ldo + row / 2] = __float2bfloat16(zb_gate_act(v[0], ZB_ACT_SWIGLU) * v[1]);
      } else {
        const size_t at = static_cast<size_t>(tok) * p.ldo + row;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (!in[i]) continue;
          if (p.bias != nullptr) v[i] += __bfloat162float(p.bias[row + i]);
          if (p.residual != nullptr) v[i] += __bfloat162float(p.residual[at + i]);
          v[i] = zb_plain_act(v[i], p.act);
          if (p.out_f32) {
            reinterpret_cast<float*>(p.out)[at + i] = v[i];
          } else {
            const __nv_bfloat16 b = __float2bfloat16(v[i]);
            reinterpret_cast<__nv_bfloat16*>(p.out)[at + i] = b;
            ss_out += __bfloat162float(b) * __bfloat162float(b);
          }
        }
      }
    }
    buf ^= 1;
    tile += gridDim.x;
  };
  for (int s = 0; s < steps; s += 2) {
    step(lo[0], hi[0], x[0], s);
    if (s + 1 < steps) step(lo[1], hi[1], x[1], s + 1);
  }
  if (p.out_sumsq != nullptr && threadIdx.x < 64) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) ss_out += __shfl_xor_sync(0xffffffffu, ss_out, o);
    if (pair == 0 && tok < p.m) p.out_sumsq[static_cast<size_t>(blockIdx.x) * p.out_ld + tok] = ss_out;
  }
}
}  // namespace

// 1 when the kernel takes the problem.
int zb_gemm_stream_wants(const void* a, const void* w, int m, int n, int k) {
  return m <= kTokens && n >= 16 && k >= 64 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

// The contract of the tcgen05 kernel's launch; epi->pf_* is ignored.  `out_parts`: parts written to epi->out_sumsq.
int zb_gemm_stream_launch(const void* a, const void* w, void* out, const void* residual, const void* bias, int m, int n, int k, int lda, int ldw,
                          int ldo, int out_f32, int static_w, const ZbGemmEpi* epi, int* out_parts, int num_sms, cudaStream_t stream) {
  StreamParams p = {};
  p.w = reinterpret_cast<const __nv_bfloat16*>(w);
  p.a = reinterpret_cast<const __nv_bfloat16*>(a);
  p.out = out;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.ldw = ldw;
  p.lda = lda;
  p.ldo = ldo;
  p.m = m;
  p.n = n;
  p.k = k;
  p.tiles = (n + kRowsTile - 1) / kRowsTile;
  p.out_f32 = out_f32;
  p.static_w = static_w;
  if (epi != nullptr) {
    p.act = epi->swiglu;
    p.in_sumsq = epi->in_sumsq;
    p.in_parts = epi->in_parts;
    p.in_ld = epi->in_ld;
    p.in_inv_d = epi->in_inv_d;
    p.in_eps = epi->in_eps;
    p.out_sumsq = epi->out_sumsq;
    p.out_ld = epi->out_ld;
  }
  // row statistics: one part per CTA, of which a consumer takes 160 at most
  const int grid = std::min(p.tiles, p.out_sumsq != nullptr ? num_sms : 2 * num_sms);
  if (out_parts != nullptr && p.out_sumsq != nullptr) *out_parts = grid;
  const cudaError_t e = zb_launch(zb_gemm_stream_kernel, dim3(grid), dim3(32 * kWarps), 0, stream, p);
  zb_count_launch(1);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}
