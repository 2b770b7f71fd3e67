// out[M,N] = a[M,K] * w[N,K]^T for at most 8 tokens, 12 or 16 for smaller matrices: the decode step of a few sequences.
//
// The work is to read the weights once.  The tcgen05 kernel (gemm_bf16.cu) streams them well once it runs, but each launch pays for
// barriers, tensor memory, descriptors, a ring of tiles through shared memory and a cluster reduction, about 8 us that a matrix of 8 MB
// (1.3 us at the copy bandwidth) does not have.  Here a CTA takes 16 weight rows at a time with 8 warps along K, on mma.sync (m16n8k16,
// weights as A, tokens as the 8 columns of B, one or two such tiles):
//   * K is summed in an order of our own.  A lane's 16-byte piece of a weight row is four pairs of consecutive columns, which are its
//     A operands of two MMAs; the same 16 bytes of a token's row are its B operands.  No shuffles, no barriers.
//   * A warp owns 128 columns of every 1024 (256 bytes a row) and keeps kDepth such groups of 16 rows on their way, by cp.async into a
//     ring of which every thread reads what it asked for itself.  (Straight into registers they need room in the L1 cache while they
//     come, and a launch that starts under a kernel with the largest shared memory finds almost none: a decode step of the 8B model with
//     4 sequences took 3.6 ms, with the ring 1.73; on the tcgen05 kernel 2.26.)
//   * With static weights the ring is requested before the kernel in front has finished (programmatic dependent launch); only the tokens
//     wait for it.  A grid that one CTA per SM can do asks for more than half of an SM's shared memory: CTAs that start early, while
//     the kernel in front still holds most SMs, would otherwise crowd on the others.
// The warps' sums meet in shared memory, once per 16 rows.
// One token, us (tcgen05 kernel; weights at the copy bandwidth): 2048 x 2048 3.1 (7.3; 1.3), 3072 x 2048 3.4 (8.0; 1.9), 16384 x 2048 with
// SwiGLU 10.7 (17.1; 10.1), 2048 x 8192 8.2 (13.0; 5.0), 28672 x 4096 36.9 (43.0; 35.3); eight tokens 0.4 - 4 more.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "host_api.h"

namespace {
constexpr int kWarps = 8, kRowsTile = 16, kGroup = 4;                    // 32-column blocks of a warp's group
constexpr int kMaxTokens = 16;
// elements of a matrix for 9 to 12 and for 13 to 16 tokens
constexpr long long kMax12 = 64ll << 20, kMax16 = 40ll << 20;
constexpr int kSpan = kWarps * kGroup * 32;                              // columns that the CTA's groups cover
constexpr int kDepth = 3;
constexpr int kRing = kDepth * 2 * kGroup * 32 * kWarps * 16;            // 96 KB
constexpr int kOnePerSm = 120 * 1024;                                    // shared memory of which two CTAs do not fit an SM

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

ZB_DEVICE void copy16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16u : 0u) : "memory");
}
ZB_DEVICE void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// TT: tiles of 8 tokens
template <int TT>
struct __align__(16) StreamShared {
  float part[2][kWarps][8 * TT][kRowsTile + (TT == 1 ? 1 : 0)];      // rows of a token at `part_at`
  float scale[8 * TT];
};
// Two CTAs share an SM (1 KB of its shared memory each is the system's).
static_assert(2 * (kRing + sizeof(StreamShared<2>) + 1024) <= 228 * 1024, "two CTAs fit an SM");
// Place of a weight row's sum among a token's 16.  Against bank conflicts one tile of tokens has a column of padding; two tiles have no room
// for it, there every other pair of tokens is turned by 8.
template <int TT>
ZB_DEVICE int part_at(int token, int row) { return TT == 1 ? row : row ^ ((token & 2) << 2); }

template <int TT>
__global__ void __launch_bounds__(32 * kWarps, 2) zb_gemm_stream_kernel(const StreamParams p) {
  extern __shared__ __align__(16) uint4 ring[];      // [kDepth][2 kGroup][threads]
  __shared__ StreamShared<TT> sh;
  auto& part = sh.part;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
  zb_pdl_launch();
  const int groups = (p.k + kSpan - 1) / kSpan;
  const int mine = (p.tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int steps = mine * groups;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const int col0 = warp * (kGroup * 32) + tq * 8;
  // position of the next group to request
  int l_tile = blockIdx.x, l_group = 0, l_left = steps;
  auto request = [&](int slot) {
    if (l_left > 0) {
      --l_left;
      const int r0 = l_tile * kRowsTile + g, c = l_group * kSpan + col0;
      const __nv_bfloat16* at = p.w + static_cast<long long>(r0) * p.ldw + c;
      const uint32_t to = zb_smem_u32(ring + slot * (2 * kGroup * 32 * kWarps) + threadIdx.x);
#pragma unroll
      for (int u = 0; u < kGroup; ++u) {
        const bool in = c + 32 * u < p.k, lo = in && r0 < p.n, hi = in && r0 + 8 < p.n;
        copy16(to + (2 * u) * (32 * kWarps * 16), lo ? at + 32 * u : p.w, lo);
        copy16(to + (2 * u + 1) * (32 * kWarps * 16), hi ? at + 8 * p.ldw + 32 * u : p.w, hi);
      }
      if (++l_group == groups) {
        l_group = 0;
        l_tile += gridDim.x;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int x_group = 0;
  auto request_x = [&](uint4 (&x)[TT][kGroup]) {
    const int c = x_group * kSpan + col0;
#pragma unroll
    for (int t = 0; t < TT; ++t)
#pragma unroll
      for (int u = 0; u < kGroup; ++u)
        x[t][u] = g + 8 * t < p.m && c + 32 * u < p.k ? *reinterpret_cast<const uint4*>(p.a + static_cast<long long>(g + 8 * t) * p.lda + c + 32 * u) : zero;
    if (++x_group == groups) x_group = 0;
  };
  uint4 x[2][TT][kGroup];
  if (!p.static_w) zb_pdl_wait();
#pragma unroll
  for (int i = 0; i < kDepth; ++i) request(i);
  if (p.static_w) zb_pdl_wait();
  request_x(x[0]);
  if (steps > 1) request_x(x[1]);
  if (p.in_sumsq != nullptr) {                       // warp t: RMSNorm factor of tokens t, t + 8
#pragma unroll
    for (int t = warp; t < 8 * TT; t += kWarps) {
      float ss = 0.f;
      if (t < p.m)
        for (int i = lane; i < p.in_parts; i += 32) ss += p.in_sumsq[static_cast<size_t>(i) * p.in_ld + t];
      ss = zb_warp_sum(ss);
      if (lane == 0) sh.scale[t] = rsqrtf(ss * p.in_inv_d + p.in_eps);
    }
  }

  float acc[TT][2][4] = {};
  int tile = blockIdx.x, group = 0, buf = 0;
  const int tok = threadIdx.x >> 3, pair = threadIdx.x & 7;              // of the first 64 TT threads: outputs (tok, 2 pair .. 2 pair + 1)
  float ss_out = 0.f;
  int slot = 0;
  auto step = [&](uint4 (&xx)[TT][kGroup], int s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
    const uint4* mine_in = ring + slot * (2 * kGroup * 32 * kWarps) + threadIdx.x;
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      const uint4 l = mine_in[(2 * u) * (32 * kWarps)], h = mine_in[(2 * u + 1) * (32 * kWarps)];
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        mma16816(acc[t][0], l.x, h.x, l.y, h.y, xx[t][u].x, xx[t][u].y);
        mma16816(acc[t][1], l.z, h.z, l.w, h.w, xx[t][u].z, xx[t][u].w);
      }
    }
    request(slot);                                   // behind the reads of what it overwrites
    if (++slot == kDepth) slot = 0;
    if (s + 2 < steps) request_x(xx);
    if (++group < groups) return;
    group = 0;
#pragma unroll
    for (int t = 0; t < TT; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int token = 8 * t + 2 * tq + (i & 1);
        part[buf][warp][token][part_at<TT>(token, g + 8 * (i >> 1))] = acc[t][0][i] + acc[t][1][i];
        acc[t][0][i] = acc[t][1][i] = 0.f;
      }
    __syncthreads();                                 // the other buffer is read by nobody any more once all warps are here
    if (threadIdx.x < 64 * TT && tok < p.m) {
      const int row = tile * kRowsTile + 2 * pair;
      float v[2] = {0.f, 0.f};
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        v[0] += part[buf][w][tok][part_at<TT>(tok, 2 * pair)];
        v[1] += part[buf][w][tok][part_at<TT>(tok, 2 * pair + 1)];
      }
      const bool in[2] = {row < p.n, row + 1 < p.n};
      if (p.in_sumsq != nullptr) {
        v[0] *= sh.scale[tok];
        v[1] *= sh.scale[tok];
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
    step(x[0], s);
    if (s + 1 < steps) step(x[1], s + 1);
  }
  if (p.out_sumsq != nullptr && threadIdx.x < 64 * TT) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) ss_out += __shfl_xor_sync(0xffffffffu, ss_out, o);
    if (pair == 0 && tok < p.m) p.out_sumsq[static_cast<size_t>(blockIdx.x) * p.out_ld + tok] = ss_out;
  }
}
}  // namespace

// 1 when the kernel takes the problem.  9 to 16 tokens double the tokens' reads (as many bytes as the weights) and the MMAs, which a large
// matrix does not hide, nor a long row of which few CTAs have a share.  12 / 16 tokens, us (tcgen05 kernel): 2048 x 2048 3.7 / 3.7 (7.2),
// 5120 x 2048 6.3 / 6.6 (10.2), 2048 x 8192 9.9 / 10.4 (13.4), 4096 x 4096 8.7 / 9.2 (12.9), 6144 x 4096 13.8 / 15.4 (18.1), 16384 x 2048
// 14.9 / 16.3 (19.2); with statistics 4096 x 14336 30.1 / 33.3 (30.1), 12288 x 4096 27.9 / 30.7 (29.0), 28672 x 4096 54.8 / 58.5 (53.4);
// 512 x 16384 13.2 / 14.9 (14.1).
int zb_gemm_stream_wants(const void* a, const void* w, int m, int n, int k) {
  const long long size = static_cast<long long>(n) * k;
  const bool few = m <= 8 || (m <= 12 && size <= kMax12) || (m <= kMaxTokens && size <= kMax16 && (k <= 8192 || n >= 1024));
  return few && n >= 16 && k >= 64 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
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
  const auto launch = [&](auto kernel, bool (&configured)[16]) {
    if (const int rc = zb_config_smem_once(kernel, kOnePerSm, configured)) return rc;
    return static_cast<int>(zb_launch(kernel, dim3(grid), dim3(32 * kWarps), grid > num_sms ? kRing : kOnePerSm, stream, p));
  };
  static bool one[16] = {}, two[16] = {};
  if (const int rc = m <= 8 ? launch(zb_gemm_stream_kernel<1>, one) : launch(zb_gemm_stream_kernel<2>, two)) return rc;
  zb_count_launch(1);
  return static_cast<int>(cudaGetLastError());
}
