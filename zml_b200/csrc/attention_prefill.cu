// Paged prefill attention without extensions on the 5th-generation tensor cores (tcgen05 / TMEM / TMA): head_dim 64, 128 and
// 256, 64-token KV pages, grouped-query attention (with an even group size up to 128).
//
// One CTA works on 128 query rows of TWO query heads that share a KV head - of one head where head_dim is 256 - and every page that it
// brings in feeds both heads' softmax pipelines:
//   warps 0-3 / 4-7 : softmax and epilogue of head A / B, one thread per query row
//   next warp       : TMA producer (Q once, then K and V pages through a ring)
//   last warps      : one thread each issues the MMAs of head A / B, so that neither head waits for the other's events
// Per page and head: S = Q K^T (fp32 in tensor memory), P = 2^(S - m) as bf16 over S, O += P V (A = P from tensor memory, B = V in
// its natural [key][head_dim] layout, MN-major).
//
// What bounds it: per page and head, 128 x 64 exponentials (16 per clock and SM: 512 clocks, both heads share them), 2 x 128 x 64 x
// head_dim multiply-adds (4096 per clock: 256 or 512) and what the softmax warps do besides (maximum, conversion, sum) - and, before all
// of these, the chain S -> softmax -> P -> O of one head, whose hand-overs two heads alone do not hide.  Hence
//   * S has two buffers of one page each and P lies over the S it came from, so the next S is there when a page's exponentials are done
//     (one buffer of 128 keys, as large in tensor memory: 1727 us; two threads per row, 1928 us; these buffers, 1380 us);
//   * the reference m of a row moves only when the maximum has grown by more than 2^kLazy (P stays below 2^kLazy, which bf16 and fp32
//     hold as well as numbers below one), so O is hardly ever rescaled;
//   * a few exponentials run as polynomials on the FMA pipes (Shape::kPoly).
// 8192 queries on 16384 keys, 32 heads on 8: head_dim 128 1.35 ms (1220 TFLOP/s; the kernel before it: 2.33), head_dim 64 1.19 ms (694;
// the mma.sync kernel: 5.17).  4 x 2048: 0.18 (0.29) and 0.15 (0.48) ms.
// Tensor memory columns: S_A 0 and 64 | S_B 128 and 192 (P in the first half of each) | O_A 256 | O_B 384, or one O from 256 on.
// head_dim 256: 1024 clocks of multiply-adds a page cover the softmax of one head; its O leaves no room for another's.  16 heads on 4:
// 8192 tokens 0.80 ms (689 TFLOP/s; the mma.sync kernel: 4.64), seven prompts of 128 to 2048 tokens 0.19 (0.88) ms.
// Every wait is bounded; a wait that runs out records a status and the CTA leaves through its normal exit.
#include <cuda.h>

#include "common.cuh"
#include "host_api.h"

int zb_make_tmap_bf16_2d(CUtensorMap* out, const void* base, int rows, int k, int ld, int box_rows);
int zb_make_tmap_kv_cache(CUtensorMap* out, const void* base, long long slots, int kv_heads, int head_dim, int box_rows);

namespace {

constexpr int kRows = 128;                           // query rows of a CTA
constexpr int kKeys = 64;                            // keys of a tile: a page
constexpr uint32_t kKernelId = 13;
constexpr uint32_t kTmemCols = 512;
constexpr float kLazy = 8.f;
// 2^f on [-1/2, 1/2], interpolated at Chebyshev nodes (relative error 2.2e-7 in fp32, that of ex2.approx)
__device__ constexpr float kExp2[6] = {1.00000012f, 0.693147182f, 0.240221068f, 0.0555035695f, 0.00967603177f, 0.00133908633f};

ZB_DEVICE float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
// 2^x of two numbers on the FMA pipes; below -126.5 zero (as ex2.approx.ftz below -126), so that a masked key has no weight; a NaN stays one.
ZB_DEVICE void exp2_fma(float& x0, float& x1) {
  const float kMagic = 12582912.f;                   // 1.5 * 2^23: the sum's low bits are x rounded to an integer
  const ZbF2 x = zb_pack2(max_nan(x0, -127.f), max_nan(x1, -127.f)), t = zb_add2(x, zb_pack2(kMagic, kMagic));
  const ZbF2 f = zb_fma2(zb_add2(t, zb_pack2(-kMagic, -kMagic)), zb_pack2(-1.f, -1.f), x);
  ZbF2 q = zb_pack2(kExp2[5], kExp2[5]);
#pragma unroll
  for (int k = 4; k >= 0; --k) q = zb_fma2(q, f, zb_pack2(kExp2[k], kExp2[k]));
  float t0, t1;
  zb_unpack2(t, t0, t1);
  const ZbF2 e = zb_pack2(__uint_as_float((__float_as_uint(t0) << 23) + 0x3f800000u), __uint_as_float((__float_as_uint(t1) << 23) + 0x3f800000u));
  zb_unpack2(zb_mul2(q, e), x0, x1);
}

struct PrefillParams {
  __nv_bfloat16* out;           // [tokens, num_q_heads, HD]
  const int32_t* block_table;   // [batch, max_pages]
  const int32_t* seq_lens;      // [batch]
  const int32_t* q_start;       // [batch + 1]
  int batch;
  int num_q_heads;
  int num_kv_heads;
  int max_pages;
  int window;
  float scale_log2;
  ZbStatus* status;
};

template <int HD>
struct Shape {
  static constexpr int kStages = HD == 64 ? 8 : (HD == 128 ? 5 : 2);
  static constexpr int kHeads = HD == 256 ? 1 : 2;                 // of a CTA
  static constexpr int kThreads = 32 * (5 * kHeads + 1);
  static constexpr int kSubs = HD / 64;                            // 64-column sub-tiles
  static constexpr int kQBytes = kRows * HD * 2, kKvBytes = kKeys * HD * 2;
  // Of 16 pairs of exponentials, those that the FMA pipes take.  8192 queries on 16384 keys, 32 heads: head_dim 64 0 / 4 / 6 / 8 pairs
  // 1246 / 1189 / 1270 / 1357 us, head_dim 128 0 / 1 / 4 1380 / 1352 / 1395 us.  More of them fill the ALU pipe (cuts, exponents).
  static constexpr int kPoly = HD == 64 ? 4 : 1;
  static constexpr int kSmem = kHeads * kQBytes + 2 * kStages * kKvBytes + 1024 + 512;
};
constexpr uint32_t kColS = 0, kColO = 256;           // S: [head][buffer][64], O: [head][128] or [256]

// max of three, one instruction
ZB_DEVICE float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int HD>
__global__ void __launch_bounds__(Shape<HD>::kThreads, 1)
zb_prefill_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                  const __grid_constant__ CUtensorMap tmap_v, const PrefillParams p) {
  using S = Shape<HD>;
  constexpr int kStages = S::kStages, kHeads = S::kHeads;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* q_s = smem;                               // [kHeads][kQBytes]
  uint8_t* k_s = q_s + kHeads * S::kQBytes;               // [kStages][kKvBytes]
  uint8_t* v_s = k_s + kStages * S::kKvBytes;        // [kStages][kKvBytes]
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + kStages * S::kKvBytes);
  uint64_t* q_full = bars;                           // 1
  uint64_t* k_full = bars + 1;                       // kStages
  uint64_t* v_full = k_full + kStages;               // kStages
  uint64_t* kv_empty = v_full + kStages;             // kStages, both heads' MMAs
  uint64_t* s_full = kv_empty + kStages;             // [2 heads][2 buffers]
  uint64_t* p_full = s_full + 4;                     // [2 heads][2 buffers], four warps
  uint64_t* o_ready = p_full + 4;                    // 2
  uint64_t* v_raw = o_ready + 2;                     // 1: V of a page that is cleared behind the sequence's end
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(v_raw + 1);
  volatile uint32_t* abort_flag = tmem_holder + 1;
  volatile uint32_t* abort_where = tmem_holder + 2;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = p.num_q_heads / p.num_kv_heads;
  const int head0 = blockIdx.x * kHeads;
  const int kvh = head0 / group;

  if (warp == 4 * kHeads && lane == 0) {
    zb_mbar_init(q_full, 1);
    for (int s = 0; s < kStages; ++s) {
      zb_mbar_init(&k_full[s], 1);
      zb_mbar_init(&v_full[s], 1);
      zb_mbar_init(&kv_empty[s], kHeads);
    }
    for (int i = 0; i < 4; ++i) {
      zb_mbar_init(&s_full[i], 1);
      zb_mbar_init(&p_full[i], 4);
    }
    zb_mbar_init(&o_ready[0], 1);
    zb_mbar_init(&o_ready[1], 1);
    zb_mbar_init(v_raw, 1);
    *abort_flag = 0u;
    *abort_where = 0u;
    zb_mbar_fence_init();
    zb_fence_proxy_async_smem();                     // the first copies go out in front of the block's barrier
    zb_tma_prefetch_desc(&tmap_q);
    zb_tma_prefetch_desc(&tmap_k);
    zb_tma_prefetch_desc(&tmap_v);
  }
  zb_pdl_wait();                                     // q, the KV cache and the batch description come from preceding work

  // The (sequence, 128-row query block) of this CTA.  Head pairs are the grid's fast index, and blocks are handed out from the end of
  // the batch backwards, within a sequence from its last (longest) block: the short ones fill the last wave.  Every warp looks at 32
  // sequences at a time, a lane each: one after the other, 40 sequences cost every CTA 3.4 us.
  int seq = -1, qb = 0;
  {
    int rem = static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y);
    for (int i0 = 0; i0 < p.batch; i0 += 32) {
      const int i = i0 + lane, nb = i < p.batch ? max(0, p.q_start[i + 1] - p.q_start[i] + kRows - 1) / kRows : 0;
      int upto = nb;                                 // blocks of the sequences up to this one
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, rem < upto);
      if (hit != 0u) {
        const int l = __ffs(hit) - 1;
        seq = i0 + l;                                // what the loops go by is found alike in all lanes (a value out of a shuffle cost them 0.7 %)
        qb = rem - __reduce_add_sync(0xffffffffu, lane < l ? nb : 0);
        break;
      }
      rem -= __reduce_add_sync(0xffffffffu, nb);
    }
  }
  if (seq < 0) return;                               // grid is an upper bound of the number of blocks
  const int q_first = p.q_start[seq], q_len = p.q_start[seq + 1] - q_first, len = p.seq_lens[seq];
  const int ctx = len - q_len;
  const int row_base = qb * kRows;
  const int tok_base = q_first + row_base;
  const int rows_valid = min(kRows, q_len - row_base);
  const int last_key = min(len, ctx + row_base + kRows);                                    // exclusive
  const int first_tile = p.window > 0 ? max(0, ctx + row_base - p.window + 1) / kKeys : 0;
  const int n_tiles = (last_key + kKeys - 1) / kKeys - first_tile;
  // Rows of the last page behind the sequence's end.  They hold whatever was there before, perhaps NaN, and a masked key's weight of zero
  // does not make that zero: these rows of V are cleared in shared memory (those of K only reach scores that the mask replaces).  The page
  // comes with a barrier of its own, and the producer warp arrives on the ring's behind its stores: the MMA threads know nothing of it (a
  // condition in their loop cost 0.4 %).
  const int behind = (first_tile + n_tiles) * kKeys - len;

  const int32_t* bt = p.block_table + static_cast<size_t>(seq) * p.max_pages;
  auto page_of = [&](int j) {
    const int page = bt[first_tile + j];
    return ZB_BC_OK(page, ZB_BC_PAGES, kKernelId, 10) ? page : 0;
  };
  auto load_page = [&](int page, uint32_t stage, bool last) {
    uint64_t* v_bar = last && behind > 0 ? v_raw : &v_full[stage];
    zb_mbar_expect_tx(&k_full[stage], S::kKvBytes);
    zb_tma_load_4d(k_s + stage * S::kKvBytes, &tmap_k, &k_full[stage], 0, page * kKeys, 0, kvh);
    zb_mbar_expect_tx(v_bar, S::kKvBytes);
    zb_tma_load_4d(v_s + stage * S::kKvBytes, &tmap_v, v_bar, 0, page * kKeys, 0, kvh);
  };
  if (warp == 4 * kHeads && lane == 0) {             // on their way while tensor memory is allocated
    zb_mbar_expect_tx(q_full, kHeads * S::kQBytes);
    for (int w = 0; w < kHeads; ++w)
      for (int c = 0; c < S::kSubs; ++c)
        zb_tma_load_2d(q_s + w * S::kQBytes + c * (kRows * 128), &tmap_q, q_full, (head0 + w) * HD + c * 64, tok_base);
    if (n_tiles > 0) load_page(page_of(0), 0, n_tiles == 1);
  }
  if (warp == 4 * kHeads + 1) {
    zb_tmem_alloc(tmem_holder, kTmemCols);
    zb_tmem_relinquish();
  }
  zb_tc_fence_before();
  __syncthreads();
  zb_tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  zb_pdl_launch();                                   // only now: a successor that also takes tensor memory must not come first

  if (warp == 4 * kHeads) {
    // ------------------------------------------------------------------ TMA producer
    bool ok = true;
    if (lane == 0) {
      uint32_t stage = 1, phase = 0;
      int next = n_tiles > 1 ? page_of(1) : 0;       // asked for a tile ahead: with two stages the wait below is what the loads hang on
      for (int j = 1; j < n_tiles; ++j) {
        const int page = next;
        if (j + 1 < n_tiles) next = page_of(j + 1);
        if (j >= kStages && !zb_mbar_wait(&kv_empty[stage], phase ^ 1u, abort_flag)) {
          *abort_where = 1u;
          ok = false;
          break;
        }
        load_page(page, stage, j == n_tiles - 1);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (n_tiles > 0 && behind > 0 && __all_sync(0xffffffffu, ok)) {
      const int at = (n_tiles - 1) % kStages;
      ok = zb_mbar_wait(v_raw, 0u, abort_flag);
      if (__all_sync(0xffffffffu, ok)) {
        uint4* v = reinterpret_cast<uint4*>(v_s + at * S::kKvBytes) + (kKeys - behind) * 8;      // the swizzle stays within a row of 128 bytes
        for (int c = 0; c < S::kSubs; ++c)
          for (int i = lane; i < behind * 8; i += 32) v[c * kKeys * 8 + i] = make_uint4(0u, 0u, 0u, 0u);
        zb_fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) zb_mbar_arrive(&v_full[at]);
      } else {
        *abort_where = 7u;
      }
    }
  } else if (warp > 4 * kHeads) {
    // ------------------------------------------------------------------ MMA issuer of head w
    if (lane == 0) {
      const int w = warp - 4 * kHeads - 1;
      constexpr uint32_t kIdescS = zb_make_idesc_bf16(kRows, kKeys);
      constexpr uint32_t kIdescO = zb_make_idesc_bf16(kRows, HD) | (1u << 16);         // B (= V) is MN-major
      const uint32_t t_s = tmem_base + kColS + w * 128, t_o = tmem_base + kColO + w * 128;
      const uint32_t qa = zb_smem_u32(q_s + w * S::kQBytes);
      uint32_t k_stage = 0, k_phase = 0, stage = 0, phase = 0, where = 0;
      // S of the next tile into buffer `b`
      auto next_s = [&](int b) {
        if (!zb_mbar_wait(&k_full[k_stage], k_phase, abort_flag)) return false;
        zb_tc_fence_after();
        const uint32_t ka = zb_smem_u32(k_s + k_stage * S::kKvBytes);
#pragma unroll
        for (int c = 0; c < S::kSubs; ++c) {
          const uint64_t dq = zb_make_desc_sw128(qa + c * (kRows * 128)), dk = zb_make_desc_sw128(ka + c * (kKeys * 128));
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) zb_umma_f16(t_s + b * kKeys, dq + 2 * kk, dk + 2 * kk, kIdescS, (c > 0 || kk > 0) ? 1u : 0u);
        }
        zb_umma_commit(&s_full[2 * w + b]);
        if (++k_stage == kStages) {
          k_stage = 0;
          k_phase ^= 1u;
        }
        return true;
      };
      if (!zb_mbar_wait(q_full, 0u, abort_flag)) {
        where = 2u;
      } else if ((n_tiles > 0 && !next_s(0)) || (n_tiles > 1 && !next_s(1))) {
        where = 3u;
      }
      for (int j = 0; where == 0u && j < n_tiles; ++j) {
        if (!zb_mbar_wait(&v_full[stage], phase, abort_flag)) {
          where = 4u;
          break;
        }
        // (a barrier per buffer: the softmax may publish the next tile's P before this one's V has come)
        if (!zb_mbar_wait(&p_full[2 * w + (j & 1)], static_cast<uint32_t>(j >> 1) & 1u, abort_flag)) {
          where = 5u;
          break;
        }
        zb_tc_fence_after();
        // O (+)= P V: steps of 16 keys; A = P in tensor memory (8 columns per step), B = V, MN-major
        const uint32_t va = zb_smem_u32(v_s + stage * S::kKvBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          zb_umma_f16_ts(t_o, t_s + (j & 1) * kKeys + 8 * k, zb_make_desc_sw128_mn(va + k * (16 * 128), kKeys * 128, 1024), kIdescO,
                         (j > 0 || k > 0) ? 1u : 0u);
        zb_umma_commit(&o_ready[w]);
        zb_umma_commit(&kv_empty[stage]);
        if (j + 2 < n_tiles && !next_s(j & 1)) {      // over P, in order behind the MMAs that read it
          where = 6u;
          break;
        }
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (where != 0u) *abort_where = where;
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue (one row per thread)
    const int w = warp >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;                  // query row inside the block
    const int qpos = ctx + row_base + r;             // its position among the keys
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_o = tmem_base + kColO + w * 128 + lane_off;
    const int lo = p.window > 0 ? max(0, qpos - p.window + 1) : 0, hi = min(qpos + 1, len);    // visible: lo <= key < hi
    const int lo_last = p.window > 0 ? max(0, ctx + row_base + kRows - p.window) : 0;           // of the block's last row
    const ZbF2 sc2 = zb_pack2(p.scale_log2, p.scale_log2);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int b = j & 1;
      const uint32_t t_s = tmem_base + kColS + w * 128 + b * kKeys + lane_off;
      if (!__all_sync(0xffffffffu, zb_mbar_wait(&s_full[2 * w + b], static_cast<uint32_t>(j >> 1) & 1u, abort_flag))) {
        *abort_where = 10u + w;
        ok = false;
        break;
      }
      zb_tc_fence_after();
      uint32_t sr[64];
      zb_tmem_ld32(t_s, reinterpret_cast<uint32_t(&)[32]>(sr[0]));
      zb_tmem_ld32(t_s + 32, reinterpret_cast<uint32_t(&)[32]>(sr[32]));
      zb_tmem_ld_wait();
      // pages below the block's first row and inside every row's window need no mask
      const int key0 = (first_tile + j) * kKeys;
      if (!(key0 + kKeys - 1 <= ctx + row_base && key0 + kKeys <= len && key0 >= lo_last)) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (key0 + i >= hi || key0 + i < lo) sr[i] = 0xff800000u;                             // -inf
      }
      float mx4[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) mx4[i] = __uint_as_float(sr[i]);
#pragma unroll
      for (int i = 4; i < 60; i += 2) mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(sr[i]), __uint_as_float(sr[i + 1]));
      mx4[0] = max3(mx4[0], __uint_as_float(sr[60]), __uint_as_float(sr[61]));
      mx4[1] = max3(mx4[1], __uint_as_float(sr[62]), __uint_as_float(sr[63]));
      const float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * p.scale_log2;              // in units of log2
      float alpha = 1.f;
      if (mx > m + kLazy) {                          // also the first visible key: m = -inf
        alpha = m == -INFINITY ? 1.f : zb_ex2(m - mx);
        m = mx;
        l *= alpha;
      }
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        // O += P V of the previous tile must be complete (that of the one before it is: S of this tile went behind it)
        if (!__all_sync(0xffffffffu, zb_mbar_wait(&o_ready[w], static_cast<uint32_t>(j - 1) & 1u, abort_flag))) {
          *abort_where = 12u + w;
          ok = false;
          break;
        }
        zb_tc_fence_after();
#pragma unroll 1
        for (int c0 = 0; c0 < HD; c0 += 16) {
          uint32_t o[16];
          zb_tmem_ld16(t_o + c0, o);
          zb_tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          zb_tmem_st16(t_o + c0, o);
        }
      }
      // p = 2^(s * scale - m)
      const float neg_m = m == -INFINITY ? 0.f : -m;
      const ZbF2 nm2 = zb_pack2(neg_m, neg_m);
      ZbF2 sum[2] = {0ull, 0ull};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pw[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int e = 32 * c + 2 * i;
          float x0, x1;
          zb_unpack2(zb_fma2(zb_pack2(__uint_as_float(sr[e]), __uint_as_float(sr[e + 1])), sc2, nm2), x0, x1);
          if (((i * S::kPoly) & 15) < S::kPoly) {
            exp2_fma(x0, x1);
          } else {
            x0 = zb_ex2(x0);
            x1 = zb_ex2(x1);
          }
          pw[i] = zb_pack_bf16x2(x0, x1);
          sum[i & 1] = zb_add2(sum[i & 1], zb_pack2(x0, x1));
        }
        zb_tmem_st16(t_s + 16 * c, pw);
      }
      l += zb_sum2(zb_add2(sum[0], sum[1]));
      // Parity does not tell a phase of o_ready from the one two before it, so that no wait may begin two phases early or end two late: the
      // last tile but one is waited for while the last one is still held back.
      if (j > 0 && j == n_tiles - 1) ok = zb_mbar_wait(&o_ready[w], static_cast<uint32_t>(j - 1) & 1u, abort_flag);
      zb_tmem_st_wait();
      zb_tc_fence_before();
      __syncwarp();
      if (lane == 0) zb_mbar_arrive(&p_full[2 * w + b]);
    }
    if (ok && n_tiles > 0) ok = zb_mbar_wait(&o_ready[w], static_cast<uint32_t>(n_tiles - 1) & 1u, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) {
      *abort_where = 14u + w;
    } else {
      zb_tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;     // no key at all (cannot happen for a causal prefill): zeros
      __nv_bfloat16* orow = p.out + (static_cast<size_t>(tok_base + r) * p.num_q_heads + head0 + w) * HD;
#pragma unroll 1
      for (int c0 = 0; c0 < HD; c0 += 32) {
        uint32_t o[32];
        zb_tmem_ld32(t_o + c0, o);
        zb_tmem_ld_wait();
        if (r < rows_valid) {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = n_tiles > 0 ? __float_as_uint(__uint_as_float(o[i]) * inv) : 0u;
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            *reinterpret_cast<uint4*>(orow + c0 + i) =
                make_uint4(zb_pack_bf16x2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), zb_pack_bf16x2(__uint_as_float(o[i + 2]), __uint_as_float(o[i + 3])),
                           zb_pack_bf16x2(__uint_as_float(o[i + 4]), __uint_as_float(o[i + 5])), zb_pack_bf16x2(__uint_as_float(o[i + 6]), __uint_as_float(o[i + 7])));
        }
      }
    }
  }

  // ------------------------------------------------------------------ common exit
  zb_tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (threadIdx.x == 0) zb_record_error(p.status, ZB_ERR_MBAR_TIMEOUT, kKernelId, *abort_where, blockIdx.y);
    const uint64_t t0 = zb_globaltimer();            // copies still in flight must land before the shared memory is reused
    while (zb_globaltimer() - t0 < 200000ull) {
    }
    __syncthreads();
  }
  if (warp == 4 * kHeads + 1) {
    zb_tc_fence_after();
    zb_tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int HD>
int launch_prefill(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const PrefillParams& p, int q_blocks, cudaStream_t s) {
  static bool configured[16] = {};
  if (const int rc = zb_config_smem_once(zb_prefill_kernel<HD>, Shape<HD>::kSmem, configured)) return rc;
  const cudaError_t le = zb_launch(zb_prefill_kernel<HD>, dim3(p.num_q_heads / Shape<HD>::kHeads, q_blocks), dim3(Shape<HD>::kThreads), Shape<HD>::kSmem, s, tq, tk, tv, p);
  zb_count_launch(1);
  return static_cast<int>(le != cudaSuccess ? le : cudaGetLastError());
}

}  // namespace

// The plain case of zb_paged_prefill_tc (attention_tc.cu), which checks the arguments.
int zb_prefill_plain(const void* q, const void* k_cache, const void* v_cache, void* out, const int32_t* block_table, const int32_t* seq_lens,
                     const int32_t* q_start, int batch, int q_blocks, int total_tokens, int num_q_heads, int num_kv_heads, int head_dim,
                     int max_pages, long long q_stride, float scale, int window, ZbStatus* status, void* stream) {
  CUtensorMap tq, tk, tv;
  int rc = zb_make_tmap_bf16_2d(&tq, q, total_tokens, num_q_heads * head_dim, static_cast<int>(q_stride), kRows);
  const long long slots = 1ll << 30;               // bound only: pages are addressed through the block table
  if (rc == 0) rc = zb_make_tmap_kv_cache(&tk, k_cache, slots, num_kv_heads, head_dim, kKeys);
  if (rc == 0) rc = zb_make_tmap_kv_cache(&tv, v_cache, slots, num_kv_heads, head_dim, kKeys);
  if (rc != 0) return rc;
  PrefillParams p;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.block_table = block_table;
  p.seq_lens = seq_lens;
  p.q_start = q_start;
  p.batch = batch;
  p.num_q_heads = num_q_heads;
  p.num_kv_heads = num_kv_heads;
  p.max_pages = max_pages;
  p.window = window;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (head_dim == 256) return launch_prefill<256>(tq, tk, tv, p, q_blocks, s);
  return head_dim == 64 ? launch_prefill<64>(tq, tk, tv, p, q_blocks, s) : launch_prefill<128>(tq, tk, tv, p, q_blocks, s);
}
