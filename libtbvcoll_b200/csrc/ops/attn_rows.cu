// attn_rows.cu — paged attention of single query rows (decode), heads of 128 channels, keys and values in caches of their own, up to eight query heads per key head.
//
// One row and key head per CTA and split; grid (rows, kv_heads, splits), cluster (1, 1, splits).  As in k_shared_rows (shared_attn.cu) every warp walks units of 16 tokens
// on its own: a ring of three units, a running maximum, sums in registers; the results of the warps are merged at the end, then those of the cluster, in fixed order.
// Tokens (scores) and channels (sums) sit on the M side of the products and heads on the N side.  A unit is four TMA boxes of 16 tokens x 64 channels (128-byte swizzle),
// one instruction each: the lanes of a warp compute no addresses and no cached byte passes a register on its way in.
//
// Bound by HBM with long contexts: 32 rows x 8192 tokens, 4 key heads, 85 us = 0.96 of a copy's 6.55 TB/s (123 us with tiles that the lanes copy, k_paged_attn_mma);
// 32 contexts of 1003 .. 7999 tokens 58 us (116), 32 x 2048 26 (34).  By the chain of context length, block table, first tile and merge with short ones: one row x 100
// tokens 3.5 us (4.4), 8 rows x 640, 8 key heads, 8.9 (9.2).  Where most splits have no token the set-up of the rings shows: one row x 16 tokens in 8 splits 5.9 us (5.3).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../pdl.cuh"
#include "attn_mma.cuh"
#include "ops.h"
#include "sm100.cuh"

using namespace attn_mma;

namespace {

constexpr int kD = 128, kTok = 16, kWarps = 4, kStages = 3, kMaxSplits = 8, kHeads = 8;
constexpr int kBox = kTok * 128, kUnit = 4 * kBox;                 // bytes: 16 tokens x 64 channels; a unit's keys and values
constexpr int kSmem = kWarps * kStages * kUnit + 1024;

struct Params {
  const __nv_bfloat16* q;    // [rows, ldq], head h at h * 128
  __nv_bfloat16* out;        // [rows, ldo]
  const int *tables, *seq_of_row, *ctx_lens;
  int ldq, ldo, kv_heads, G, block_size, max_blocks, splits;
  float scale_log2;
  int settled;               // 1: context lengths, tables and all cached tokens but each row's last were complete before the kernel in front of this one began
  int* err;
};

__global__ void __launch_bounds__(kWarps * 32, 2) k_attn_rows(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const Params p) {
  extern __shared__ uint8_t raw[];
  __shared__ unsigned long long full[kWarps][kStages];
  __shared__ float sh_m[kWarps][kHeads], sh_l[kWarps][kHeads], sh_ml[kHeads][2], sh_fac[kMaxSplits][kHeads], sh_sm[kMaxSplits][kHeads];
  __shared__ int abort_flag;
  pdl::launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r8 = lane >> 2, quad = lane & 3;
  if (lane == 0) {
    for (int s = 0; s < kStages; s++) sm100::mbar_init(smem_addr(&full[warp][s]), 1);
    if (warp == 0) {
      abort_flag = 0;
      sm100::tma_prefetch_desc(&tmK);
      sm100::tma_prefetch_desc(&tmV);
    }
    sm100::mbar_fence_init();
  }
  __syncthreads();
  if (!p.settled) pdl::grid_dependency_wait();
  const int row = blockIdx.x, h = blockIdx.y, sp = blockIdx.z, S = p.splits, G = p.G;
  const int ctx = min(p.ctx_lens[row], p.max_blocks * p.block_size);   // never walk past the block table (a captured loop replayed beyond the reserved length)
  const int* bt = p.tables + size_t(p.seq_of_row ? p.seq_of_row[row] : row) * p.max_blocks;
  int chunk = (ctx + S - 1) / S;
  chunk = (chunk + kTok - 1) / kTok * kTok;
  const int t0 = min(ctx, sp * chunk), t1 = min(ctx, t0 + chunk);
  const int units = (t1 - t0 + kTok - 1) / kTok, mine = units > warp ? (units - warp + kWarps - 1) / kWarps : 0;
  const uint32_t base = (smem_addr(raw) + 1023u) & ~1023u, ring = base + uint32_t(warp) * kStages * kUnit;

  // cache rows of this warp's unit i: looked up for 32 units at a time, a lane each
  int slot = 0;
  auto issue = [&](int i) {               // whole warp; unit i of this warp into its stage
    if (i >= mine) return;
    if ((i & 31) == 0) {
      const int tok = t0 + (warp + kWarps * (i + lane)) * kTok;
      slot = tok < t1 ? bt[tok / p.block_size] * p.block_size + tok % p.block_size : 0;
    }
    const int y = __shfl_sync(0xffffffffu, slot, i & 31);
    const uint32_t bar = smem_addr(&full[warp][i % kStages]);
    if (lane == 0) sm100::mbar_expect_tx(bar, kUnit);
    __syncwarp();
    if (lane < 4)                         // keys, keys, values, values: 64 channels each
      sm100::tma_load_2d(ring + (i % kStages) * kUnit + lane * kBox, lane < 2 ? &tmK : &tmV, h * kD + (lane & 1) * 64, y, bar);
  };
  if (p.settled) {
    // units without the last token, which the kernel in front writes, are on their way before it has finished
    int early = 0;
    while (early < min(mine, kStages) && t0 + (warp + kWarps * early + 1) * kTok < ctx) issue(early++);
    pdl::grid_dependency_wait();
    for (; early < kStages; early++) issue(early);
  } else {
#pragma unroll
    for (int i = 0; i < kStages; i++) issue(i);
  }

  // right operand of the scores: q^T, channels x heads
  uint32_t qf[kD / 16][2];
  const __nv_bfloat16* q = p.q + size_t(row) * p.ldq + size_t(h * G + (r8 < G ? r8 : 0)) * kD + quad * 2;
#pragma unroll
  for (int k = 0; k < kD / 16; k++)
#pragma unroll
    for (int j = 0; j < 2; j++) qf[k][j] = r8 < G ? *reinterpret_cast<const uint32_t*>(q + k * 16 + j * 8) : 0u;
  float o[kD / 16][4];                    // channels 16 k + r8 (+ 8), heads 2 quad (+ 1)
#pragma unroll
  for (int k = 0; k < kD / 16; k++) o[k][0] = o[k][1] = o[k][2] = o[k][3] = 0.f;
  float m[2] = {kNegBig, kNegBig}, l[2] = {0.f, 0.f};

  int done = 0;
  for (; done < mine; done++) {
    const int i = done, n = min(kTok, t1 - t0 - (warp + kWarps * i) * kTok);
    const uint32_t sk = ring + (i % kStages) * kUnit, sv = sk + 2 * kBox;
    if (!__all_sync(0xffffffffu, sm100::mbar_wait(smem_addr(&full[warp][i % kStages]), uint32_t(i / kStages) & 1u, &abort_flag, 2000000000ull))) break;
    if (n < kTok) {                       // behind the last token (the last unit there is): a weight of zero must not meet a stale bit pattern
      for (int c = lane; c < (kTok - n) * 16; c += 32) st_zero16(sv + (c & 1) * kBox + (n + (c >> 4)) * 128 + ((c >> 1) & 7) * 16);
      __syncwarp();
    }
    float s[4] = {0.f, 0.f, 0.f, 0.f};    // tokens r8 (+ 8), heads as in o
#pragma unroll
    for (int k = 0; k < kD / 16; k++) {
      uint32_t a[4];
      const int r = lane & 15, c = k * 2 + (lane >> 4);
      ldmatrix_x4(sk + (c >> 3) * kBox + r * 128 + (((c & 7) ^ (r & 7)) << 4), a);
      mma_bf16(s, a, qf[k][0], qf[k][1]);
    }
    float mx[2] = {m[0], m[1]};
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        float& v = s[2 * r + j];
        v = r * 8 + r8 < n ? v * p.scale_log2 : kNegBig;
        mx[j] = fmaxf(mx[j], v);
      }
    bool grew = false;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 4));
      mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 8));
      mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 16));
      grew |= mx[j] > m[j];
    }
    if (__any_sync(0xffffffffu, grew)) {
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float c = exp2f(m[j] - mx[j]);
        m[j] = mx[j];
        l[j] *= c;
#pragma unroll
        for (int k = 0; k < kD / 16; k++) { o[k][j] *= c; o[k][2 + j] *= c; }
      }
    }
    // weights as the right operand of the sums (tokens x heads): the accumulator tiles transposed
    uint32_t w[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const float p0 = exp2f(s[2 * r] - m[0]), p1 = exp2f(s[2 * r + 1] - m[1]);
      l[0] += p0;
      l[1] += p1;
      w[r] = transpose_8x8(pack_bf16(p0, p1));
    }
#pragma unroll
    for (int k = 0; k < kD / 16; k++) {
      uint32_t a[4];                      // values transposed: channels x tokens
      const int r = (lane & 7) + ((lane >> 4) << 3), c = k * 2 + ((lane >> 3) & 1);
      ldmatrix_x4_trans(sv + (c >> 3) * kBox + r * 128 + (((c & 7) ^ (r & 7)) << 4), a);
      mma_bf16(o[k], a, w[0], w[1]);
    }
    __syncwarp();
    issue(i + kStages);
  }
  if (done < mine) {
    // gave up: let the copies in flight land before this memory goes away, and report
    for (int i = done; i < mine && i < done + kStages; i++)
      for (int spin = 0; spin < 20000 && !sm100::mbar_try_wait(smem_addr(&full[warp][i % kStages]), uint32_t(i / kStages) & 1u); spin++) __nanosleep(50);
    if (lane == 0 && p.err) atomicExch(p.err, 1);
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    l[j] += __shfl_xor_sync(0xffffffffu, l[j], 4);
    l[j] += __shfl_xor_sync(0xffffffffu, l[j], 8);
    l[j] += __shfl_xor_sync(0xffffffffu, l[j], 16);
    if (r8 == 0) {
      sh_m[warp][quad * 2 + j] = m[j];
      sh_l[warp][quad * 2 + j] = l[j];
    }
  }
  __syncthreads();                        // the rings are free: their space takes the warps' sums [warps][8][128]
  float* so = reinterpret_cast<float*>(raw + (base - smem_addr(raw)));
#pragma unroll
  for (int k = 0; k < kD / 16; k++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int head = quad * 2 + (j & 1);
      if (head < G) so[(warp * kHeads + head) * kD + k * 16 + r8 + (j >> 1) * 8] = o[k][j];
    }
  if (tid < kHeads) {
    float mm = kNegBig, ll = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; w++) mm = fmaxf(mm, sh_m[w][tid]);
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
      const float f = exp2f(sh_m[w][tid] - mm);
      ll = fmaf(sh_l[w][tid], f, ll);
      sh_m[w][tid] = f;                   // factor of the warp from here on
    }
    sh_ml[tid][0] = mm;
    sh_ml[tid][1] = ll;
  }
  __syncthreads();
  __nv_bfloat16* out = p.out + size_t(row) * p.ldo + size_t(h) * G * kD;
  const int total = G * kD / 4;
  for (int i = tid; i < total; i += kWarps * 32) {
    const int head = i * 4 / kD;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
      const float4 v = *reinterpret_cast<const float4*>(so + w * kHeads * kD + i * 4);
      const float f = sh_m[w][head];
      a.x = fmaf(v.x, f, a.x); a.y = fmaf(v.y, f, a.y); a.z = fmaf(v.z, f, a.z); a.w = fmaf(v.w, f, a.w);
    }
    if (S == 1) {
      const float ll = sh_ml[head][1], f = ll > 0.f ? 1.f / ll : 0.f;
      *reinterpret_cast<uint2*>(out + i * 4) = make_uint2(pack_bf16(a.x * f, a.y * f), pack_bf16(a.z * f, a.w * f));
    } else {
      *reinterpret_cast<float4*>(so + i * 4) = a;
    }
  }
  if (S == 1) return;
  cluster_sync();
  if (tid < kHeads * kMaxSplits) {
    const int r = tid >> 3, head = tid & 7;
    const uint32_t a = smem_addr(&sh_ml[head][0]);
    sh_sm[r][head] = r < S && head < G ? ld_cluster_f32(a, r) : kNegBig;
    sh_fac[r][head] = r < S && head < G ? ld_cluster_f32(a + 4, r) : 0.f;
  }
  __syncthreads();
  if (tid < kHeads) {
    float mm = kNegBig, ll = 0.f;
    for (int r = 0; r < S; r++) mm = fmaxf(mm, sh_sm[r][tid]);
    for (int r = 0; r < S; r++) ll = fmaf(sh_fac[r][tid], exp2f(sh_sm[r][tid] - mm), ll);
    for (int r = 0; r < S; r++) sh_fac[r][tid] = ll > 0.f ? exp2f(sh_sm[r][tid] - mm) / ll : 0.f;
  }
  __syncthreads();
  const int per = (total + S - 1) / S;
  const uint32_t soa = smem_addr(so);
  for (int i = tid; i < per; i += kWarps * 32) {
    const int idx = sp * per + i;
    if (idx >= total) break;
    const int head = idx * 4 / kD;
    float4 v[kMaxSplits], a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < kMaxSplits; r++)
      if (r < S) v[r] = ld_cluster_f32x4(soa + idx * 16, r);
#pragma unroll
    for (int r = 0; r < kMaxSplits; r++)
      if (r < S) {
        const float f = sh_fac[r][head];
        a.x = fmaf(v[r].x, f, a.x); a.y = fmaf(v[r].y, f, a.y); a.z = fmaf(v[r].z, f, a.z); a.w = fmaf(v[r].w, f, a.w);
      }
    *reinterpret_cast<uint2*>(out + idx * 4) = make_uint2(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
  }
  cluster_sync();                         // nobody leaves while a peer may still read its shared memory
}

}  // namespace

namespace tbvops {

// kernel's limits: up to eight query heads per key head, blocks of a multiple of 16 tokens, aligned rows
bool attn_rows_takes(const void* q, const void* k_cache, const void* v_cache, const void* out, int heads, int kv_heads, int ldq, int ldo, int block_size) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache);
  return heads / kv_heads <= kHeads && !(at & 15) && !(reinterpret_cast<uintptr_t>(q) & 3) && !(reinterpret_cast<uintptr_t>(out) & 7) && !(ldq % 2) && !(ldo % 4) &&
         block_size % kTok == 0;
}

int attn_rows(const void* q, const void* k_cache, const void* v_cache, const int* tables, const int* seq_of_row, const int* ctx_lens, void* out, int rows, int heads,
              int kv_heads, int ldq, int ldo, int block_size, int max_blocks, int splits, float scale, bool settled, cudaStream_t st) {
  static std::atomic<unsigned> done{0};
  if (pdl::allow_smem(k_attn_rows, kSmem, done) != cudaSuccess) return -1;
  const unsigned long long width = (unsigned long long)kv_heads * kD;
  CUtensorMap mk, mv;
  if (make_tensor_map_bf16(&mk, k_cache, kAnyCacheRows, width, width, kTok) != 0 || make_tensor_map_bf16(&mv, v_cache, kAnyCacheRows, width, width, kTok) != 0) return -3;
  const Params p{static_cast<const __nv_bfloat16*>(q), static_cast<__nv_bfloat16*>(out), tables, seq_of_row, ctx_lens, ldq, ldo, kv_heads, heads / kv_heads, block_size,
                 max_blocks, splits, scale * kLog2e, settled, gemm_err_flag()};
  const cudaError_t e = pdl::launch(k_attn_rows, dim3(rows, kv_heads, splits), dim3(kWarps * 32), kSmem, st, splits, mk, mv, p);
  if (e != cudaSuccess) fprintf(stderr, "[tbvops] paged attention launch failed: %s\n", cudaGetErrorString(e));
  return e == cudaSuccess ? 0 : -1;
}

}  // namespace tbvops
