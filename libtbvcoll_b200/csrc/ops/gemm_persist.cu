// gemm_persist.cu — the many-token (prefill) form of the bf16 tcgen05 GEMM: a persistent kernel, one CTA per SM.
//
//   Y[n, m] = epilogue( sum_k X[n, k] * W[m, k] )      X: [N tokens, K], W: [M features, K], both bf16 row-major
//
// The decode form (gemm.cu) puts features on the 128-row UMMA M axis because a handful of tokens would
// waste it.  With hundreds of tokens the natural orientation is the other one: tokens on UMMA M and up to 256
// features on UMMA N.  A thread of the epilogue then owns one token row and reads consecutive features per
// TMEM load; gate/up pairs of the SiLU-mul epilogue sit in the same thread, so that epilogue needs no shuffles.
//
// Tile shapes (templates TH, FEAT); an SM takes in some 70 bytes per clock through TMA (measured with three quarters of the MMAs left out, 133 GB/s), which bounds the smaller ones:
//   TH = 1, FEAT = 128  128 tokens x 128 features: a quarter less work per byte than 256 features, for problems whose wider tiles would leave SMs idle
//           (1024 tokens, 2048 x 7168 37 us against 45, 512 tokens, 3072 x 2048 with rotation 20 against 23).
//   TH = 1  128 tokens x 256 features, two accumulator sets: the epilogue of a tile runs under the MMAs of the next.  For gated units, the rotation, and where
//           tiles are few.  4096 tokens: 28672 x 4096 with the SiLU unit 641 us = 1500 TFLOP/s (793 .. 848 with TH = 2), 6144 x 4096 with rotation 159 (166 with a TH = 2 that is gone).
//   TH = 2  256 tokens x 256 features as two 128-row MMAs that share one 256-row weight tile: a third less traffic per operation, but both accumulators belong
//           to one tile, so the epilogue (eight warps here, four per half) is exposed once per tile.  For stores, bf16 or fp32 (the choice does not look at an activation), and gated units of one or two rounds: 4096 x 4096 97 us (104 with TH = 1), 4096 x 14336 361 (402).
//
// The CTAs walk tiles id = first + i * step with the token tile fastest: the CTAs running at any
// moment share a few weight tiles (streamed from HBM once) and the activations stay in L2.  Warp 0
// lane 0 feeds a TMA ring that runs ahead across tile boundaries, warp 1 lane 0 issues tcgen05.mma, warps 2..
// drain TMEM.  The copying and the issuing thread have some 500 clocks per k-block: stage and phase are counted, a division by the number of
// stages or k-blocks cost a fifth of the rate.  Every wait is bounded; a wait that gives up raises the CTA's abort flag, all roles leave their
// loops, TMEM is freed and the host-visible error flag is set.  (The reference has no GEMM; see gemm.cu for
// what this path replaces.)
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdio.h>

#include <type_traits>

#include "gemm.cuh"
#include "ops.h"

using namespace sm100;

namespace {

constexpr int kHalfBytes = 128 * gemm::kBK * 2;      // one 128-token operand tile: 16 KB
constexpr int kMaxStages = 6;

template <int TH, int FEAT> struct Shape {
  static constexpr int kTok = 128 * TH;                        // tokens per tile
  static constexpr int kXBytes = kHalfBytes * TH;
  static constexpr int kStageBytes = kXBytes + FEAT * gemm::kBK * 2;        // 48 / 32 / 64 KB
  static constexpr int kStages = 192 * 1024 / kStageBytes;     // 4 / 6 / 3
  static constexpr int kBuffers = TH == 1 ? 2 : 1;             // accumulator sets that alternate between tiles
  static constexpr int kCols = 2 * FEAT;                       // TMEM columns of two sets, or of two halves
  static constexpr int kEpiWarps = 4 * TH;
  static constexpr int kThreads = 64 + 32 * kEpiWarps;         // a warp of copies, one of products, the epilogue's
};

constexpr int kMaxRowGroups = 512;

// Where a tile of a row-grouped problem lies: tiles are numbered group after group, inside a group token tile fastest.
struct RowGroups {
  int off[kMaxRowGroups + 1];      // first row of every group
  int tile[kMaxRowGroups + 1];     // first tile of every group
};
constexpr int kFeatTile = 256;     // of row-grouped problems

// first token row, end of the rows, first feature and its weight row of a tile
struct At { int n0, nend, f0, w0; };
template <int TOK>
__device__ __forceinline__ At find_tile(const RowGroups& groups, int tile, int ngroups, int M) {
  int lo = 0, hi = ngroups - 1;                    // the last group whose first tile is not beyond `tile`; empty groups are passed over
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (groups.tile[mid] <= tile) lo = mid;
    else hi = mid - 1;
  }
  const int local = tile - groups.tile[lo], tt = (groups.off[lo + 1] - groups.off[lo] + TOK - 1) / TOK;
  const int f0 = local / tt * kFeatTile;
  return At{groups.off[lo] + local % tt * TOK, groups.off[lo + 1], f0, lo * M + f0};
}

// Fills the table from the rows' offsets (device memory); whole CTA of THREADS.
template <int TOK, int THREADS>
__device__ __forceinline__ void count_tiles(RowGroups& groups, const gemm::Params& p, int feat_tiles) {
  for (int g = threadIdx.x; g <= p.groups; g += THREADS) groups.off[g] = p.row_off[g];
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x, per = (p.groups + 31) / 32, a = min(p.groups, lane * per), b = min(p.groups, a + per);
    auto count = [&](int g) { return (groups.off[g + 1] - groups.off[g] + TOK - 1) / TOK * feat_tiles; };
    int sum = 0;
    for (int g = a; g < b; g++) sum += count(g);
    int inc = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    int run = inc - sum;
    for (int g = a; g < b; g++) { groups.tile[g] = run; run += count(g); }
    if (lane == 31) groups.tile[p.groups] = inc;
  }
  __syncthreads();
}

struct PSmem {
  unsigned long long full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {  // 32 lanes x 32 consecutive fp32 columns
  tmem_ld16(taddr, r);
  tmem_ld16(taddr + 16u, r + 16);
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
// Same arithmetic as the decode kernel's SiLU-mul: every intermediate an unfused bf16 pipeline would
// have stored is rounded to bf16.
__device__ __forceinline__ float silu_mul_bf16(float g, float u) {
  g = bf16_round(g);
  u = bf16_round(u);
  const float s = bf16_round(g / (1.0f + __expf(-g)));
  return s * u;
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// One 32-byte store: a whole sector per thread, where rows of different tokens sit in neighbouring threads.
__device__ __forceinline__ void st_global_f32x8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]),
               "f"(v[6]), "f"(v[7]) : "memory");
}

__device__ __forceinline__ void st_global_b32x8(void* p, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// One token row, 16 features starting at f: the bf16 results (8 words, or 4 where gate and up make one) into w, fp32 results to memory.
template <int EPI>
__device__ __forceinline__ void finish16(const gemm::Params& p, int n, int f, const uint32_t* q, uint32_t* w) {
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; j++) v[j] = __uint_as_float(q[j]);
  if (p.bias) {
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] += __bfloat162float(p.bias[f + j]);
  }
  if (EPI == gemm::kEpiF32) {
    if (p.act == gemm::kActSoftplus) {              // one branch, not one per value
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = gemm::apply_act(v[j], gemm::kActSoftplus, 0.f);
    } else if (p.act != gemm::kActNone) {
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = gemm::apply_act(v[j], p.act, p.act_a);
    }
    float* dst = p.yf + size_t(n) * p.ldy + f;      // 64-byte aligned rows: M and ldy are multiples of 16 and 8
    st_global_f32x8(dst, v);
    st_global_f32x8(dst + 8, v + 8);
    if (p.y2) {
      uint4* d2 = reinterpret_cast<uint4*>(p.y2 + size_t(n) * p.ldy + f);
      d2[0] = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
      d2[1] = make_uint4(pack_bf16(v[8], v[9]), pack_bf16(v[10], v[11]), pack_bf16(v[12], v[13]), pack_bf16(v[14], v[15]));
    }
  } else if (EPI == gemm::kEpiClampGlu) {
#pragma unroll
    for (int j = 0; j < 4; j++)
      w[j] = pack_bf16(gemm::clamp_glu(v[4 * j], v[4 * j + 1], p.act_a, p.act_b, p.act_c), gemm::clamp_glu(v[4 * j + 2], v[4 * j + 3], p.act_a, p.act_b, p.act_c));
  } else if (EPI == gemm::kEpiSiluMul) {
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = pack_bf16(silu_mul_bf16(v[4 * j], v[4 * j + 1]), silu_mul_bf16(v[4 * j + 2], v[4 * j + 3]));
  } else {
    if (p.act != gemm::kActNone && f < p.act_m) {   // act_m is a multiple of 16
      if (p.act == gemm::kActSilu) {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = gemm::apply_act(v[j], gemm::kActSilu, 0.f);
      } else if (p.act == gemm::kActGelu) {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = gemm::apply_act(v[j], gemm::kActGelu, 0.f);
      } else {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = gemm::apply_act(v[j], p.act, p.act_a);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) w[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
  }
}
// 32 features of one token row.  The rows of a warp lie far apart in memory, so the stores cost a pass of the load / store unit per row and instruction: 32 bytes at a time
// (p.wide: rows and base allow it) are half as many as 16.
template <int EPI>
__device__ __forceinline__ void store32(const gemm::Params& p, int n, int f, const uint32_t* q) {
  uint32_t w[16];
  constexpr bool kHalf = EPI == gemm::kEpiSiluMul || EPI == gemm::kEpiClampGlu;
  finish16<EPI>(p, n, f, q, w);
  const bool second = f + 16 < p.M;                 // M is a multiple of 16
  if (second) finish16<EPI>(p, n, f + 16, q + 16, w + (kHalf ? 4 : 8));
  if constexpr (EPI != gemm::kEpiF32) {
    __nv_bfloat16* dst = p.y + size_t(n) * p.ldy + (kHalf ? f >> 1 : f);
    if (kHalf) {
      if (p.wide && second) {
        st_global_b32x8(dst, w);
      } else {
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        if (second) *reinterpret_cast<uint4*>(dst + 8) = make_uint4(w[4], w[5], w[6], w[7]);
      }
    } else if (p.wide) {
      st_global_b32x8(dst, w);
      if (second) st_global_b32x8(dst + 16, w + 8);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j < 2 || second) *reinterpret_cast<uint4*>(dst + 8 * j) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
    }
  }
}

// cos and sin of 16 channels for a row's position, rounded as the two-kernel form rounds them
struct Angles { float c[16], s[16]; };
__device__ __forceinline__ void ld_global_f32x8(const float* p, float* v) {
  asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}
__device__ __forceinline__ void load_angles(const gemm::Params& p, int pos, int d, Angles& a) {
  const float* t = p.rope.cos_sin + size_t(pos) * 128 + d;
  ld_global_f32x8(t, a.c);
  ld_global_f32x8(t + 8, a.c + 8);
  ld_global_f32x8(t + 64, a.s);
  ld_global_f32x8(t + 72, a.s + 8);
#pragma unroll
  for (int j = 0; j < 16; j++) { a.c[j] = bf16_round(a.c[j]); a.s[j] = bf16_round(a.s[j]); }
}
// One token row, 16 channels d .. of a head and their rotation partners 64 further (`a`, `b`: accumulators): bias, rounding to bf16, rotation, stores to the activations and
// the cache.  Same arithmetic as k_gemm_qkv_rope.
__device__ __forceinline__ void store_rope16(const gemm::Params& p, int n, int head, int d, const Angles& g, long long slot, const uint32_t* a, const uint32_t* b) {
  float lo[16], hi[16];
#pragma unroll
  for (int j = 0; j < 16; j++) { lo[j] = __uint_as_float(a[j]); hi[j] = __uint_as_float(b[j]); }
  if (p.bias) {
    const __nv_bfloat16* bias = p.bias + head * 128 + d;
#pragma unroll
    for (int j = 0; j < 16; j++) { lo[j] += __bfloat162float(bias[j]); hi[j] += __bfloat162float(bias[64 + j]); }
  }
  if (head < p.rope.nq + p.rope.nkv) {
#pragma unroll
    for (int j = 0; j < 16; j++) gemm::rotate(bf16_round(lo[j]), bf16_round(hi[j]), g.c[j], g.s[j], lo[j], hi[j]);
  }
  uint32_t w[16];
#pragma unroll
  for (int j = 0; j < 8; j++) { w[j] = pack_bf16(lo[2 * j], lo[2 * j + 1]); w[8 + j] = pack_bf16(hi[2 * j], hi[2 * j + 1]); }
  auto put = [&](__nv_bfloat16* row) {                // 32-byte aligned: see tbv_op_gemm_qkv_rope
    st_global_b32x8(row + d, w);
    st_global_b32x8(row + d + 64, w + 8);
  };
  put(p.y + size_t(n) * p.ldy + head * 128);
  if (slot >= 0 && head >= p.rope.nq) {
    const bool value = head >= p.rope.nq + p.rope.nkv;
    put((value ? p.rope.v_cache : p.rope.k_cache) + (size_t(slot) * p.rope.nkv + (head - p.rope.nq - (value ? p.rope.nkv : 0))) * 128);
  }
}

// A warp's 32 rows of an accumulator of FEAT columns (`trow`: its TMEM address), token row n of this lane, features f0 ..; release(): called by the whole warp when the
// accumulator has been read.
template <int EPI, int FEAT, typename F>
__device__ __forceinline__ void drain(const gemm::Params& p, int n, bool row_ok, int f0, uint32_t trow, F release) {
  if constexpr (EPI == gemm::kEpiRope) {
    // rotation partners lie 64 columns apart: 16 channels of every head of the tile and their partners at a time, with the angles they share
    int pos = 0;
    long long slot = -1;
    if (row_ok) {
      pos = p.rope.positions[n];
      pos = pos < 0 ? 0 : (pos >= p.rope.max_pos ? p.rope.max_pos - 1 : pos);
      if (p.rope.slot_mapping) slot = p.rope.slot_mapping[n];
    }
    const bool turned = (f0 >> 7) < p.rope.nq + p.rope.nkv;       // otherwise the tile holds values only
    Angles g;
#pragma unroll 1
    for (int d = 0; d < 64; d += 16) {
      if (turned) load_angles(p, pos, d, g);
#pragma unroll
      for (int h = 0; h < FEAT; h += 128) {
        uint32_t a[16], b[16];
        __syncwarp();
        tmem_ld16(trow + uint32_t(h + d), a);
        tmem_ld16(trow + uint32_t(h + d + 64), b);
        tmem_ld_wait();
        if (d == 48 && h + 128 == FEAT) {
          tc_fence_before();
          __syncwarp();
          release();
        }
        if (row_ok && f0 + h < p.M) store_rope16(p, n, (f0 + h) >> 7, d, g, slot, a, b);   // M is a multiple of 128
      }
    }
  } else {
    for (int c = 0; c < FEAT; c += 32) {
      uint32_t r[32];
      __syncwarp();   // rows past the end skip the stores below: reconverge before the warp-wide load
      tmem_ld32(trow + uint32_t(c), r);
      tmem_ld_wait();
      if (c + 32 == FEAT) {
        // accumulator fully read by this warp: hand it back to the MMA warp before the last stores go out
        tc_fence_before();
        __syncwarp();
        release();
      }
      if (row_ok && f0 + c < p.M) store32<EPI>(p, n, f0 + c, r);
    }
  }
}

// EPI (gemm::Epi) of all kernels here: 0 store (+bias); 1 SiLU-mul over interleaved gate/up features (output has M / 2 features); 2 fp32 store with
// an activation; 3 clamped gated unit over interleaved gate/up features; 4 rotation and cache write of a qkv projection.
// ROWS: row-grouped problem (p.row_off; FEAT = 256).
template <int EPI, int TH, int FEAT, bool ROWS>
__global__ void __launch_bounds__(Shape<TH, FEAT>::kThreads, 1)
k_gemm_tok(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ gemm::Params p) {
  using S = Shape<TH, FEAT>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ PSmem s;
  __shared__ typename std::conditional<ROWS, RowGroups, int>::type groups;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const int tok_tiles = (p.N + S::kTok - 1) / S::kTok, feat_tiles = (p.M + FEAT - 1) / FEAT, nkb = p.kb_total;

  if (threadIdx.x == 0) {
    for (int i = 0; i < S::kStages; i++) {
      mbar_init(smem_u32(&s.full[i]), 1);
      mbar_init(smem_u32(&s.empty[i]), 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(smem_u32(&s.acc_full[i]), 1);
      mbar_init(smem_u32(&s.acc_empty[i]), S::kEpiWarps);   // one arrival per epilogue warp
    }
    s.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&s.tmem_base), S::kCols);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl::launch_dependents();
  int tiles = tok_tiles * feat_tiles;
  if constexpr (ROWS) {
    pdl::grid_dependency_wait();                 // the groups' rows were counted on the device by a kernel before this one
    count_tiles<S::kTok, S::kThreads>(groups, p, feat_tiles);
    tiles = groups.tile[p.groups];
  }
  const int my_tiles = int(blockIdx.x) < tiles ? (tiles - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x) : 0;
  const int ngroups = p.groups, feats = p.M, all_rows = p.N;
  // (by value: a capture of the parameter block would put it in local memory)
  auto locate = [=](int tile) -> At {
    if constexpr (ROWS) return find_tile<S::kTok>(groups, tile, ngroups, feats);
    const int f0 = tile / tok_tiles * FEAT;
    return At{tile % tok_tiles * S::kTok, all_rows, f0, f0};
  };
  const uint32_t tmem0 = s.tmem_base;
  volatile int* abortp = &s.abort_flag;

  if (warp == 0 && lane == 0) {
    // ---- TMA producer: one flat sequence of k-blocks over all of this CTA's tiles ----
    const uint64_t pol_x = policy_evict_last();
    // Weights are never written by a kernel: the first ring fill of weight tiles goes out before the
    // preceding kernel has finished; the activations follow once it has.
    const int pre = my_tiles ? min(S::kStages, nkb) : 0;
    At at = my_tiles ? locate(int(blockIdx.x)) : At{};
    for (int i = 0; i < pre; i++) {
      const uint32_t fb = smem_u32(&s.full[i]);
      mbar_expect_tx(fb, S::kStageBytes);
      tma_load_2d(base + i * S::kStageBytes + S::kXBytes, &tmW, i * gemm::kBK, at.w0, fb);
    }
    pdl::grid_dependency_wait();
    for (int i = 0; i < pre; i++) tma_load_2d_hint(base + i * S::kStageBytes, &tmX, i * gemm::kBK, at.n0, smem_u32(&s.full[i]), pol_x);
    int st = pre == S::kStages ? 0 : pre;
    uint32_t ph = pre == S::kStages ? 1u : 0u;   // of the ring's current round
    bool ok = true;
    for (int t = 0; t < my_tiles && ok; t++) {
      if (t) at = locate(int(blockIdx.x) + t * int(gridDim.x));
      for (int kb = t ? 0 : pre; kb < nkb; kb++) {
        if (!mbar_wait(smem_u32(&s.empty[st]), ph ^ 1u, abortp, p.limit_ns)) { ok = false; break; }
        const uint32_t fb = smem_u32(&s.full[st]);
        mbar_expect_tx(fb, S::kStageBytes);
        tma_load_2d_hint(base + st * S::kStageBytes, &tmX, kb * gemm::kBK, at.n0, fb, pol_x);
        tma_load_2d(base + st * S::kStageBytes + S::kXBytes, &tmW, kb * gemm::kBK, at.w0, fb);
        if (++st == S::kStages) { st = 0; ph ^= 1u; }
      }
    }
    if (*abortp && pre) {
      // gave up: let the copies already in flight land before this CTA's shared memory goes away (a millisecond is many times what a copy takes)
      const unsigned long long t0 = globaltimer();
      while (globaltimer() - t0 < 1000000ull) __nanosleep(1000);
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer ----
    const uint32_t idesc = umma_idesc_bf16(128, FEAT);
    int st = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = 0; t < my_tiles && ok; t++) {
      const int buf = t % S::kBuffers, use = t / S::kBuffers;
      // the epilogue must have drained this accumulator set (kBuffers tiles ago); passes at once on first use
      if (!mbar_wait(smem_u32(&s.acc_empty[buf]), (uint32_t(use) & 1u) ^ 1u, abortp, p.limit_ns)) break;
      tc_fence_after();
      for (int kb = 0; kb < nkb; kb++) {
        if (!mbar_wait(smem_u32(&s.full[st]), ph, abortp, p.limit_ns)) { ok = false; break; }
        tc_fence_after();
        const uint64_t bd = umma_desc_sw128(base + st * S::kStageBytes + S::kXBytes);
#pragma unroll
        for (int h = 0; h < TH; h++) {           // the 128-token halves share the weight tile
          const uint64_t ad = umma_desc_sw128(base + st * S::kStageBytes + h * kHalfBytes);
          const uint32_t tmem_d = tmem0 + uint32_t((TH == 1 ? buf : h) * FEAT);
#pragma unroll
          for (int k = 0; k < gemm::kBK / 16; k++)
            umma_bf16(tmem_d, ad + uint64_t(2 * k), bd + uint64_t(2 * k), idesc, (kb | k) != 0 ? 1u : 0u);
        }
        umma_commit(smem_u32(&s.empty[st]));
        if (++st == S::kStages) { st = 0; ph ^= 1u; }
      }
      if (ok) umma_commit(smem_u32(&s.acc_full[buf]));
    }
  } else if (warp >= 2) {
    // ---- epilogue: thread = one token row of the tile (TH = 2: warps 2..5 first half, 6..9 second half) ----
    const int quarter = warp & 3, half = TH == 1 ? 0 : (warp - 2) >> 2;
    for (int t = 0; t < my_tiles; t++) {
      const int buf = t % S::kBuffers, use = t / S::kBuffers;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s.acc_full[buf]), uint32_t(use) & 1u, abortp, p.limit_ns));   // together, before the warp-wide TMEM loads
      if (!ok) break;
      tc_fence_after();
      const At at = locate(int(blockIdx.x) + t * int(gridDim.x));
      const int n = at.n0 + half * 128 + quarter * 32 + lane;   // token row
      drain<EPI, FEAT>(p, n, n < at.nend, at.f0, tmem0 + (uint32_t(quarter * 32) << 16) + uint32_t((TH == 1 ? buf : half) * FEAT), [&] {
        if (lane == 0) mbar_arrive(smem_u32(&s.acc_empty[buf]));
      });
    }
  }

  // ---- teardown: everybody is done with TMEM ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(s.tmem_base, S::kCols);
  }
  if (threadIdx.x == 0 && s.abort_flag && p.err) atomicExch(p.err, 1);
}

template <int EPI, int TH, int FEAT, bool ROWS = false>
cudaError_t launch_tok(const void* w, const void* x, const gemm::Params& p, int ldx, cudaStream_t st, int* map_rc) {
  using S = Shape<TH, FEAT>;
  CUtensorMap tmX, tmW;
  *map_rc = 0;
  if (tbvops::make_tensor_map_bf16(&tmX, x, ROWS ? p.x_rows : p.N, p.K, ldx, S::kTok) != 0 ||
      tbvops::make_tensor_map_bf16(&tmW, w, (unsigned long long)(ROWS ? p.groups : 1) * p.M, p.K, p.K, FEAT) != 0) {
    *map_rc = -3;
    return cudaSuccess;
  }
  constexpr size_t smem = size_t(S::kStages) * S::kStageBytes + 1024;
  static std::atomic<unsigned> done{0};
  const cudaError_t attr = pdl::allow_smem(k_gemm_tok<EPI, TH, FEAT, ROWS>, smem, done);
  if (attr != cudaSuccess) return attr;
  const int tiles = (ROWS ? p.x_rows / S::kTok + p.groups : (p.N + S::kTok - 1) / S::kTok) * ((p.M + FEAT - 1) / FEAT);   // ROWS: at most
  const int sms = tbvops::sm_count();
  return pdl::launch(k_gemm_tok<EPI, TH, FEAT, ROWS>, dim3(tiles < sms ? tiles : sms), dim3(S::kThreads), smem, st, 1, tmX, tmW, p);
}

}  // namespace

namespace tbvops {

// Which form takes an [N tokens] x [M features] problem: 0 = the decode-form kernel (gemm.cu), k_gemm_tok with 1 / 2 = 128- / 256-token tiles of 256 features, 3 = 128 x 128
// tiles.  `mode`: 1 = choose, 2 / 3 / 4 = force the first / second / third tile wherever the shape allows (tests, measurements; the qkv projection, which asks for epilogue 1, has no 256-token tile and takes 128 x 256 instead).
//
// Every CTA walks ceil(tiles / SMs) tiles.  A k-block of a 128 x 128 tile takes two thirds of the time of a 128 x 256 one (both bound by what TMA brings in), and one of
// 256 x 256 nine tenths of two of those.  512 tokens, 4096 x 4096 24 / 28 / 45 us with 128 x 128 / 128 x 256 / 256 x 256 tiles,
// 1024 tokens, 14336 x 2048 with the SiLU unit 75 / 61.  A gated unit's epilogue is long (10 us for 128 rows) and exposed in 256-token tiles: they pay where all of the problem is
// one round of them instead of two, or two instead of four of long K, and with short K, where the epilogue is all there is and they have twice the warps for it (us, 128 x 256 / 256 x 256 with the SiLU unit: 512 tokens, 14336 x 4096 62 / 56, 2048 tokens, 4096 x 14336
// 189 / 165, 4096 x 1792 35 / 32, 1024 tokens, 7168 x 8192 107 / 95; 4096 tokens, 4096 x 8192 217 / 197, 14336 x 128 143 / 85, 14336 x 1024 158 / 144; but 14336 x 2048 on 1000 60 / 64, 8192 x 4096 on 3000 150 / 162).
// Fewer than 384 tokens, and problems of few tiles, go to the decode form, which shares K out over clusters (512 tokens, fp32, 2048 x 4096: 19 us
// against 24; 1024 tokens 28 against 24; 512 tokens, 2048 x 2048 15.3 against 13.5).  With long K a CTA here walks all of it (0.3 us per k-block of a 128 x 128 tile, one after
// another) while the decode form takes some 1.6 us per 128 x 256 tile of its own, and per k-block only a little: it wins while it has fewer tiles than a fifth of the k-blocks
// (us, decode form / here: 512 tokens, 288 x 8192 17 / 38, 1280 x 8192 34 / 39, 1024 x 14336 43 / 67, 512 x 28672 32 / 126; 2048 tokens, 288 x 8192 33 / 39,
// 1024 x 28672 143 / 156; the other side: 512 tokens, 1024 x 5120 28 / 26, 2048 x 7168 48 / 36, 1024 tokens, 1280 x 8192 47 / 41, 2048 tokens, 2048 x 28672 247 / 185).  With fp32
// results the decode form keeps to a CTA per SM and wins further (2048 tokens, 512 x 8192 24 / 41, 1024 x 14336 58 / 68; 512 tokens, 2560 x 8192 39 / 42; the other side: 1536 tokens, 1024 x 5120 31 / 28,
// 2048 tokens, 2048 x 28672 212 / 208).
int gemm_tok_choose(int M, int N, int K, int ldy, int epi, int mode, int sms) {
  if (!(N >= 384 && (M % 16) == 0 && (K % 8) == 0 && (ldy % 8) == 0 && epi >= 0 && epi <= 3)) return 0;
  const bool stores = epi == gemm::kEpiStore || epi == gemm::kEpiF32;
  if (mode >= 2) return mode == 4 ? 3 : (mode == 3 ? 2 : 1);
  const long f256 = (M + 255) / 256, f128 = (M + 127) / 128, n128 = (N + 127) / 128, n256 = (N + 255) / 256;
  auto rounds = [&](long tiles) { return (tiles + sms - 1) / sms; };
  const long kb = (K + 63) / 64, decode = f128 * n256;
  if (K <= 4096 ? n128 * f128 * (K > 2048 ? 2 : 4) <= sms : epi == gemm::kEpiF32 ? decode <= 32 || (decode <= 96 && 5 * decode <= 2 * kb) : 5 * decode < kb) return 0;
  const long r1 = rounds(n128 * f256), r2 = rounds(n256 * f256);
  if (2 * rounds(n128 * f128) < 3 * r1) return 3;
  if (stores) return 18 * r2 <= 10 * r1 ? 2 : 1;
  if (K <= 1024) return 3 * r2 <= 2 * r1 ? 2 : 1;
  return 2 * r2 <= r1 && (r2 == 1 || (r2 == 2 && K > 4096)) ? 2 : 1;
}

// Row-grouped: 0 the decode form, 1 / 2 k_gemm_tok with 128- / 256-token tiles of 256 features (`mode` 2 and 4 / 3 force them).  The decode form re-reads a group's weights
// for every tile of up to 128 rows; k_gemm_tok wastes what a group's last tile lacks, on average half a tile.
//
// How the rows spread over the groups is not known here, and 256-token tiles lose up to half where they need a round more (8 x 513 rows, 2048 x 3584: 89 us against 59).
// They pay for plain stores where K is long (their epilogue is exposed), groups are large against a tile and rounds are many: 4096 x 7168, 8 groups of 768 / 1000 /
// 2048 rows 259 / 338 / 601 us against 282 / 367 / 664, 16 of 1500 1031 against 1040; but 16 of 500 428 against 398; with K 3584 8 of 2000 340 against 330.
int gemm_tok_rows_choose(int M, int x_rows, int groups, int K, int epi, int mode, int sms) {
  if ((M % 16) || groups > kMaxRowGroups || x_rows / groups < 64) return 0;
  if (epi != gemm::kEpiStore || mode == 2 || mode == 4) return 1;
  if (mode == 3) return 2;
  const long tiles = (x_rows / 256 + groups / 2) * (long)((M + 255) / 256);
  return K > 4096 && x_rows / groups >= 768 && tiles >= 3l * sms ? 2 : 1;
}

int gemm_tok_launch(const void* w, const void* x, void* y, const void* bias, int M, int N, int K, int ldx, int ldy, int epi, int th,
                    void* stream) {
  gemm::Params p{};
  p.M = M; p.N = N; p.K = K; p.ldy = ldy;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.y = static_cast<__nv_bfloat16*>(y);
  return gemm_tok_launch_p(w, x, p, ldx, epi, th, stream);
}

int gemm_tok_launch_p(const void* w, const void* x, gemm::Params& p, int ldx, int epi, int th, void* stream) {
  p.bn = 256; p.splits = 1;
  p.kb_total = (p.K + 63) / 64;
  p.wide = !(reinterpret_cast<uintptr_t>(p.y) & 31) && p.ldy % 16 == 0;
  p.limit_ns = 2000000000ull;
  p.err = gemm_err_flag();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int map_rc = 0;
  cudaError_t e;
  if (p.row_off) {
    e = epi == gemm::kEpiClampGlu ? launch_tok<3, 1, 256, true>(w, x, p, ldx, st, &map_rc) :
        th == 2 ? launch_tok<0, 2, 256, true>(w, x, p, ldx, st, &map_rc) : launch_tok<0, 1, 256, true>(w, x, p, ldx, st, &map_rc);
  } else switch (epi) {
    case gemm::kEpiSiluMul:
      e = th == 3 ? launch_tok<1, 1, 128>(w, x, p, ldx, st, &map_rc) : th == 2 ? launch_tok<1, 2, 256>(w, x, p, ldx, st, &map_rc) : launch_tok<1, 1, 256>(w, x, p, ldx, st, &map_rc);
      break;
    case gemm::kEpiF32:
      e = th == 3 ? launch_tok<2, 1, 128>(w, x, p, ldx, st, &map_rc) : th == 2 ? launch_tok<2, 2, 256>(w, x, p, ldx, st, &map_rc) : launch_tok<2, 1, 256>(w, x, p, ldx, st, &map_rc);
      break;
    case gemm::kEpiClampGlu:
      e = th == 3 ? launch_tok<3, 1, 128>(w, x, p, ldx, st, &map_rc) : th == 2 ? launch_tok<3, 2, 256>(w, x, p, ldx, st, &map_rc) : launch_tok<3, 1, 256>(w, x, p, ldx, st, &map_rc);
      break;
    case gemm::kEpiRope:   // no 256-token form
      e = th == 3 ? launch_tok<4, 1, 128>(w, x, p, ldx, st, &map_rc) : launch_tok<4, 1, 256>(w, x, p, ldx, st, &map_rc); break;
    default:
      e = th == 3 ? launch_tok<0, 1, 128>(w, x, p, ldx, st, &map_rc) : th == 2 ? launch_tok<0, 2, 256>(w, x, p, ldx, st, &map_rc) : launch_tok<0, 1, 256>(w, x, p, ldx, st, &map_rc);
      break;
  }
  if (map_rc != 0) return map_rc;
  if (e != cudaSuccess) {
    fprintf(stderr, "[tbvops] many-token gemm launch failed: %s (M=%d N=%d K=%d tile %d)\n", cudaGetErrorString(e), p.M, p.N, p.K, th);
    return -1;
  }
  return 0;
}

}  // namespace tbvops
