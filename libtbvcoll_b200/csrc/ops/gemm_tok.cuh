// gemm_tok.cuh — what the many-token GEMM kernels (gemm_persist.cu, gemm_pair.cu) share: the tiles of row-grouped problems and the epilogues, in which a thread owns one
// token row of an accumulator in TMEM.
#pragma once
#include "gemm.cuh"

namespace gemm_tok {

using namespace sm100;

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

__device__ __forceinline__ void ld_global_b32x8(const void* p, uint32_t* v) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "l"(p) : "memory");
}
// One token row, 32 features from f on: the residual stream (`old`: as it was), its gained copy; returns the squares' sum
__device__ __forceinline__ float store_resid32(const gemm::Params& p, int n, int f, const uint32_t* q, const uint32_t* old) {
  uint32_t h[16], y[16];
  float sum = 0.f;
  const uint4* gain = reinterpret_cast<const uint4*>(p.gain + f);
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const uint4 gq = __ldg(gain + u);
    const uint32_t g[4] = {gq.x, gq.y, gq.z, gq.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int j = 4 * u + i;
      h[j] = pack_bf16(__uint_as_float(q[2 * j]) + __uint_as_float(old[j] << 16), __uint_as_float(q[2 * j + 1]) + __uint_as_float(old[j] & 0xffff0000u));
      const float a = __uint_as_float(h[j] << 16), b = __uint_as_float(h[j] & 0xffff0000u);
      sum = fmaf(a, a, fmaf(b, b, sum));
      y[j] = pack_bf16(a * __uint_as_float(g[i] << 16), b * __uint_as_float(g[i] & 0xffff0000u));
    }
  }
  const size_t off = size_t(n) * p.ldy + f;
  st_global_b32x8(p.h + off, h);
  st_global_b32x8(p.h + off + 16, h + 8);
  st_global_b32x8(p.y + off, y);
  st_global_b32x8(p.y + off + 16, y + 8);
  return sum;
}

struct NoMore { __device__ __forceinline__ void operator()(int, int, uint32_t*) const {} };
// A warp's 32 rows of an accumulator of FEAT columns (`trow`: its TMEM address), token row n of this lane, features f0 ..; release(): called by the whole warp when the
// accumulator has been read; more(c, n, r): adds what others have of columns c .. c + n - 1.
template <int EPI, int FEAT, typename F, typename G = NoMore>
__device__ __forceinline__ void drain(const gemm::Params& p, int n, bool row_ok, int f0, uint32_t trow, F release, G more = G{}) {
  // behind a norm: the row's scale
  constexpr bool kScales = EPI == gemm::kEpiStore || EPI == gemm::kEpiSiluMul || EPI == gemm::kEpiRope;
  const bool scaled = kScales && p.sq;
  const float scale = scaled && row_ok ? gemm::row_scale(p, n) : 1.f;
  if constexpr (EPI == gemm::kEpiResid) {
    // the stream's old values are fetched 32 features ahead of their use (M is a multiple of 128)
    const __nv_bfloat16* h = p.h + size_t(n) * p.ldy + f0;
    const bool any = row_ok && f0 < p.M;
    uint32_t old[2][16];
    if (any) { ld_global_b32x8(h, old[0]); ld_global_b32x8(h + 16, old[0] + 8); }
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < FEAT; c += 32) {
      uint32_t r[32];
      __syncwarp();
      tmem_ld32(trow + uint32_t(c), r);
      if (c + 32 < FEAT && row_ok && f0 + c + 32 < p.M) { ld_global_b32x8(h + c + 32, old[(c >> 5) + 1 & 1]); ld_global_b32x8(h + c + 48, old[(c >> 5) + 1 & 1] + 8); }
      tmem_ld_wait();
      more(c, 32, r);
      if (c + 32 == FEAT) {
        tc_fence_before();
        __syncwarp();
        release();
      }
      if (row_ok && f0 + c < p.M) sum += store_resid32(p, n, f0 + c, r, old[c >> 5 & 1]);
    }
    if (any) p.sq_out[size_t(f0 / FEAT) * p.N + n] = sum;
  } else if constexpr (EPI == gemm::kEpiRope) {
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
        more(h + d, 16, a);
        more(h + d + 64, 16, b);
        if (scaled) {
#pragma unroll
          for (int j = 0; j < 16; j++) { a[j] = __float_as_uint(__uint_as_float(a[j]) * scale); b[j] = __float_as_uint(__uint_as_float(b[j]) * scale); }
        }
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
      more(c, 32, r);
      if (scaled) {
#pragma unroll
        for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) * scale);
      }
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

}  // namespace gemm_tok
