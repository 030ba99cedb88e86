// Row attention for prefill chunks with the query heads of one KV head handled together.
//
// The up to 16 query heads that share a KV head are rows of the M = 16 side of m16n8k16 tiles.  A warp keeps everything of its tile in
// registers: scores of a key tile, their exponentials (a score fragment is the A fragment of P V as it stands), the
// running maximum and sum of its rows, 16 x 128 outputs.  Two forms:
//   selection list / dense prefix   one CTA per (KV head, row); each of the four warps walks every fourth tile of 16 keys
//       through a ring of its own (no barrier inside the walk) and the four partial results are merged at the end.
//       Bound by the gather, 1.3 MB per CTA at 2048 keys: 2048 rows x 4 KV heads in 1.51 ms, 7.1 TB/s out of the L2.
//   sliding window   one CTA per (KV head, 4 warps x 16 / heads rows): neighbouring rows share all but one key of their
//       window, so the rows' keys are staged once, 32 at a time, and every warp masks what its rows do not see.  Window 128,
//       2048 rows x 64 heads: 116 us, 2.5 of them for the look at what came out (attn_window_kernel's end).
// A 16,001-token document of two sparse and four window layers spends 27.8 ms in them; 61.2 ms when every row gathered its keys for
// itself into tiles that eight warps shared between four barriers.
// Against fp64 (bf16 outputs, windows / lists of 2048 / prefixes): 1.82e-3 / 1.81e-3 / 1.79e-3; before 1.84e-3 / 1.91e-3 / 1.88e-3.
// With M = 16 live rows there is no 128-lane UMMA shape to fill, which is why this uses warp-level MMAs rather than tcgen05.
//
// Output: bf16-rounded o, written as bf16 and/or as the e4m3 packet (one power-of-two scale per head) that
// the o_proj GEMM consumes.  Probabilities are rounded to bf16 before P V (and summed as rounded), so results
// differ from attn_rows_kernel in the last bits; the step/verify path keeps attn_rows_kernel.
//
// Reference counterpart: naivert/kernels/naive_n0p5/prefill_ext (FA4 CuTe sliding-window attention,
// naive_ops sparse attention); same math, different tiling.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include <string.h>

#include <type_traits>

#include "gemm.cuh"
#include "launch.hpp"

using namespace nrt;

namespace {

struct AttnArgs {               // must match target_kernels.cu
  const __nv_bfloat16* q;
  const __nv_bfloat16* k_cache;
  const __nv_bfloat16* v_cache;
  const int* pos0;
  int rows, heads, kv_heads, head_dim, v_dim;
  float scale;
  int mode;
  int window, ring;
  const __nv_bfloat16* sink;
  const int* sel;
  int top_k;
  const __nv_bfloat16* k_blk;
  const __nv_bfloat16* v_blk;
  __nv_bfloat16* o_bf16;
  uint8_t* o8;
  float* o_scale;
  float* part;
  unsigned int* tickets;
  unsigned long long* stamps;   // opt-in phase stamps of the tensor-core decode kernel (%globaltimer, ns), [CTA][8]; null: none
};

constexpr int kHd = 192, kVd = 128, kM = 16;
constexpr int kKRow = kHd * 2 + 16, kVRow = kVd * 2 + 16;      // bytes of a staged row: odd in 16-byte words, so ldmatrix rows miss one another's banks
constexpr int kListWarps = 4, kListKeys = 16, kListStages = 2;
constexpr int kListStage = kListKeys * (kKRow + kVRow);
constexpr int kPartRow = kVd + 4;                                // fp32
constexpr int kListSmem = kListWarps * kListStages * kListStage;
static_assert(kListWarps * (kM * kPartRow + 2 * kM) * 4 <= kListSmem, "the merge reuses the rings");
constexpr int kWinWarps = 4, kWinKeys = 32, kWinStages = 3;
constexpr int kWinStage = kWinKeys * (kKRow + kVRow);
constexpr int kWinSmem = kWinStages * kWinStage;

// 16-byte asynchronous copy global -> shared; `valid` false writes zeros (nothing is read)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mma16816(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t r[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t r[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ float wmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float rbf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// What a warp carries over the keys: fragment rows `lane / 4` ("lo") and `lane / 4 + 8` ("hi") of its sixteen.
struct Walk {
  uint32_t q[kHd / 16][4];
  float o[kVd / 8][4];
  float m[2], l[2];                                    // l: this thread's share of the sum

  // q_lo / q_hi: the rows' queries, null: a dead row
  __device__ __forceinline__ void open(const __nv_bfloat16* q_lo, const __nv_bfloat16* q_hi, int qc) {
#pragma unroll
    for (int ks = 0; ks < kHd / 16; ++ks) {
      q[ks][0] = q_lo ? *reinterpret_cast<const uint32_t*>(q_lo + ks * 16 + qc) : 0u;
      q[ks][1] = q_hi ? *reinterpret_cast<const uint32_t*>(q_hi + ks * 16 + qc) : 0u;
      q[ks][2] = q_lo ? *reinterpret_cast<const uint32_t*>(q_lo + ks * 16 + qc + 8) : 0u;
      q[ks][3] = q_hi ? *reinterpret_cast<const uint32_t*>(q_hi + ks * 16 + qc + 8) : 0u;
    }
#pragma unroll
    for (int t = 0; t < kVd / 8; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) o[t][j] = 0.f;
    m[0] = m[1] = -FLT_MAX;
    l[0] = l[1] = 0.f;
  }

  // One tile of KEYS staged keys; seen(hi, key of the tile) says whether a row sees a key.  ONE: the walk has one token row (queries of the
  // others are null), and value rows that it does not see (kept(key)) are zero whatever memory holds.
  template <int KEYS, bool ONE = false, typename Seen, typename Kept>
  __device__ __forceinline__ void tile(uint32_t sk, uint32_t sv, int lane, float scale, Seen&& seen, Kept&& kept) {
    float s[KEYS / 8][4];
#pragma unroll
    for (int t = 0; t < KEYS / 8; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[t][j] = 0.f;
    const uint32_t ka = sk + ((lane & 7) + ((lane >> 4) << 3)) * kKRow + ((lane >> 3) & 1) * 16;
#pragma unroll
    for (int ks = 0; ks < kHd / 16; ++ks)
#pragma unroll
      for (int t = 0; t < KEYS / 16; ++t) {
        uint32_t b[4];
        ldmatrix_x4(b, ka + t * 16 * kKRow + ks * 32);
        mma16816(s[2 * t], q[ks], b[0], b[1]);
        mma16816(s[2 * t + 1], q[ks], b[2], b[3]);
      }
    const int qc = (lane & 3) * 2;
    float corr[2];
    uint32_t p[KEYS / 8][2];
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      float mx = -FLT_MAX;
#pragma unroll
      for (int t = 0; t < KEYS / 8; ++t)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float& v = s[t][2 * hi + j];
          v = seen(hi, t * 8 + qc + j) ? v * scale : -FLT_MAX;
          mx = fmaxf(mx, v);
        }
      const float mn = fmaxf(m[hi], quad_max(mx));
      corr[hi] = __expf(m[hi] - mn);
      m[hi] = mn;
      float sum = 0.f;
#pragma unroll
      for (int t = 0; t < KEYS / 8; ++t) {
        const float p0 = seen(hi, t * 8 + qc) ? rbf16(__expf(s[t][2 * hi] - mn)) : 0.f;
        const float p1 = seen(hi, t * 8 + qc + 1) ? rbf16(__expf(s[t][2 * hi + 1] - mn)) : 0.f;
        sum += p0 + p1;
        p[t][hi] = bf16_pair(p0, p1);
      }
      l[hi] = l[hi] * corr[hi] + sum;
    }
    if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
      for (int t = 0; t < kVd / 8; ++t) { o[t][0] *= corr[0]; o[t][1] *= corr[0]; o[t][2] *= corr[1]; o[t][3] *= corr[1]; }
    }
    const uint32_t va = sv + ((lane & 7) + ((lane >> 3) & 1) * 8) * kVRow + (lane >> 4) * 16;
#pragma unroll
    for (int t = 0; t < KEYS / 16; ++t) {
      const uint32_t pa[4] = {p[2 * t][0], p[2 * t][1], p[2 * t + 1][0], p[2 * t + 1][1]};
      uint32_t keep[2] = {0xffffffffu, 0xffffffffu};                // of this thread's keys qc, qc + 1 and qc + 8, qc + 9
      if (ONE)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int key = t * 16 + h * 8 + qc;
          keep[h] = (kept(key) ? 0xffffu : 0u) | (kept(key + 1) ? 0xffff0000u : 0u);
        }
#pragma unroll
      for (int c = 0; c < kVd / 16; ++c) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, va + t * 16 * kVRow + c * 32);
        if (ONE)
#pragma unroll
          for (int i = 0; i < 4; ++i) b[i] &= keep[i & 1];
        mma16816(o[2 * c], pa, b[0], b[1]);
        mma16816(o[2 * c + 1], pa, b[2], b[3]);
      }
    }
  }
};

// factor of a row's output: the sink column (no value) joins the sum, then normalisation
__device__ __forceinline__ float row_factor(float m, float l, const __nv_bfloat16* sink, int head) {
  float corr = 1.f;
  if (sink) {
    const float sv = __bfloat162float(sink[head]);
    const float mn = fmaxf(m, sv);
    corr = __expf(m - mn);
    l = l * corr + __expf(sv - mn);
  }
  return l > 0.f ? corr / l : 0.f;
}

// ------------------------------------------------------------------------------------ selection list or dense prefix
__global__ void __launch_bounds__(kListWarps * 32, 2) attn_list_kernel(const AttnArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  griddep_wait();
  griddep_launch();
  const int g = blockIdx.x, r = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hpg = a.heads / a.kv_heads, h0 = g * hpg;               // live query heads (<= 16)
  const int pos = *a.pos0 + r;
  const bool use_sel = pos + 1 > a.top_k;
  const int count = use_sel ? a.top_k : pos + 1, tiles = (count + kListKeys - 1) / kListKeys;
  const int* sel = use_sel ? a.sel + (size_t)r * a.top_k : nullptr;
  const uint32_t ring = smem_u32(smem) + warp * kListStages * kListStage;
  const uint8_t* kc = reinterpret_cast<const uint8_t*>(a.k_cache + (size_t)g * kHd) + (lane & 7) * 16;
  const uint8_t* vc = reinterpret_cast<const uint8_t*>(a.v_cache + (size_t)g * kVd) + (lane & 7) * 16;
  const size_t k_pitch = (size_t)a.kv_heads * kHd * 2, v_pitch = (size_t)a.kv_heads * kVd * 2;

  auto ids_of = [&](int t) {                                        // lane i < 16: key i of the tile (-1: none)
    const int j = t * kListKeys + lane;
    return lane < kListKeys && t < tiles && j < count ? (sel ? sel[j] : j) : -1;
  };
  // eight lanes copy one key, 128 bytes at a time
  auto request = [&](int stage, int ids) {
    const uint32_t sk = ring + stage * kListStage + (lane & 7) * 16, sv = sk + kListKeys * kKRow;
#pragma unroll
    for (int i = 0; i < kListKeys / 4; ++i) {
      const int key = i * 4 + (lane >> 3), id = __shfl_sync(0xffffffffu, ids, key);
      const bool valid = id >= 0;
      const size_t slot = !valid ? 0 : a.ring > 0 ? (size_t)(id % a.ring) : (size_t)id;
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async16(sk + key * kKRow + c * 128, kc + slot * k_pitch + c * 128, valid);
#pragma unroll
      for (int c = 0; c < 2; ++c) cp_async16(sv + key * kVRow + c * 128, vc + slot * v_pitch + c * 128, valid);
    }
  };
  int ids = ids_of(warp);
  request(0, ids);
  cp_async_commit();
  ids = ids_of(warp + kListWarps);
  Walk w;
  {
    const int qr = lane >> 2;
    const __nv_bfloat16* q = a.q + ((size_t)r * a.heads + h0) * kHd;
    w.open(qr < hpg ? q + qr * kHd : nullptr, qr + 8 < hpg ? q + (qr + 8) * kHd : nullptr, (lane & 3) * 2);
  }
  int stage = 0;
#pragma unroll 1
  for (int t = warp; t < tiles; t += kListWarps) {
    if (t + kListWarps < tiles) request(stage ^ 1, ids);
    cp_async_commit();
    ids = ids_of(t + 2 * kListWarps);
    cp_async_wait<1>();
    __syncwarp();
    const uint32_t sk = ring + stage * kListStage;
    const int live = count - t * kListKeys;
    w.tile<kListKeys>(sk, sk + kListKeys * kKRow, lane, a.scale, [&](int, int key) { return key < live; }, [](int) { return true; });
    __syncwarp();                                                   // every lane has read the stage before it is filled anew
    stage ^= 1;
  }
  cp_async_wait<0>();
  __syncthreads();
  // merge: the warps' results side by side in shared memory, then a warp per head
  float* part = reinterpret_cast<float*>(smem);                     // [warp][16][kPartRow]
  float* ml = part + kListWarps * kM * kPartRow;                    // [warp][16][2]
  {
    const int qr = lane >> 2, qc = (lane & 3) * 2;
    const float l_lo = quad_sum(w.l[0]), l_hi = quad_sum(w.l[1]);
    float* o = part + (warp * kM + qr) * kPartRow + qc;
#pragma unroll
    for (int t = 0; t < kVd / 8; ++t) {
      *reinterpret_cast<float2*>(o + t * 8) = make_float2(w.o[t][0], w.o[t][1]);
      *reinterpret_cast<float2*>(o + 8 * kPartRow + t * 8) = make_float2(w.o[t][2], w.o[t][3]);
    }
    if ((lane & 3) == 0) {
      ml[(warp * kM + qr) * 2] = w.m[0];
      ml[(warp * kM + qr) * 2 + 1] = l_lo;
      ml[(warp * kM + qr + 8) * 2] = w.m[1];
      ml[(warp * kM + qr + 8) * 2 + 1] = l_hi;
    }
  }
  __syncthreads();
  const size_t ldo = (size_t)a.heads * kVd;
#pragma unroll 1
  for (int h = warp; h < hpg; h += kListWarps) {
    float m = -FLT_MAX, l = 0.f;
#pragma unroll
    for (int i = 0; i < kListWarps; ++i) m = fmaxf(m, ml[(i * kM + h) * 2]);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kListWarps; ++i) {
      const float f = __expf(ml[(i * kM + h) * 2] - m);
      l = fmaf(ml[(i * kM + h) * 2 + 1], f, l);
      const float4 p = *reinterpret_cast<const float4*>(part + (i * kM + h) * kPartRow + lane * 4);
      v = make_float4(fmaf(p.x, f, v.x), fmaf(p.y, f, v.y), fmaf(p.z, f, v.z), fmaf(p.w, f, v.w));
    }
    const float f = row_factor(m, l, a.sink, h0 + h);
    v = make_float4(rbf16(v.x * f), rbf16(v.y * f), rbf16(v.z * f), rbf16(v.w * f));
    const size_t base = (size_t)r * ldo + (size_t)(h0 + h) * kVd + lane * 4;
    if (a.o_bf16) *reinterpret_cast<uint2*>(a.o_bf16 + base) = make_uint2(bf16_pair(v.x, v.y), bf16_pair(v.z, v.w));
    if (a.o8) {
      const float sc = pow2_scale(wmax(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)))));
      const __nv_fp8_e4m3 c[4] = {__nv_fp8_e4m3(v.x / sc), __nv_fp8_e4m3(v.y / sc), __nv_fp8_e4m3(v.z / sc), __nv_fp8_e4m3(v.w / sc)};
      uint32_t word = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) word |= (uint32_t)c[i].__x << (8 * i);
      *reinterpret_cast<uint32_t*>(a.o8 + base) = word;
      if (lane == 0) a.o_scale[(size_t)r * (ldo / 128) + h0 + h] = sc;
    }
  }
}

// ------------------------------------------------------------------------------------ sliding window
__global__ void __launch_bounds__(kWinWarps * 32, 2) attn_window_kernel(const AttnArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  griddep_wait();
  griddep_launch();
  const int g = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hpg = a.heads / a.kv_heads, h0 = g * hpg, rpw = kM / hpg;     // rows per warp
  const int r0 = blockIdx.y * kWinWarps * rpw, pos0 = *a.pos0;
  const int r_last = min(r0 + kWinWarps * rpw, a.rows) - 1;
  const int key0 = max(0, pos0 + r0 - a.window + 1), key_end = pos0 + r_last + 1;       // keys of the CTA's rows
  const int tiles = (key_end - key0 + kWinKeys - 1) / kWinKeys;
  const uint32_t base = smem_u32(smem);
  const int chunk = (threadIdx.x & 7) * 16;                                             // eight threads copy one key
  const uint8_t* kc = reinterpret_cast<const uint8_t*>(a.k_cache + (size_t)g * kHd) + chunk;
  const uint8_t* vc = reinterpret_cast<const uint8_t*>(a.v_cache + (size_t)g * kVd) + chunk;
  const size_t k_pitch = (size_t)a.kv_heads * kHd * 2, v_pitch = (size_t)a.kv_heads * kVd * 2;
  auto request = [&](int t) {
    const uint32_t st = base + (t % kWinStages) * kWinStage + chunk;
#pragma unroll
    for (int key = threadIdx.x >> 3; key < kWinKeys; key += kWinWarps * 4) {
      const int id = key0 + t * kWinKeys + key;
      const bool valid = id < key_end;
      const size_t slot = !valid ? 0 : a.ring > 0 ? (size_t)(id % a.ring) : (size_t)id;
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async16(st + key * kKRow + c * 128, kc + slot * k_pitch + c * 128, valid);
#pragma unroll
      for (int c = 0; c < 2; ++c) cp_async16(st + kWinKeys * kKRow + key * kVRow + c * 128, vc + slot * v_pitch + c * 128, valid);
    }
  };
  auto open_ring = [&]() {
#pragma unroll
    for (int t = 0; t < kWinStages - 1; ++t) {
      if (t < tiles) request(t);
      cp_async_commit();
    }
  };
  // fragment row -> (token row, head); rows beyond the chunk see no key
  int row[2], head[2], low[2], high[2];
#pragma unroll
  for (int hi = 0; hi < 2; ++hi) {
    const int at = (lane >> 2) + 8 * hi, slot = at / hpg;
    row[hi] = slot < rpw ? min(r0 + warp * rpw + slot, a.rows) : a.rows;
    head[hi] = h0 + at - slot * hpg;
    const int pos = pos0 + row[hi];
    low[hi] = row[hi] < a.rows ? max(0, pos - a.window + 1) : 0;
    high[hi] = row[hi] < a.rows ? pos : -1;
  }
  Walk w;
  auto query = [&](int hi) { return a.q + ((size_t)row[hi] * a.heads + head[hi]) * kHd; };
  // keys that any token row of the warp sees; `one`: only its row at `slot` is worked on
  auto walk = [&](auto one, int slot) {
    constexpr bool ONE = decltype(one)::value;
    const int r_lo = r0 + warp * rpw + (ONE ? slot : 0), r_hi = ONE ? r_lo + 1 : min(r_lo + rpw, a.rows);
    const int w_low = pos0 + r_lo - a.window + 1, w_high = pos0 + r_hi - 1;
    const bool on[2] = {row[0] < a.rows && (!ONE || row[0] == r_lo), row[1] < a.rows && (!ONE || row[1] == r_lo)};
    w.open(on[0] ? query(0) : nullptr, on[1] ? query(1) : nullptr, (lane & 3) * 2);
#pragma unroll 1
    for (int t = 0; t < tiles; ++t) {
      cp_async_wait<kWinStages - 2>();
      __syncthreads();                                                // tile t has landed; everybody is done with tile t - 1
      if (t + kWinStages - 1 < tiles) request(t + kWinStages - 1);
      cp_async_commit();
      const int k0 = key0 + t * kWinKeys;
      if (k0 > w_high || k0 + kWinKeys <= w_low || r_lo >= a.rows) continue;
      const uint32_t sk = base + (t % kWinStages) * kWinStage;
      w.tile<kWinKeys, ONE>(sk, sk + kWinKeys * kKRow, lane, a.scale, [&](int hi, int i) { return (!ONE || on[hi]) && k0 + i >= low[hi] && k0 + i <= high[hi]; },
                            [&](int i) { return k0 + i >= w_low && k0 + i <= w_high; });
    }
    cp_async_wait<0>();
  };
  const size_t ldo = (size_t)a.heads * kVd;
  auto store = [&](int slot) {                                        // the rows of one slot, -1: all
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const float l = quad_sum(w.l[hi]);
      const bool live = row[hi] < a.rows && (slot < 0 || row[hi] == r0 + warp * rpw + slot);
      const float f = live ? row_factor(w.m[hi], l, a.sink, head[hi]) : 0.f;
      float am = 0.f;
#pragma unroll
      for (int t = 0; t < kVd / 8; ++t)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float& v = w.o[t][2 * hi + j];
          v = rbf16(v * f);
          am = fmaxf(am, fabsf(v));
        }
      const float sc = pow2_scale(quad_max(am));
      if (!live) continue;
      const size_t at = (size_t)row[hi] * ldo + (size_t)head[hi] * kVd + (lane & 3) * 2;
      if (a.o_bf16)
#pragma unroll
        for (int t = 0; t < kVd / 8; ++t) *reinterpret_cast<uint32_t*>(a.o_bf16 + at + t * 8) = bf16_pair(w.o[t][2 * hi], w.o[t][2 * hi + 1]);
      if (a.o8) {
#pragma unroll
        for (int t = 0; t < kVd / 8; ++t) {
          const __nv_fp8_e4m3 c0(w.o[t][2 * hi] / sc), c1(w.o[t][2 * hi + 1] / sc);
          *reinterpret_cast<uint16_t*>(a.o8 + at + t * 8) = (uint16_t)(c0.__x | (uint32_t)c1.__x << 8);
        }
        if ((lane & 3) == 0) a.o_scale[(size_t)row[hi] * (ldo / 128) + head[hi]] = sc;
      }
    }
  };
  open_ring();
  walk(std::false_type{}, 0);
  // A probability of zero does not hide an infinity or NaN of a value row that only other rows of the CTA see; what it
  // leaves in an output stays non-finite to the end.  Then every token row is walked again by itself, unseen values zeroed.
  float bad = 0.f;                                                    // zero times a finite value is zero
#pragma unroll
  for (int t = 0; t < kVd / 8; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) bad = fmaf(w.o[t][j], 0.f, bad);
  if (!__syncthreads_or(bad != 0.f)) {
    store(-1);
    return;
  }
#pragma unroll 1
  for (int slot = 0; slot < rpw; ++slot) {
    __syncthreads();                                                  // the stages are free
    open_ring();
    walk(std::true_type{}, slot);
    store(slot);
  }
}

}  // namespace

extern "C" int nrt_attn_group_args_size() { return (int)sizeof(AttnArgs); }

// Grouped-head row attention; modes 0 (sliding window) and 1 (dense prefix / selection list), head_dim 192,
// v_dim 128, at most 16 query heads per KV head.  Returns -3 for other geometries (use nrt_attn_rows).
extern "C" int nrt_attn_group(const void* args, void* stream, int pdl) {
  AttnArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.head_dim != kHd || a.v_dim != kVd || a.kv_heads < 1 || a.heads % a.kv_heads || a.heads / a.kv_heads > kM) return -3;
  if (a.mode != 0 && a.mode != 1) return -3;
  if (a.rows > 65535) return -3;
  if (const int rc = a.mode == 1 ? allow_shared(attn_list_kernel, kListSmem) : allow_shared(attn_window_kernel, kWinSmem)) return rc;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (a.mode == 1) return launch_pdl(attn_list_kernel, dim3(a.kv_heads, a.rows), dim3(kListWarps * 32), kListSmem, s, pdl != 0, a);
  const int rows = kWinWarps * (kM / (a.heads / a.kv_heads));
  return launch_pdl(attn_window_kernel, dim3(a.kv_heads, (a.rows + rows - 1) / rows), dim3(kWinWarps * 32), kWinSmem, s, pdl != 0, a);
}
