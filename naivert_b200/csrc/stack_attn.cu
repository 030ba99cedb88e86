// Grouped-query attention of layer stacks around the chunk kernels of latent_attn.cu: preparation of queries, keys and values
// (norm per head, rotary positions, cache rows), the feature-major copy of the values, and the one-token step.
#include "stack.cuh"
#include "launch.hpp"

#include <string.h>

using namespace nrt;

namespace {

constexpr int kMaxHead = 512;                 // head width the kernels hold in shared memory

// One head of a token, by one warp: x[0, n) -> normed (w != null) and rotated by the angles in (cs, sn), times `scale`, in `out`
// (shared, n values).  All reads of `src` happen before the first write of `out`.
__device__ __forceinline__ void head_vector(const float* src, int n, const __nv_bfloat16* w, float eps, int half, const float* cs, const float* sn,
                                            float scale, float* out, int lane) {
  float ss = 0.f;
  for (int c = lane; c < n; c += 32) {
    const float v = __ldcg(src + c);
    out[c] = v;
    ss = fmaf(v, v, ss);
  }
  if (w) {
    const float r = 1.0f / sqrtf(lane_sum(ss) / (float)n + eps);
    for (int c = lane; c < n; c += 32) out[c] = out[c] * r * bf(w + c);
  }
  __syncwarp();
  for (int i = lane; i < half; i += 32) {
    const float u = out[i], v = out[i + half], c = cs[i], s = sn[i];
    out[i] = u * c - v * s;
    out[i + half] = v * c + u * s;
  }
  __syncwarp();
  if (scale != 1.f)
    for (int c = lane; c < n; c += 32) out[c] *= scale;
  __syncwarp();
}
__device__ __forceinline__ void angles(const GroupPrepArgs& p, int pos, float* cs, float* sn) {
  for (int i = threadIdx.x; i < p.rot_dims / 2; i += blockDim.x) sincosf((float)pos * p.freq[i], sn + i, cs + i);
}

// ------------------------------------------------------------------------------------ chunk path: preparation
// One CTA per row; a warp takes one head at a time: queries, then keys, then values.
__global__ void __launch_bounds__(256) group_prep_kernel(const GroupPrepArgs p) {
  __shared__ float buf[8][kMaxHead], cs[kMaxHead / 2], sn[kMaxHead / 2];
  griddep_wait();
  griddep_launch();
  const int r = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = p.rot_dims / 2;
  const int pos = *p.pos0 + r;
  if (pos < 0 || pos >= p.capacity) return;
  angles(p, pos, cs, sn);
  __syncthreads();
  const float* row = p.proj + r * p.ld;
  for (int u = warp; u < p.heads + 2 * p.kv_heads; u += 8) {
    if (u < p.heads + p.kv_heads) {
      const bool is_q = u < p.heads;
      const int h = is_q ? u : u - p.heads;
      head_vector(row + (is_q ? p.q_off : p.k_off) + h * p.dim, p.dim, is_q ? p.q_norm : p.k_norm, p.eps, half, cs, sn, is_q ? p.scale : 1.f, buf[warp], lane);
      void* dst = is_q ? p.q : p.k_cache;
      const long long at = is_q ? ((long long)r * p.heads + h) * p.dp : ((long long)pos * p.kv_heads + h) * p.dp;
      for (int c = lane; c < p.dp; c += 32) store_act(dst, at + c, c < p.dim ? buf[warp][c] : 0.f, p.f32);
      __syncwarp();
    } else {
      const int h = u - p.heads - p.kv_heads;
      for (int c = lane; c < p.vdim; c += 32) store_act(p.v_cache, ((long long)pos * p.kv_heads + h) * p.vp + c, row[p.v_off + h * p.vdim + c], p.f32);
    }
  }
}

// dst[c][r] = src[r][c], 64 x 64 tiles, two values per access; rows beyond the last become zeros up to the tile's end
__global__ void __launch_bounds__(256) transpose_kernel(const TransposeArgs a) {
  __shared__ __nv_bfloat16 tile[64][66];
  griddep_wait();
  griddep_launch();
  const int r0 = blockIdx.x * 64, c0 = blockIdx.y * 64, tx = (threadIdx.x & 31) * 2, ty = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 64; i += 8) {
    const int r = r0 + ty + i;
    uint32_t v = 0u;
    if (r < a.rows && c0 + tx < a.cols) v = *reinterpret_cast<const uint32_t*>(a.src + (long long)r * a.cols + c0 + tx);
    *reinterpret_cast<uint32_t*>(&tile[ty + i][tx]) = v;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 64; i += 8) {
    const int c = c0 + ty + i;
    if (c >= a.cols || r0 + tx >= a.dst_ld) continue;
    __nv_bfloat162 v;
    v.x = tile[tx][ty + i];
    v.y = tile[tx + 1][ty + i];
    *reinterpret_cast<__nv_bfloat162*>(a.dst + (long long)c * a.dst_ld + r0 + tx) = v;
  }
}

// ------------------------------------------------------------------------------------ one token
// The splits of the context of one key head are a cluster; their partial results meet through distributed shared memory.  Every CTA
// whose keys end at the token itself prepares and stores the token's key and value (equal values where there are several).
//
// Plain form (32-bit caches, wide heads): grid (splits, key heads, groups of eight query heads); eight lanes share a key, the query
// heads of the CTA are scored together; then threads own value columns.
constexpr int kHB = 8, kTile = 64, kDecThreads = 256;

__host__ __device__ inline int group_smem_floats(int dp, int vp) { return kHB * dp + kMaxHead + kTile * kHB + 3 * kHB + kHB * vp; }

template <bool F32, int VC>                    // VC value columns per thread
__global__ void __launch_bounds__(kDecThreads) group_decode_kernel(const GroupDecodeArgs a) {
  extern __shared__ __align__(16) float sh[];
  const GroupPrepArgs& p = a.p;
  float* sq = sh;                              // [8][dp]
  float* cs = sq + kHB * p.dp;
  float* sn = cs + kMaxHead / 2;
  float* sp = sn + kMaxHead / 2;               // [64][8]
  float* sm = sp + kTile * kHB;
  float* sl = sm + kHB;
  float* scorr = sl + kHB;
  float* so = scorr + kHB;                     // [8][vp]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = lane & 7;
  const int split = blockIdx.x, hk = blockIdx.y, group = p.heads / p.kv_heads, h0 = blockIdx.z * kHB, nh = min(kHB, group - h0);
  const int half = p.rot_dims / 2;
  griddep_wait();
  griddep_launch();
  const int pos = *reinterpret_cast<const volatile int*>(p.pos0);
  const int start = a.window > 0 ? pos / a.window * a.window : 0, n = pos + 1 - start;
  const int per = ((n + a.splits - 1) / a.splits + kTile - 1) / kTile * kTile;
  const int j_lo = min(n, split * per), j_hi = min(n, j_lo + per);
  const bool inside = pos >= 0 && pos < p.capacity;
  angles(p, pos, cs, sn);
  for (int i = tid; i < kHB * p.dp; i += kDecThreads) sq[i] = 0.f;
  for (int i = tid; i < kHB * p.vp; i += kDecThreads) so[i] = 0.f;
  if (tid < kHB) { sm[tid] = -FLT_MAX; sl[tid] = 0.f; }
  __syncthreads();
  if (inside && j_lo < j_hi) {
    if (j_hi == n) {
      // the token's own key and value (sp is free until the first tile)
      if (warp == 0) {
        head_vector(p.proj + p.k_off + hk * p.dim, p.dim, p.k_norm, p.eps, half, cs, sn, 1.f, sp, lane);
        for (int c = lane; c < p.dim; c += 32) store_act(p.k_cache, ((long long)pos * p.kv_heads + hk) * p.dp + c, sp[c], F32);
      } else if (warp == 1) {
        for (int c = lane; c < p.vdim; c += 32)
          store_act(p.v_cache, ((long long)pos * p.kv_heads + hk) * p.vp + c, __ldcg(p.proj + p.v_off + hk * p.vdim + c), F32);
      }
    }
    for (int h = warp; h < nh; h += kDecThreads / 32)
      head_vector(p.proj + p.q_off + (hk * group + h0 + h) * p.dim, p.dim, p.q_norm, p.eps, half, cs, sn, p.scale, sq + h * p.dp, lane);
    __syncthreads();
    const int pieces = p.dp / 8;
    int vc = 32;
    while (vc < p.vdim && vc < kDecThreads) vc *= 2;
    const int subs = kDecThreads / vc, sub = tid / vc, c0 = tid & (vc - 1);
    float acc[kHB][VC];
#pragma unroll
    for (int h = 0; h < kHB; ++h)
#pragma unroll
      for (int i = 0; i < VC; ++i) acc[h][i] = 0.f;
    float m = -FLT_MAX, sum = 0.f;                                       // of head `warp`
    for (int j0 = j_lo; j0 < j_hi; j0 += kTile) {
      const int live = min(kTile, j_hi - j0);
#pragma unroll
      for (int t0 = 0; t0 < kTile; t0 += kDecThreads / 8) {
        const int t = t0 + tid / 8;
        float d[kHB];
#pragma unroll
        for (int h = 0; h < kHB; ++h) d[h] = 0.f;
        if (t < live) {
          const long long at = ((long long)(start + j0 + t) * p.kv_heads + hk) * p.dp;
#pragma unroll 2
          for (int i = l; i < pieces; i += 8) {
            float4 x, y;
            if (F32) {
              const float4* k = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.k_cache) + at + i * 8);
              x = __ldcg(k);
              y = __ldcg(k + 1);
            } else {
              const uint4 k = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.k_cache) + at + i * 8));
              x = make_float4(bf16_lo(k.x), bf16_hi(k.x), bf16_lo(k.y), bf16_hi(k.y));
              y = make_float4(bf16_lo(k.z), bf16_hi(k.z), bf16_lo(k.w), bf16_hi(k.w));
            }
#pragma unroll
            for (int h = 0; h < kHB; ++h) {
              const float4 q0 = *reinterpret_cast<const float4*>(sq + h * p.dp + i * 8), q1 = *reinterpret_cast<const float4*>(sq + h * p.dp + i * 8 + 4);
              d[h] = fmaf(x.x, q0.x, fmaf(x.y, q0.y, fmaf(x.z, q0.z, fmaf(x.w, q0.w, d[h]))));
              d[h] = fmaf(y.x, q1.x, fmaf(y.y, q1.y, fmaf(y.z, q1.z, fmaf(y.w, q1.w, d[h]))));
            }
          }
        }
        float mine = 0.f;
#pragma unroll
        for (int h = 0; h < kHB; ++h) {
          float v = d[h];
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          v += __shfl_xor_sync(0xffffffffu, v, 4);
          if (h == l) mine = v;
        }
        sp[t * kHB + l] = mine;
      }
      __syncthreads();
      {                                                                  // softmax of head `warp`
        const float s0 = lane < live ? sp[lane * kHB + warp] : -FLT_MAX, s1 = lane + 32 < live ? sp[(lane + 32) * kHB + warp] : -FLT_MAX;
        float mt = fmaxf(s0, s1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
        const float mn = fmaxf(m, mt), corr = expf(m - mn);
        const float p0 = lane < live ? expf(s0 - mn) : 0.f, p1 = lane + 32 < live ? expf(s1 - mn) : 0.f;
        sum = fmaf(sum, corr, lane_sum(p0 + p1));
        m = mn;
        sp[lane * kHB + warp] = p0;
        sp[(lane + 32) * kHB + warp] = p1;
        if (lane == 0) scorr[warp] = corr;
      }
      __syncthreads();
#pragma unroll
      for (int h = 0; h < kHB; ++h)
#pragma unroll
        for (int i = 0; i < VC; ++i) acc[h][i] *= scorr[h];
#pragma unroll 4
      for (int t = sub; t < live; t += subs) {
        const float4 pa = *reinterpret_cast<const float4*>(sp + t * kHB), pb = *reinterpret_cast<const float4*>(sp + t * kHB + 4);
        const long long at = ((long long)(start + j0 + t) * p.kv_heads + hk) * p.vp;
#pragma unroll
        for (int i = 0; i < VC; ++i) {
          const int c = c0 + i * kDecThreads;
          if (c < p.vdim) {
            const float v = F32 ? __ldcg(reinterpret_cast<const float*>(p.v_cache) + at + c)
                                : __bfloat162float(__ldcg(reinterpret_cast<const __nv_bfloat16*>(p.v_cache) + at + c));
            acc[0][i] = fmaf(pa.x, v, acc[0][i]);
            acc[1][i] = fmaf(pa.y, v, acc[1][i]);
            acc[2][i] = fmaf(pa.z, v, acc[2][i]);
            acc[3][i] = fmaf(pa.w, v, acc[3][i]);
            acc[4][i] = fmaf(pb.x, v, acc[4][i]);
            acc[5][i] = fmaf(pb.y, v, acc[5][i]);
            acc[6][i] = fmaf(pb.z, v, acc[6][i]);
            acc[7][i] = fmaf(pb.w, v, acc[7][i]);
          }
        }
      }
      __syncthreads();                                                   // sp is rewritten
    }
    if (lane == 0) { sm[warp] = m; sl[warp] = sum; }
    // key subsets join in a fixed order
    for (int s = 0; s < subs; ++s) {
      if (sub == s) {
#pragma unroll
        for (int h = 0; h < kHB; ++h)
#pragma unroll
          for (int i = 0; i < VC; ++i)
            if (c0 + i * kDecThreads < p.vdim) so[h * p.vp + c0 + i * kDecThreads] += acc[h][i];
      }
      __syncthreads();
    }
  }
  cluster_sync_all();
  // every CTA of the cluster finishes a share of the heads' columns
  for (int i = split * kDecThreads + tid; i < nh * p.vdim; i += a.splits * kDecThreads) {
    const int h = i / p.vdim, c = i - h * p.vdim;
    float m = -FLT_MAX, o = 0.f, sum = 0.f;
    for (int s = 0; s < a.splits; ++s) m = fmaxf(m, ld_cluster_f32(sm + h, s));
    for (int s = 0; s < a.splits; ++s) {
      const float w = expf(ld_cluster_f32(sm + h, s) - m);
      sum = fmaf(w, ld_cluster_f32(sl + h, s), sum);
      o = fmaf(w, ld_cluster_f32(so + h * p.vp + c, s), o);
    }
    a.out[(long long)(hk * group + h0 + h) * p.vp + c] = o / sum;
  }
  cluster_sync_all();                                                    // nobody leaves while its shared memory is read
}

// Tensor-core form: grid (splits, key heads, tiles of 16 query heads).  The query heads of a key head are the M side of bf16 m16n8k16
// MMAs.  A warp walks every so-many-th tile of 16 keys of the split through a ring of its own and keeps scores, probabilities (a score
// fragment is the A fragment of P V as it stands) and outputs in registers: no barrier inside the walk, and the eight rings together keep the
// 140 KB in flight that one SM's share of the memory's rate needs.  The warps' results are merged once, then the cluster's.  The first
// tiles are requested before the wait for the predecessor (older rows do not depend on it; the token's own row is put into its tile by
// hand).  tcgen05 is not used: the kernel streams the cache once, and most of its M = 128 rows would idle.
// 12,290 keys, 8 key heads of 4 x 128: 44 us inside a step from launch to end (the wait for the predecessor included), 59 us with tiles of 64
// keys that all warps worked on between four barriers; alone 39.7 and 53.9 us.  Groups of more than 16 heads take a CTA per 16, each of
// which reads the split's rows (the second from L2): 32 heads of one key head 41.6 us alone, 83.9 us as one tile of 32 rows in that form.
constexpr int kTcHead = 256, kWalkKeys = 16, kWalkM = 16, kWalkSmem = 225 * 1024;
__host__ __device__ inline int tc_pitch(int n) { return (n + 15) / 16 * 16 + 8; }              // bf16 elements; rows fall into distinct banks
struct WalkShape { int warps, stages; };               // walking warps of a CTA, ring stages of each
__host__ __device__ inline int walk_ring(int dp, int vp, WalkShape w) { return 2 * w.warps * w.stages * kWalkKeys * (tc_pitch(dp) + tc_pitch(vp)); }
__host__ __device__ inline int walk_smem(int dp, int vp, WalkShape w) {
  return walk_ring(dp, vp, w) + 2 * kWalkM * tc_pitch(dp) + 4 * (2 * kWalkM * (w.warps + 1) + 8 * kTcHead + kTcHead) + 2 * (dp + vp);
}

// DIM: most columns of keys and values (registers of the outputs).  Up to 128 the kernel keeps to half of an SM's registers: its rings (224 KB of
// shared memory at 128 x 128) leave room for a state step's few KB beside them, but not for the launch of a product.
template <int DIM>
__global__ void __launch_bounds__(kDecThreads, DIM <= 128 ? 2 : 1) group_decode_tc_kernel(const GroupDecodeArgs a, const WalkShape ws) {
  extern __shared__ __align__(16) uint8_t raw[];
  const GroupPrepArgs& p = a.p;
  const int kp = tc_pitch(p.dp), vpitch = tc_pitch(p.vp), rp = (p.dp + 15) / 16 * 16, stage_elems = kWalkKeys * (kp + vpitch);
  __nv_bfloat16* ring = reinterpret_cast<__nv_bfloat16*>(raw);           // [warps][stages][16 keys, 16 values]
  __nv_bfloat16* sq = ring + ws.warps * ws.stages * stage_elems;         // [16][kp]
  float* sm = reinterpret_cast<float*>(sq + kWalkM * kp);                // [16], then [warps][16]
  float* sl = sm + kWalkM * (ws.warps + 1);
  float* cs = sl + kWalkM * (ws.warps + 1);
  float* sn = cs + kTcHead / 2;
  float* buf = sn + kTcHead / 2;                                         // [8][256]
  __nv_bfloat16* new_k = reinterpret_cast<__nv_bfloat16*>(buf + 8 * kTcHead);
  __nv_bfloat16* new_v = new_k + p.dp;
  // after the walk the rings hold the warps' outputs and the CTA's
  const int part_row = p.vp + 4;
  float* part = reinterpret_cast<float*>(raw);                           // [warps][16][part_row]
  float* so = part + ws.warps * kWalkM * part_row;                       // [16][vp]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.x, hk = blockIdx.y, group = p.heads / p.kv_heads, h0 = blockIdx.z * kWalkM, nh = min(kWalkM, group - h0);
  const int half = p.rot_dims / 2;
  const int pos = *reinterpret_cast<const volatile int*>(p.pos0);
  const bool inside = pos >= 0 && pos < p.capacity;
  const int start = a.window > 0 ? pos / a.window * a.window : 0, n = inside ? pos + 1 - start : 0;
  const int per = ((n + a.splits - 1) / a.splits + kTile - 1) / kTile * kTile;
  const int j_lo = min(n, split * per), j_hi = min(n, j_lo + per);
  const bool owner = j_hi == n && j_lo < j_hi;
  const int step = ws.warps * kWalkKeys;                                 // keys from one tile of a warp to its next
  const __nv_bfloat16* kc = reinterpret_cast<const __nv_bfloat16*>(p.k_cache) + (long long)hk * p.dp;
  const __nv_bfloat16* vc = reinterpret_cast<const __nv_bfloat16*>(p.v_cache) + (long long)hk * p.vp;
  __nv_bfloat16* mine = ring + warp * ws.stages * stage_elems;
  // a lane copies one 16-byte piece of every so-many-th row; rows beyond the split become zero
  auto rows_in = [&](int j0, __nv_bfloat16* dst, int pitch, const __nv_bfloat16* src, int width) {
    int lanes = 1;
    while (lanes < width / 8) lanes *= 2;
    const int c = lane & (lanes - 1), rows = 32 / lanes;
    if (c >= width / 8) return;
    const long long row_step = (long long)p.kv_heads * width;
    // Rolled where a pass of the lanes is two rows or more: a launch inside a step fetches its instructions anew, and at short contexts it is
    // little more than that (1.5 us less).  Wider rows take sixteen passes, which have to overlap (2 x 32 heads of 256, 12,289 keys: 84 / 96 us).
#pragma unroll (DIM <= 128 ? 1 : 8)
    for (int t = lane / lanes; t < kWalkKeys; t += rows) {
      const bool in = j0 + t < j_hi && j0 + t != n - 1;                  // the token's own row is not in the cache yet
      cp16(dst + t * pitch + c * 8, in ? src + (long long)(start + j0 + t) * row_step + c * 8 : src, in);
    }
  };
  auto request = [&](int j0, int st) {         // the 16 rows from j0 on (none beyond the split: an empty group keeps the count)
    if (j0 < j_hi) {
      rows_in(j0, mine + st * stage_elems, kp, kc, p.dp);
      rows_in(j0, mine + st * stage_elems + kWalkKeys * kp, vpitch, vc, p.vp);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int j_first = j_lo + warp * kWalkKeys;
  const bool walks = warp < ws.warps;
  if (walks) {
    if (rp > p.dp)                                                       // columns between the head and a whole step stay zero
      for (int i = lane; i < ws.stages * kWalkKeys; i += 32)
        *reinterpret_cast<uint4*>(mine + i / kWalkKeys * stage_elems + i % kWalkKeys * kp + p.dp) = make_uint4(0u, 0u, 0u, 0u);
    for (int i = 0; i + 1 < ws.stages; ++i) request(j_first + i * step, i);
  }
  for (int i = tid; i < kWalkM * kp / 8; i += kDecThreads) reinterpret_cast<uint4*>(sq)[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < kWalkM * (ws.warps + 1); i += kDecThreads) { sm[i] = -FLT_MAX; sl[i] = 0.f; }
  griddep_wait();
  griddep_launch();
  if (j_lo < j_hi) {
    angles(p, pos, cs, sn);
    __syncthreads();
    for (int u = warp; u < nh + (owner ? 2 : 0); u += kDecThreads / 32) {
      float* b = buf + warp * kTcHead;
      if (u < nh) {
        head_vector(p.proj + p.q_off + (hk * group + h0 + u) * p.dim, p.dim, p.q_norm, p.eps, half, cs, sn, p.scale, b, lane);
        for (int c = lane; c < p.dim; c += 32) sq[u * kp + c] = __float2bfloat16_rn(b[c]);
      } else if (u == nh) {
        head_vector(p.proj + p.k_off + hk * p.dim, p.dim, p.k_norm, p.eps, half, cs, sn, 1.f, b, lane);
        for (int c = lane; c < p.dp; c += 32) {
          const __nv_bfloat16 x = __float2bfloat16_rn(c < p.dim ? b[c] : 0.f);
          new_k[c] = x;
          reinterpret_cast<__nv_bfloat16*>(p.k_cache)[((long long)pos * p.kv_heads + hk) * p.dp + c] = x;
        }
      } else {
        for (int c = lane; c < p.vp; c += 32) {
          const __nv_bfloat16 x = __float2bfloat16_rn(c < p.vdim ? __ldcg(p.proj + p.v_off + hk * p.vdim + c) : 0.f);
          new_v[c] = x;
          reinterpret_cast<__nv_bfloat16*>(p.v_cache)[((long long)pos * p.kv_heads + hk) * p.vp + c] = x;
        }
      }
      __syncwarp();
    }
    __syncthreads();
    const int fr = lane >> 2, fc = (lane & 3) * 2;
    float o[DIM / 8][4], m[2] = {-FLT_MAX, -FLT_MAX}, l[2] = {0.f, 0.f};    // rows fr and fr + 8 of the sixteen heads
#pragma unroll
    for (int t = 0; t < DIM / 8; ++t)
#pragma unroll
      for (int q = 0; q < 4; ++q) o[t][q] = 0.f;
    if (walks) {
      const float c2 = 1.4426950408889634f;                              // scores in powers of two
      const __nv_bfloat16* qrow = sq + (lane & 15) * kp + (lane >> 4) * 8;
      int st = 0;
#pragma unroll 1
      for (int j0 = j_first; j0 < j_hi; j0 += step, st = st + 1 == ws.stages ? 0 : st + 1) {
        request(j0 + (ws.stages - 1) * step, st == 0 ? ws.stages - 1 : st - 1);
        if (ws.stages == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
        else if (ws.stages == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        __nv_bfloat16* kt = mine + st * stage_elems;
        __nv_bfloat16* vt = kt + kWalkKeys * kp;
        if (owner && j0 < n && n - 1 < j0 + kWalkKeys) {                 // the token's own row
          if (lane < p.dp / 8) reinterpret_cast<uint4*>(kt + (n - 1 - j0) * kp)[lane] = reinterpret_cast<const uint4*>(new_k)[lane];
          if (lane < p.vp / 8) reinterpret_cast<uint4*>(vt + (n - 1 - j0) * vpitch)[lane] = reinterpret_cast<const uint4*>(new_v)[lane];
          __syncwarp();
        }
        float s[2][4] = {}, s2[2][4] = {};                               // keys 0-7 and 8-15; even and odd steps: two chains
        const __nv_bfloat16* krow = kt + ((lane & 7) + ((lane >> 4) << 3)) * kp + ((lane >> 3) & 1) * 8;
#pragma unroll
        for (int k = 0; k < DIM / 16; ++k)
          if (k * 16 < rp) {
            uint32_t q[4], b[4];
            ldsm4(q, qrow + k * 16);
            ldsm4(b, krow + k * 16);
            mma16816(k & 1 ? s2[0] : s[0], q, b[0], b[1]);
            mma16816(k & 1 ? s2[1] : s[1], q, b[2], b[3]);
          }
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i >> 2][i & 3] += s2[i >> 2][i & 3];
        const int live = j_hi - j0;
        float corr[2];
        uint32_t pf[4];
#pragma unroll
        for (int hi = 0; hi < 2; ++hi) {
          float v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = (i >> 1) * 8 + fc + (i & 1) < live ? s[i >> 1][2 * hi + (i & 1)] * c2 : -FLT_MAX;
          float mx = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
          const float mn = fmaxf(m[hi], mx);
          corr[hi] = exp2_approx(m[hi] - mn);
          m[hi] = mn;
          float e[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) e[i] = (i >> 1) * 8 + fc + (i & 1) < live ? exp2_approx(v[i] - mn) : 0.f;
          l[hi] = fmaf(l[hi], corr[hi], (e[0] + e[1]) + (e[2] + e[3]));
          pf[hi] = pack_bf16x2(e[0], e[1]);
          pf[2 + hi] = pack_bf16x2(e[2], e[3]);
        }
        if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
          for (int t = 0; t < DIM / 8; ++t) { o[t][0] *= corr[0]; o[t][1] *= corr[0]; o[t][2] *= corr[1]; o[t][3] *= corr[1]; }
        }
        const __nv_bfloat16* vrow = vt + ((lane & 7) + ((lane >> 3) & 1) * 8) * vpitch + (lane >> 4) * 8;
#pragma unroll
        for (int c = 0; c < DIM / 16; ++c)
          if (c * 16 < p.vp) {
            uint32_t b[4];
            ldsm4t(b, vrow + c * 16);
            mma16816(o[2 * c], pf, b[0], b[1]);
            mma16816(o[2 * c + 1], pf, b[2], b[3]);
          }
        __syncwarp();                                                    // every lane has read the stage before it is filled anew
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        l[hi] += __shfl_xor_sync(0xffffffffu, l[hi], 1);
        l[hi] += __shfl_xor_sync(0xffffffffu, l[hi], 2);
        if ((lane & 3) == 0) {
          sm[(warp + 1) * kWalkM + fr + 8 * hi] = m[hi];
          sl[(warp + 1) * kWalkM + fr + 8 * hi] = l[hi];
        }
      }
    }
    __syncthreads();                                                     // the rings are free
    const int fed = min(ws.warps, (j_hi - j_lo + kWalkKeys - 1) / kWalkKeys);      // warps that had a tile: short contexts have few to merge
    if (warp < fed) {
      float* d = part + (warp * kWalkM + fr) * part_row + fc;
#pragma unroll
      for (int t = 0; t < DIM / 8; ++t)
        if (t * 8 < p.vp) {
          if (fr < nh) *reinterpret_cast<float2*>(d + t * 8) = make_float2(o[t][0], o[t][1]);
          if (fr + 8 < nh) *reinterpret_cast<float2*>(d + 8 * part_row + t * 8) = make_float2(o[t][2], o[t][3]);
        }
    }
    __syncthreads();
    const int v4 = p.vp / 4;
    for (int i = tid; i < nh * v4; i += kDecThreads) {
      const int h = i / v4, c = (i - h * v4) * 4;
      float mx = -FLT_MAX, sum = 0.f;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int w = 0; w < fed; ++w) mx = fmaxf(mx, sm[(w + 1) * kWalkM + h]);
#pragma unroll 4
      for (int w = 0; w < fed; ++w) {
        const float f = exp2_approx(sm[(w + 1) * kWalkM + h] - mx);
        const float4 x = *reinterpret_cast<const float4*>(part + (w * kWalkM + h) * part_row + c);
        sum = fmaf(f, sl[(w + 1) * kWalkM + h], sum);
        v = make_float4(fmaf(f, x.x, v.x), fmaf(f, x.y, v.y), fmaf(f, x.z, v.z), fmaf(f, x.w, v.w));
      }
      *reinterpret_cast<float4*>(so + h * p.vp + c) = v;
      if (c == 0) { sm[h] = mx; sl[h] = sum; }
    }
  } else {
    for (int i = tid; i < nh * p.vp; i += kDecThreads) so[i] = 0.f;
  }
  cluster_sync_all();
  // every CTA of the cluster finishes a share of the heads' columns
  for (int i = split * kDecThreads + tid; i < nh * p.vdim && inside; i += a.splits * kDecThreads) {
    const int h = i / p.vdim, c = i - h * p.vdim;
    float m = -FLT_MAX, v = 0.f, sum = 0.f;
    for (int s = 0; s < a.splits; ++s) m = fmaxf(m, ld_cluster_f32(sm + h, s));
    for (int s = 0; s < a.splits; ++s) {
      const float w = exp2_approx(ld_cluster_f32(sm + h, s) - m);
      sum = fmaf(w, ld_cluster_f32(sl + h, s), sum);
      v = fmaf(w, ld_cluster_f32(so + h * p.vp + c, s), v);
    }
    a.out[(long long)(hk * group + h0 + h) * p.vp + c] = v / sum;
  }
  cluster_sync_all();                                                    // nobody leaves while its shared memory is read
}

template <int DIM>
int launch_decode_tc(const GroupDecodeArgs& a, cudaStream_t stream, bool pdl) {
  if (const int rc = allow_shared(group_decode_tc_kernel<DIM>, kWalkSmem)) return rc;
  // eight warps with the most stages that fit, four where the rows are too wide for two stages of eight (or the merge for their rings)
  WalkShape w = {8, 4};
  const int dp = a.p.dp, vp = a.p.vp;
  auto merge = [&]() { return 4 * kWalkM * (w.warps * (vp + 4) + vp); };
  while (w.stages > 2 && walk_smem(dp, vp, w) > kWalkSmem) --w.stages;
  if (walk_smem(dp, vp, w) > kWalkSmem || merge() > walk_ring(dp, vp, w)) w = {4, 3};
  const int smem = walk_smem(dp, vp, w);
  if (smem > kWalkSmem || merge() > walk_ring(dp, vp, w)) return -3;
  const int group = a.p.heads / a.p.kv_heads;
  return launch_cluster(group_decode_tc_kernel<DIM>, dim3(a.splits, a.p.kv_heads, (group + kWalkM - 1) / kWalkM), dim3(kDecThreads), dim3(a.splits, 1, 1),
                        smem, stream, pdl, a, w);
}

template <bool F32, int VC>
int launch_decode(const GroupDecodeArgs& a, cudaStream_t stream, bool pdl) {
  const int smem = 4 * group_smem_floats(a.p.dp, a.p.vp);
  if (const int rc = allow_shared(group_decode_kernel<F32, VC>, 64 * 1024)) return rc;
  const int group = a.p.heads / a.p.kv_heads;
  return launch_cluster(group_decode_kernel<F32, VC>, dim3(a.splits, a.p.kv_heads, (group + kHB - 1) / kHB), dim3(kDecThreads), dim3(a.splits, 1, 1), smem, stream,
                        pdl, a);
}

bool prep_ok(const GroupPrepArgs& p) {
  return p.heads >= 1 && p.kv_heads >= 1 && p.heads % p.kv_heads == 0 && p.dim >= 1 && p.dim <= p.dp && p.dp <= kMaxHead && p.vdim >= 1 &&
         p.vdim <= p.vp && p.vp <= kMaxHead && p.dp % 8 == 0 && p.vp % 8 == 0 && p.rot_dims >= 0 && p.rot_dims % 2 == 0 && p.rot_dims <= p.dim &&
         (p.rot_dims == 0 || p.freq) && p.rows >= 1;
}

}  // namespace

#define S(stream) reinterpret_cast<cudaStream_t>(stream)

extern "C" int nrt_group_prep_args_size() { return (int)sizeof(GroupPrepArgs); }
extern "C" int nrt_transpose_args_size() { return (int)sizeof(TransposeArgs); }
extern "C" int nrt_group_decode_args_size() { return (int)sizeof(GroupDecodeArgs); }

extern "C" int nrt_group_prep(const void* args, void* stream, int pdl) {
  GroupPrepArgs p;
  memcpy(&p, args, sizeof(p));
  if (!prep_ok(p) || !p.q) return -3;
  return launch_pdl(group_prep_kernel, dim3(p.rows), dim3(256), 0, S(stream), pdl != 0, p);
}

extern "C" int nrt_transpose(const void* args, void* stream, int pdl) {
  TransposeArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.rows < 1 || a.cols < 1 || a.cols % 2 || a.dst_ld % 2 || a.dst_ld < a.rows) return -3;
  return launch_pdl(transpose_kernel, dim3((a.rows + 63) / 64, (a.cols + 63) / 64), dim3(256), 0, S(stream), pdl != 0, a);
}

extern "C" int nrt_group_decode(const void* args, void* stream, int pdl) {
  GroupDecodeArgs a;
  memcpy(&a, args, sizeof(a));
  if (!prep_ok(a.p) || a.p.rows != 1 || a.splits < 1 || a.splits > 8 || a.window < 0) return -3;
  const bool wide = a.p.vdim > kDecThreads, p = pdl != 0;
  if (!a.p.f32 && a.p.dp <= kTcHead && a.p.vp <= kTcHead) return a.p.dp <= 128 && a.p.vp <= 128 ? launch_decode_tc<128>(a, S(stream), p) : launch_decode_tc<256>(a, S(stream), p);
  if (a.p.f32) return wide ? launch_decode<true, 2>(a, S(stream), p) : launch_decode<true, 1>(a, S(stream), p);
  return wide ? launch_decode<false, 2>(a, S(stream), p) : launch_decode<false, 1>(a, S(stream), p);
}
