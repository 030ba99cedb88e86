// Block-draft specific kernels: block input rows (anchor embedding + mask embeddings) and the
// sequential Markov head (low-rank previous-token bias + Gumbel-max proposal per row).
//
// The reference precomputes a [vocab, vocab/8] bf16 bias table (5.8 GB per rank,
// naivert/entry/dspark_head_markov_entry.cu:31,87) and looks up one row per step; here the
// rank-256 factors stay factored: each step evaluates bias = W2_shard . W1[prev] on the fly
// (W2_shard is 9.7 MB per rank at tp = 8 and stays L2 resident across the seven steps).
// Reference math: naivert/body/dspark_head_markov/markov_body.cuh:6-27,
// naivert/body/dspark_sampling/random.cuh:17-20 (Gumbel-max over (logits + bias) / T).
#include "contract.h"
#include "fabric.cuh"
#include "launch.hpp"

#include <float.h>
#include <string.h>

using namespace nrt;

namespace {

// x[0] = embed[anchor], x[1..rows) = mask embedding, x[rows..16) = 0
__global__ void draft_block_input_kernel(const int* block_ids, const __nv_bfloat16* __restrict__ embed,
                                         const __nv_bfloat16* __restrict__ mask, __nv_bfloat16* __restrict__ x, int hidden,
                                         int rows, int vocab) {
  griddep_wait();
  griddep_launch();
  const int r = blockIdx.x;
  uint4* dst = reinterpret_cast<uint4*>(x + (size_t)r * hidden);
  const uint4* src = nullptr;
  if (r == 0) {
    int t = block_ids[0];
    t = t < 0 ? 0 : (t >= vocab ? vocab - 1 : t);
    src = reinterpret_cast<const uint4*>(embed + (size_t)t * hidden);
  } else if (r < rows) {
    src = reinterpret_cast<const uint4*>(mask);
  }
  for (int i = threadIdx.x; i < hidden / 8; i += blockDim.x) dst[i] = src ? src[i] : make_uint4(0, 0, 0, 0);
}

struct MarkovArgs {
  const float* logits;            // [16][ld] draft head logits (row j proposes token j+1)
  int ld;
  const __nv_bfloat16* w1;        // [vocab][rank]
  const __nv_bfloat16* w2;        // [vlocal][rank]
  int rank_dim, vlocal, vbase, vocab;
  int* block_ids;                 // [8]; block_ids[step] is the previous token, block_ids[step+1] is written
  float* zq;                      // [8][ld] logits + bias (the draft distribution the sampler sees)
  const float* params;            // sampler params ([6] = 1/T of the draft)
  const unsigned long long* seed;
  const int* ctrl;                // round counter at [8]
  unsigned long long* best;       // scratch: packed (ordered value << 32 | ~token)
  unsigned int* ticket;
  XchgArgs x;
};

// Eight lanes share one token row; lane `sub` takes channels k * 64 + sub * 8 .. + 8 of every 64-channel chunk k, so that
// a 16-byte load of a warp covers whole 128-byte lines.  Every form of the head uses this order of the sum (explicit
// fused multiply-adds, then lanes 1, 2, 4 apart): a proposal does not depend on the form that drew it.
__device__ __forceinline__ float markov_fold(float acc, const uint4 v, const float* w) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __bfloat1622float2(h[j]);
    acc = fmaf(f.x, w[2 * j], acc);
    acc = fmaf(f.y, w[2 * j + 1], acc);
  }
  return acc;
}
__device__ __forceinline__ float markov_lanes(float acc) {
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  acc += __shfl_xor_sync(0xffffffffu, acc, 4);
  return acc;
}

// grid = ceil(vlocal / 128) CTAs of 256 threads; 8 lanes per token row, 4 rounds of 32 rows.
__global__ void __launch_bounds__(256) markov_step_kernel(const MarkovArgs a, int step) {
  __shared__ float w1s[512];
  __shared__ unsigned long long sbest;
  __shared__ bool s_last;
  __shared__ uint64_t xv[16];
  griddep_wait();
  griddep_launch();
  int prev = a.block_ids[step];
  (void)NRT_INDEX_OK(prev, a.vocab, kBoundsMarkovPrev);
  prev = prev < 0 ? 0 : (prev >= a.vocab ? a.vocab - 1 : prev);
  for (int i = threadIdx.x; i < a.rank_dim; i += 256) w1s[i] = __bfloat162float(a.w1[(size_t)prev * a.rank_dim + i]);
  if (threadIdx.x == 0) sbest = 0ull;
  __syncthreads();
  const float inv_t = a.params[6];
  const unsigned long long seed = *a.seed;
  const uint32_t ctr = (uint32_t)a.ctrl[NRT_CTRL_ROUND] * 8u + (uint32_t)step;
  unsigned long long best = 0ull;
  const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3;         // 32 groups per CTA
  for (int i = 0; i < 4; ++i) {
    const int t = blockIdx.x * 128 + i * 32 + grp;
    float acc = 0.f;
    if (t < a.vlocal) {
      const uint4* wr = reinterpret_cast<const uint4*>(a.w2 + (size_t)t * a.rank_dim) + sub;
      for (int k = 0; k < a.rank_dim / 64; ++k) acc = markov_fold(acc, wr[k * 8], w1s + k * 64 + sub * 8);
    }
    acc = markov_lanes(acc);
    if (sub == 0 && t < a.vlocal) {
      const float z = a.logits[(size_t)step * a.ld + t] + round_bf16(acc);
      a.zq[(size_t)step * a.ld + t] = z;
      const float u = philox_uniform(seed, 3u, ctr, (uint32_t)(t + a.vbase));
      const float g = -__logf(-__logf(u));
      const float s = z * inv_t + g;
      // larger score wins; ties go to the lower token id
      const unsigned long long key = ((unsigned long long)float_order(s) << 32) | (uint32_t)(~(uint32_t)(t + a.vbase));
      best = key > best ? key : best;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(&sbest, best);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(a.best, sbest);
    __threadfence();
    const unsigned int tk = atomicAdd(a.ticket, 1u);
    s_last = tk == gridDim.x - 1;
    if (s_last) *a.ticket = 0u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x < 16) xv[threadIdx.x] = threadIdx.x == 0 ? *reinterpret_cast<volatile unsigned long long*>(a.best) : 0ull;
  __syncthreads();
  xchg_reduce_u64<kXMax>(xv, 1, a.x, 16 + step);
  if (threadIdx.x == 0) {
    a.block_ids[step + 1] = (int)(~(uint32_t)xv[0]);
    *a.best = 0ull;
  }
}

// End of a step inside the one-launch forms, first half: every CTA folds its best candidate into best[step] and adds
// itself to a monotonic arrival counter.  The CTA that completes the count runs the tensor-parallel exchange, writes
// block_ids[step + 1] and publishes the step's generation.  A single rank has nothing to exchange: there the count itself
// releases the other CTAs, which read the winner on their own (one hop through the L2 less, 1.7 us of a step), and a
// step's word is cleared by the last CTA of the next step, when everybody has read it.
struct MarkovTurn {
  unsigned long long count;       // arrivals that complete this step
  unsigned int gen;               // its generation
  bool last;                      // (thread 0) this CTA completed it
};
__device__ __forceinline__ MarkovTurn markov_arrive(const MarkovArgs& a, int step, int steps, unsigned long long best,
                                                    unsigned long long* arrive, unsigned int* step_gen) {
  __shared__ unsigned long long s_best[32];
  __shared__ unsigned long long s_old;
  __shared__ uint64_t xv[16];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)blockDim.x / 32; ++i) best = s_best[i] > best ? s_best[i] : best;
    atomicMax(a.best + step, best);
    __threadfence();
    s_old = atomicAdd(arrive, 1ull);
  }
  __syncthreads();
  MarkovTurn t;
  t.count = (s_old / gridDim.x + 1ull) * gridDim.x;
  t.gen = (unsigned int)(s_old / gridDim.x + 1ull);
  t.last = s_old + 1ull == t.count;
  if (t.last) {
    __threadfence();
    if (threadIdx.x < 16) xv[threadIdx.x] = threadIdx.x == 0 ? *reinterpret_cast<volatile unsigned long long*>(a.best + step) : 0ull;
    __syncthreads();
    xchg_reduce_u64<kXMax>(xv, 1, a.x, 16 + step);
    if (threadIdx.x == 0) {
      a.block_ids[step + 1] = (int)(~(uint32_t)xv[0]);
      if (a.x.tp > 1 || step + 1 == steps) a.best[step] = 0ull;
      if (a.x.tp <= 1 && step > 0) a.best[step - 1] = 0ull;
      if (a.x.tp > 1) {
        __threadfence();
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(step_gen), "r"(t.gen) : "memory");
      }
    }
  }
  return t;
}
// Second half: the next step's previous token (-1: the bounded wait gave up).  Not called after the last step.
__device__ __forceinline__ int markov_wait(const MarkovArgs& a, int step, const MarkovTurn& t, const unsigned long long* arrive,
                                           const unsigned int* step_gen) {
  __shared__ int s_prev;
  if (threadIdx.x == 0) {
    bool ok = true;
    if (!(t.last && a.x.tp > 1)) {
      const uint64_t deadline = globaltimer() + kWaitLimitNs;
      for (uint32_t i = 0;; ++i) {
        // counts and generations only grow: a later step's value also releases this wait
        if (a.x.tp > 1 ? (int)(ld_acquire_gpu(step_gen) - t.gen) >= 0 : ld_acquire_gpu64(arrive) >= t.count) break;
        if ((i & 255u) == 255u) {
          if (*reinterpret_cast<volatile uint32_t*>(a.x.status) != 0u) { ok = false; break; }
          if (globaltimer() > deadline) { report(a.x.status, kSiteGrid | 0x20u | (uint32_t)step); ok = false; break; }
        }
      }
    }
    int prev = a.x.tp > 1 ? __ldcg(a.block_ids + step + 1) : (int)(~(uint32_t)*reinterpret_cast<const volatile unsigned long long*>(a.best + step));
    (void)NRT_INDEX_OK(prev, a.vocab, kBoundsMarkovPrev);
    prev = prev < 0 ? 0 : (prev >= a.vocab ? a.vocab - 1 : prev);
    s_prev = ok ? prev : -1;
  }
  __syncthreads();
  return s_prev;
}

// All proposals of a block in one launch: the same per-step work as markov_step_kernel, with the hand-over of the
// sampled token between steps done inside the grid (markov_arrive, markov_wait).  The grid must be resident at once (checked at
// launch), which bounds it to shards of 148 * 2 * 128 tokens; markov_wide_kernel takes larger ones.
__global__ void __launch_bounds__(256, 2) markov_chain_kernel(const MarkovArgs a, int steps, unsigned long long* arrive,
                                                           unsigned int* step_gen) {
  __shared__ float w1s[512];
  const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3;
  // rank 256 (the shipped geometry): a thread's slice of the second factor - four tokens x 32 channels - does not
  // depend on the step, so it is loaded once and stays in registers for all steps; per step only the previous
  // token's row of the first factor and the step's base logits are fetched, all loads in flight together
  const bool fast = a.rank_dim == 256;
  uint4 wv[4][4];
  if (fast) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = blockIdx.x * 128 + i * 32 + grp;
      const bool on = t < a.vlocal;
      const uint4* wr = reinterpret_cast<const uint4*>(a.w2 + (size_t)(on ? t : 0) * 256) + sub;
#pragma unroll
      for (int k = 0; k < 4; ++k) wv[i][k] = on ? __ldg(wr + k * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  griddep_wait();                                  // the factor is a weight: its loads above overlap the predecessor's tail
  griddep_launch();
  const float inv_t = a.params[6];
  const unsigned long long seed = *a.seed;
  const uint32_t round = (uint32_t)a.ctrl[NRT_CTRL_ROUND];
  int prev = a.block_ids[0];
  (void)NRT_INDEX_OK(prev, a.vocab, kBoundsMarkovPrev);
  prev = prev < 0 ? 0 : (prev >= a.vocab ? a.vocab - 1 : prev);
  for (int step = 0; step < steps; ++step) {
    float base[4];
    if (fast) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = blockIdx.x * 128 + i * 32 + grp;
        base[i] = (t < a.vlocal && sub == 0) ? a.logits[(size_t)step * a.ld + t] : 0.f;
      }
    }
    for (int i = threadIdx.x; i < a.rank_dim; i += 256) w1s[i] = __bfloat162float(a.w1[(size_t)prev * a.rank_dim + i]);
    __syncthreads();
    const uint32_t ctr = round * 8u + (uint32_t)step;
    unsigned long long best = 0ull;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = blockIdx.x * 128 + i * 32 + grp;
      float acc = 0.f;
      if (fast) {
#pragma unroll
        for (int k = 0; k < 4; ++k) acc = markov_fold(acc, wv[i][k], w1s + k * 64 + sub * 8);
      } else if (t < a.vlocal) {
        const uint4* wr = reinterpret_cast<const uint4*>(a.w2 + (size_t)t * a.rank_dim) + sub;
        for (int k = 0; k < a.rank_dim / 64; ++k) acc = markov_fold(acc, wr[k * 8], w1s + k * 64 + sub * 8);
      }
      acc = markov_lanes(acc);
      if (sub == 0 && t < a.vlocal) {
        const float z = (fast ? base[i] : a.logits[(size_t)step * a.ld + t]) + round_bf16(acc);
        a.zq[(size_t)step * a.ld + t] = z;
        const float u = philox_uniform(seed, 3u, ctr, (uint32_t)(t + a.vbase));
        const float g = -__logf(-__logf(u));
        const float sc = z * inv_t + g;
        const unsigned long long key = ((unsigned long long)float_order(sc) << 32) | (uint32_t)(~(uint32_t)(t + a.vbase));
        best = key > best ? key : best;
      }
    }
    const MarkovTurn turn = markov_arrive(a, step, steps, best, arrive, step_gen);
    if (step + 1 < steps && (prev = markov_wait(a, step, turn, arrive, step_gen)) < 0) return;
  }
}

// The same chain for a shard whose second factor does not fit the register files of one resident grid (a whole
// vocabulary on one GPU: 78 MB at 152,576 tokens).  One CTA of 16 warps per SM; a warp owns 4 * iters consecutive
// tokens and keeps the first `cached` groups of four in shared memory for all steps, the rest is read from L2 in every
// step.  Bound by that read: 7 of 17 groups stay on the SM (31 MB over the chip), so that the remaining 45 MB also fit
// the half of the L2 that is near an SM.  Measured (152,576 tokens, seven steps): 81 us against 166 us for seven launches in a
// loop; inside a round, where those find the factor evicted, 0.32 ms less.  The Gumbel noise of a token does not depend on the previous token: a step's
// noise and base logits are taken, a token per lane, while the grid waits for the step before.
constexpr int kWideWarps = 16, kWideCached = 7, kWideBatches = 3;
__global__ void __launch_bounds__(kWideWarps * 32, 1) markov_wide_kernel(const MarkovArgs a, int steps, int iters,
                                                                         unsigned long long* arrive, unsigned int* step_gen) {
  extern __shared__ uint4 sw[];                     // [cached][warp][4][lane]: a lane reads back what it wrote
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 7, grp = lane >> 3;
  const int first = (blockIdx.x * kWideWarps + warp) * 4 * iters;
  const int cached = min(iters, kWideCached);
  const uint4* w2 = reinterpret_cast<const uint4*>(a.w2) + sub;
  const auto row = [&](int j) { return w2 + (size_t)min(first + j * 4 + grp, a.vlocal - 1) * 32; };
  const auto token = [&](int b) {                   // this lane's token of batch b (eight groups of four), -1: none
    const int j = b * 8 + sub, t = first + j * 4 + grp;
    return j < iters && t < a.vlocal ? t : -1;
  };
  uint4* mine = sw + warp * 128 + lane;
  for (int j = 0; j < cached; ++j) {
    const uint4* r = row(j);
#pragma unroll
    for (int k = 0; k < 4; ++k) mine[j * kWideWarps * 128 + k * 32] = __ldg(r + k * 8);
  }
  griddep_wait();                                   // the factor is a weight: its loads above overlap the predecessor's tail
  griddep_launch();
  const float inv_t = a.params[6];
  const unsigned long long seed = *a.seed;
  const uint32_t round = (uint32_t)a.ctrl[NRT_CTRL_ROUND];
  float base[kWideBatches], noise[kWideBatches];
  const auto ahead = [&](int step) {
#pragma unroll
    for (int b = 0; b < kWideBatches; ++b) {
      const int t = token(b);
      base[b] = t >= 0 ? a.logits[(size_t)step * a.ld + t] : 0.f;
    }
#pragma unroll
    for (int b = 0; b < kWideBatches; ++b) {
      const int t = token(b);
      const float u = t >= 0 ? philox_uniform(seed, 3u, round * 8u + (uint32_t)step, (uint32_t)(t + a.vbase)) : 0.5f;
      noise[b] = -__logf(-__logf(u));
    }
  };
  ahead(0);
  int prev = a.block_ids[0];
  (void)NRT_INDEX_OK(prev, a.vocab, kBoundsMarkovPrev);
  prev = prev < 0 ? 0 : (prev >= a.vocab ? a.vocab - 1 : prev);
  for (int step = 0; step < steps; ++step) {
    float w[32];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.w1 + (size_t)prev * 256) + k * 8 + sub);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        w[k * 8 + 2 * j] = f.x;
        w[k * 8 + 2 * j + 1] = f.y;
      }
    }
    unsigned long long best = 0ull;
#pragma unroll
    for (int b = 0; b < kWideBatches; ++b) {
      if (b * 8 >= iters) break;
      float bias = 0.f;
#pragma unroll 4
      for (int i = 0; i < 8; ++i) {
        const int j = b * 8 + i;
        if (j >= iters) break;
        uint4 v[4];
        if (j < cached) {
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = mine[j * kWideWarps * 128 + k * 32];
        } else {
          const uint4* r = row(j);
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = __ldg(r + k * 8);
        }
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) acc = markov_fold(acc, v[k], w + k * 8);
        acc = markov_lanes(acc);
        bias = sub == i ? acc : bias;
      }
      const int t = token(b);
      if (t >= 0) {
        const float z = base[b] + round_bf16(bias);
        a.zq[(size_t)step * a.ld + t] = z;
        const float sc = z * inv_t + noise[b];
        const unsigned long long key = ((unsigned long long)float_order(sc) << 32) | (uint32_t)(~(uint32_t)(t + a.vbase));
        best = key > best ? key : best;
      }
    }
    const MarkovTurn turn = markov_arrive(a, step, steps, best, arrive, step_gen);
    if (step + 1 == steps) break;
    ahead(step + 1);
    if ((prev = markov_wait(a, step, turn, arrive, step_gen)) < 0) return;
  }
}

}  // namespace

#define S(stream) reinterpret_cast<cudaStream_t>(stream)

extern "C" int nrt_draft_block_input(const int* block_ids, const void* embed, const void* mask, void* x, int hidden,
                                     int rows, int vocab, void* stream, int pdl) {
  return launch_pdl(draft_block_input_kernel, dim3(16), dim3(128), 0, S(stream), pdl != 0, block_ids,
                    (const __nv_bfloat16*)embed, (const __nv_bfloat16*)mask, (__nv_bfloat16*)x, hidden, rows, vocab);
}
extern "C" int nrt_markov_args_size() { return (int)sizeof(MarkovArgs); }
NRT_BOUNDS_EXPORT(draft)
// steps proposals in one launch.  `sync`: two 64-bit words (arrival counter, step generation), zero-initialised once.
extern "C" int nrt_markov_chain(const void* args, int steps, void* sync, void* stream, int pdl) {
  MarkovArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.rank_dim > 512 || a.rank_dim % 64 || steps < 1 || steps > 8 || !sync) return -3;
  const int grid = (a.vlocal + 127) / 128;
  constexpr int wide_smem = kWideCached * kWideWarps * 128 * (int)sizeof(uint4);
  static int resident = -1, wide = -1;            // CTAs of the two forms that fit at once
  if (resident < 0) {
    int per_sm = 0, wide_per_sm = 0, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, markov_chain_kernel, 256, 0) != cudaSuccess) return -3;
    if (allow_shared(markov_wide_kernel, wide_smem) ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&wide_per_sm, markov_wide_kernel, kWideWarps * 32, wide_smem) != cudaSuccess)
      wide_per_sm = 0;                            // the other forms do not need it
    wide = wide_per_sm * sms;
    resident = per_sm * sms;
  }
  unsigned long long* w = reinterpret_cast<unsigned long long*>(sync);
  // the in-grid hand-over needs every CTA resident: shards beyond what the register form holds at once take the wide one
  if (grid > resident) {
    if (a.rank_dim != 256 || wide < 1 || allow_shared(markov_wide_kernel, wide_smem)) return -9;
    const int iters = (a.vlocal + wide * kWideWarps * 4 - 1) / (wide * kWideWarps * 4);
    if (iters > 8 * kWideBatches) return -9;      // beyond 227,328 tokens: one launch per step
    const int ctas = (a.vlocal + kWideWarps * 4 * iters - 1) / (kWideWarps * 4 * iters);
    return launch_pdl(markov_wide_kernel, dim3(ctas), dim3(kWideWarps * 32), wide_smem, S(stream), pdl != 0, a, steps, iters, w,
                      reinterpret_cast<unsigned int*>(w + 1));
  }
  return launch_pdl(markov_chain_kernel, dim3(grid), dim3(256), 0, S(stream), pdl != 0, a, steps, w,
                    reinterpret_cast<unsigned int*>(w + 1));
}
extern "C" int nrt_markov_step(const void* args, int step, void* stream, int pdl) {
  MarkovArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.rank_dim > 512 || a.rank_dim % 64) return -3;
  return launch_pdl(markov_step_kernel, dim3((a.vlocal + 127) / 128), dim3(256), 0, S(stream), pdl != 0, a, step);
}
