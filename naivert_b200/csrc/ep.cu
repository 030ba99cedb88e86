// Expert-parallel all-to-all for prefill: dispatch fused with RMS-normalised activation
// quantisation and the expert permutation, and the combine (return of expert outputs to the
// token owner, probability-weighted sum + residual), all over peer memory.
//
//   ep_count     every rank histograms its (token, k) -> expert choices, the [ranks x experts] count
//                matrix is exchanged with tagged words, and every rank derives (a) the destination row of
//                each of its (token, k) pairs - rows land *expert-sorted and contiguous* in the expert
//                rank's receive buffer, each expert segment padded to 16 rows - and (b) the work list
//                (expert, first row) of 16-row groups for the grouped GEMM on its own experts.
//   ep_dispatch  one CTA per token: e4m3 + power-of-two scale per 128 channels, then one 4 KiB row + scales
//                + metadata stored straight into the destination rank's receive buffer for each of the
//                token's experts; the last CTA publishes a per-source "dispatch complete" flag to every rank.
//   (grouped block-scaled GEMMs run on the receive buffer: csrc/gemm.cuh, group-item mode)
//   ep_return    epilogue helper of the down projection: bf16 expert outputs are pushed as tagged words
//                into the owner's combine buffer slot (token, k).
//   ep_combine   owner side: waits for the top-k slots of each token, adds them in fixed k order weighted by
//                the routing probability in fp32 on top of the residual.
//
// Reference counterparts: vendored DeepEP intranode dispatch (naivert/prefill/native/deepep.py),
// Triton scatter/permute (naivert/kernels/naive_n0p5/prefill_sglang/), sgl per-token-group fp8 quant, and
// naivert/prefill/native/native_combine.cu (tagged-word combine).
#include "fabric.cuh"
#include "gemm.cuh"
#include "launch.hpp"

#include <string.h>

using namespace nrt;

namespace {

constexpr int kEpMaxExperts = 512;

struct EpArgs {
  // routing of the local tokens
  const int* topk_ids;        // [tokens][top_k] global expert ids
  const float* topk_p;        // [tokens][top_k]
  int tokens, top_k, experts, experts_local, hidden;
  // count outputs (local)
  int* slot_of;               // [tokens*top_k] destination row of each pair
  int* n_items;               // grouped-GEMM work list of this rank's experts
  int* item_expert;           // [max_items] local expert id
  int* item_row;              // [max_items] first row of the item's row group
  int* seg_rows;              // [experts_local] rows received per local expert (unpadded)
  int max_items;
  int cap_rows;               // receive buffer capacity in rows
  // dispatch
  const __nv_bfloat16* x;     // [tokens][hidden] residual rows
  const __nv_bfloat16* gamma; // RMSNorm weight (null: rows are already normalised)
  float eps;
  uint8_t* recv8[kXchgPeers];    // [cap_rows][hidden] e4m3
  float* recvs[kXchgPeers];      // [cap_rows][hidden/128]
  int4* meta[kXchgPeers];        // [cap_rows] {src rank, token, k, tag}
  uint64_t* flags[kXchgPeers];   // [tp] dispatch-complete words
  unsigned int* ticket;
  int call;                      // tag call index of this layer's dispatch
  int item_rows;                 // rows per grouped-GEMM work item and segment padding (16 or 64; 0 = 16)
  XchgArgs x_args;
  int* item_live;                // [max_items] rows of the item that carry a token (null: not wanted)
};

// ----------------------------------------------------------------------------- counts + layout
constexpr int kBatch = 8;                  // pairs of a lane that are loaded at once
// sum over the lower lanes of a warp
__device__ __forceinline__ int lanes_before(int v, int lane) {
  int s = v;
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const int t = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += t;
  }
  return s - v;
}
__global__ void __launch_bounds__(1024) ep_count_kernel(const EpArgs a) {
  __shared__ unsigned int hist[kEpMaxExperts + 1];
  __shared__ uint64_t xv[kXchgMaxWords];          // [tp][experts]
  __shared__ int seg_base[kEpMaxExperts + 1];
  griddep_wait();
  griddep_launch();
  const int tp = a.x_args.tp, rank = a.x_args.rank;
  const int n = a.tokens * a.top_k;
  const int ir = a.item_rows > 0 ? a.item_rows : 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Up to 256 experts every warp owns one contiguous range of the pairs.  Pass 1 counts the range's pairs per expert (warp-private row of
  // 16-bit counters, in the unused upper half of the exchange buffer: 32 x 256 x 2 bytes), a prefix over the warps turns the counts into
  // each range's offset inside the expert's segment, pass 2 walks the range in index order and hands out rows.  Same stable order as ranking
  // the pairs one by one (lower index first).  A pass is a chain of loads and exchanges over 32 pairs at a time, so eight loads are made at
  // once, nothing else reads the pairs, and lanes find their like by votes: 65,536 pairs of 256 experts 80 us (295 us with a load at a
  // time, a match over the warp and a histogram in front), 16,384 pairs 27 us (95 us).
  const bool ranges = a.experts <= 256 && tp * a.experts <= kXchgMaxWords / 2;
  unsigned short (*wc)[256] = reinterpret_cast<unsigned short (*)[256]>(xv + kXchgMaxWords / 2);
  const int per = (n + 31) / 32, lo = warp * per, hi = min(n, lo + per);
  auto walk = [&](auto&& each) {                             // each(pair, its expert or -1, lanes with the same)
    for (int i0 = lo; i0 < hi; i0 += 32 * kBatch) {
      int e[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * 32 + lane;
        e[b] = i < hi ? a.topk_ids[i] : -1;
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        if (i0 + b * 32 >= hi) break;
        // lanes with the same expert: nine votes (a match over the warp takes a turn per different value)
        unsigned peers = __ballot_sync(0xffffffffu, e[b] >= 0);
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
          const unsigned with = __ballot_sync(0xffffffffu, (e[b] >> bit) & 1);
          peers &= (e[b] >> bit) & 1 ? with : ~with;
        }
        each(i0 + b * 32 + lane, e[b], peers);
        __syncwarp();
      }
    }
  };
  for (int i = threadIdx.x; i < tp * a.experts; i += 1024) xv[i] = 0ull;
  if (ranges) {
    for (int i = threadIdx.x; i < 32 * 256; i += 1024) (&wc[0][0])[i] = 0;
    __syncthreads();
    walk([&](int, int e, unsigned peers) {
      if (e >= 0 && (peers & ((1u << lane) - 1u)) == 0u) wc[warp][e] += (unsigned short)__popc(peers);
    });
    __syncthreads();
    if ((int)threadIdx.x < a.experts) {
      unsigned run = 0;
#pragma unroll 8
      for (int w = 0; w < 32; ++w) { const unsigned t = wc[w][threadIdx.x]; wc[w][threadIdx.x] = (unsigned short)run; run += t; }
      xv[rank * a.experts + threadIdx.x] = run;
    }
  } else {
    for (int i = threadIdx.x; i < a.experts; i += 1024) hist[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += 1024) atomicAdd(&hist[a.topk_ids[i]], 1u);
    __syncthreads();
    for (int e = threadIdx.x; e < a.experts; e += 1024) xv[rank * a.experts + e] = hist[e];
  }
  __syncthreads();
  xchg_reduce_u64<kXSum>(xv, tp * a.experts, a.x_args, 32 + (a.call & 15));
  // padded segment bases on every destination rank (all ranks compute the same table): a warp per rank, a lane per run of its experts
  if (warp < tp) {
    const int run = (a.experts_local + 31) / 32, first = lane * run, last = min(a.experts_local, first + run);
    auto padded = [&](int el) {
      int rows = 0;
      for (int s = 0; s < tp; ++s) rows += (int)xv[s * a.experts + warp * a.experts_local + el];
      return (rows + ir - 1) / ir * ir;
    };
    int sum = 0;
    for (int el = first; el < last; ++el) sum += padded(el);
    int base = lanes_before(sum, lane);
    for (int el = first; el < last; ++el) {
      seg_base[warp * a.experts_local + el] = base;
      base += padded(el);
    }
  }
  __syncthreads();
  // destination row of each local (token, k): segment base + rows of lower ranks + stable local rank.
  // `hist` becomes the running count per expert; pairs are ranked in index order: chunks of 1024 in order,
  // warps of a chunk in order, lanes of a warp by their position among equal experts.
  for (int e = threadIdx.x; e < a.experts; e += 1024) {
    int pos = seg_base[e];
    for (int s = 0; s < rank; ++s) pos += (int)xv[s * a.experts + e];
    hist[e] = (unsigned)pos;
  }
  __syncthreads();
  if (ranges) {
    walk([&](int i, int e, unsigned peers) {
      const int below = __popc(peers & ((1u << lane) - 1u));
      if (e >= 0) a.slot_of[i] = (int)(hist[e] + wc[warp][e]) + below;
      __syncwarp();
      if (e >= 0 && below == 0) wc[warp][e] += (unsigned short)__popc(peers);
    });
    __syncthreads();
  } else
  for (int c0 = 0; c0 < n; c0 += 1024) {
    const int i = c0 + threadIdx.x;
    const int e = i < n ? a.topk_ids[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, e);
    const int below = __popc(peers & ((1u << lane) - 1u));
    const bool lead = below == 0;
    for (int w = 0; w < 32; ++w) {
      if (warp == w && e >= 0) {
        unsigned base = 0;
        if (lead) { base = hist[e]; hist[e] = base + __popc(peers); }
        base = __shfl_sync(peers, base, __ffs(peers) - 1);
        a.slot_of[i] = (int)base + below;
      }
      __syncthreads();
    }
  }
  // work list of my own experts: one thread per local expert counts its row groups, a prefix over the experts gives
  // each its first item, then every thread writes its own items (same list as a sequential walk over the experts)
  {
    int* first_item = reinterpret_cast<int*>(hist);          // hist is free again: [experts_local + 1]
    int my_rows = 0, my_items = 0;
    const int el = threadIdx.x;
    if (el < a.experts_local) {
      const int e = rank * a.experts_local + el;
      for (int s = 0; s < tp; ++s) my_rows += (int)xv[s * a.experts + e];
      a.seg_rows[el] = my_rows;
      my_items = (my_rows + ir - 1) / ir;
    }
    __syncthreads();                                          // everybody is done with hist as running positions
    if (el < a.experts_local) first_item[el + 1] = my_items;
    if (el == 0) first_item[0] = 0;
    __syncthreads();
    if (warp == 0) {
      const int run = (a.experts_local + 31) / 32, first = lane * run, last = min(a.experts_local, first + run);
      int sum = 0;
      for (int i = first; i < last; ++i) sum += first_item[i + 1];
      int before = lanes_before(sum, lane);
      for (int i = first; i < last; ++i) first_item[i + 1] = before += first_item[i + 1];
      __syncwarp();
      if (lane == 0) *a.n_items = min(first_item[a.experts_local], a.max_items);
    }
    __syncthreads();
    if (el < a.experts_local) {
      const int e = rank * a.experts_local + el;
      for (int k = 0; k < my_items; ++k) {
        const int idx = first_item[el] + k;
        if (idx < a.max_items) {
          a.item_expert[idx] = el;
          a.item_row[idx] = seg_base[e] + k * ir;
          if (a.item_live) a.item_live[idx] = min(ir, my_rows - k * ir);
        }
      }
    }
  }
}

__device__ __forceinline__ uint8_t e4m3_of(float v) {
  const __nv_fp8_e4m3 q(v);
  return *reinterpret_cast<const uint8_t*>(&q);
}

// ----------------------------------------------------------------------------- dispatch
// One CTA (256 threads) per local token.
__global__ void __launch_bounds__(256) ep_dispatch_kernel(const EpArgs a) {
  __shared__ float red[8];
  __shared__ bool s_last;
  griddep_wait();
  griddep_launch();
  const int t = blockIdx.x;
  const int per = a.hidden / 8;
  const int tp = a.x_args.tp, rank = a.x_args.rank;
  const uint32_t tag = (*a.x_args.epoch) * 1024u + (uint32_t)a.call + 1u;
  const uint4* src = reinterpret_cast<const uint4*>(a.x + (size_t)t * a.hidden);
  float rs = 1.f;
  if (a.gamma) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < per; i += 256) {
      const uint4 v = src[i];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(h[j]); ss += f.x * f.x + f.y * f.y; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.f;
    for (int i = 0; i < 8; ++i) ss += red[i];
    rs = rsqrtf(ss / (float)a.hidden + a.eps);
  }
  for (int i = threadIdx.x; i < per; i += 256) {
    const uint4 v = src[i];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
    float o[8];
    float am = 0.f;
    if (a.gamma) {
      const uint4 gv = reinterpret_cast<const uint4*>(a.gamma)[i];
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]), g = __bfloat1622float2(gh[j]);
        o[2 * j] = round_bf16(f.x * rs * g.x);
        o[2 * j + 1] = round_bf16(f.y * rs * g.y);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(h[j]); o[2 * j] = f.x; o[2 * j + 1] = f.y; }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(o[j]));
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, off));
    const float sc = pow2_scale(am);
    uint2 q;
    uint8_t* qb = reinterpret_cast<uint8_t*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) qb[j] = e4m3_of(o[j] / sc);
    for (int k = 0; k < a.top_k; ++k) {
      const int e = a.topk_ids[t * a.top_k + k];
      const int d = e / a.experts_local;
      const int row = a.slot_of[t * a.top_k + k];
      if (row >= a.cap_rows) continue;
      reinterpret_cast<uint2*>(a.recv8[d] + (size_t)row * a.hidden)[i] = q;
      if ((i & 15) == 0) a.recvs[d][(size_t)row * (a.hidden / 128) + (i >> 4)] = sc;
    }
  }
  if (threadIdx.x < a.top_k) {
    const int k = threadIdx.x;
    const int e = a.topk_ids[t * a.top_k + k];
    const int row = a.slot_of[t * a.top_k + k];
    if (row < a.cap_rows) a.meta[e / a.experts_local][row] = make_int4(rank, t, k, (int)tag);
  }
  // last CTA: everything this rank sends is out -> publish the flag on every rank
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int tk = atomicAdd(a.ticket, 1u);
    s_last = tk == gridDim.x - 1;
    if (s_last) *a.ticket = 0u;
  }
  __syncthreads();
  if (s_last && threadIdx.x < tp) {
    asm volatile("fence.acq_rel.sys;" ::: "memory");
    st_tagged(a.flags[threadIdx.x] + rank, tag, 1u);
  }
}

// ----------------------------------------------------------------------------- combine (owner side)
struct EpCombineArgs {
  const uint64_t* slots;      // [tokens*top_k][hidden/2] tagged words {tag, bf16x2}
  const float* topk_p;        // [tokens][top_k]
  const __nv_bfloat16* resid; // [tokens][hidden]
  __nv_bfloat16* out;         // [tokens][hidden]
  const uint32_t* epoch;
  uint32_t* status;
  int tokens, top_k, hidden, call;
  unsigned long long timeout_ns;
};

__global__ void __launch_bounds__(256) ep_combine_kernel(const EpCombineArgs a) {
  griddep_wait();
  griddep_launch();
  const int t = blockIdx.x;
  const uint32_t tag = (*a.epoch) * 1024u + (uint32_t)a.call + 1u;
  const int words = a.hidden / 2;
  const uint64_t deadline = globaltimer() + a.timeout_ns;
  // Two words (each complete in itself) per load where rows lie so; those that have not arrived are waited for in turn.  2048 rows of 8
  // choices x 4096: 79 us, 100 us word by word, 112 us with the words of eight choices at once.
  const bool pairs_lie = (words & 1) == 0 && (reinterpret_cast<uintptr_t>(a.slots) & 15) == 0 &&
                         ((reinterpret_cast<uintptr_t>(a.resid) | reinterpret_cast<uintptr_t>(a.out)) & 7) == 0;
  const int pairs = pairs_lie ? words / 2 : 0;
  for (int w = threadIdx.x; w < pairs; w += 256) {
    const uint2 r = reinterpret_cast<const uint2*>(a.resid + (size_t)t * a.hidden)[w];
    float s[4] = {bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y)};
    bool ok = true;
#pragma unroll 4
    for (int k = 0; k < a.top_k && ok; ++k) {                 // fixed k order
      const uint64_t* src = a.slots + ((size_t)(t * a.top_k + k)) * words + 2 * w;
      uint64_t x, y;
      asm volatile("ld.relaxed.sys.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(src) : "memory");
      uint32_t u = (uint32_t)x, v = (uint32_t)y;
      if ((uint32_t)(x >> 32) != tag) ok = wait_tagged(src, tag, u, deadline, a.status, kSiteMailbox | 0x80 | (uint32_t)k);
      if ((uint32_t)(y >> 32) != tag && ok) ok = wait_tagged(src + 1, tag, v, deadline, a.status, kSiteMailbox | 0x80 | (uint32_t)k);
      const float p = a.topk_p[t * a.top_k + k];
      s[0] += p * bf16_lo(u);
      s[1] += p * bf16_hi(u);
      s[2] += p * bf16_lo(v);
      s[3] += p * bf16_hi(v);
    }
    reinterpret_cast<uint2*>(a.out + (size_t)t * a.hidden)[w] = make_uint2(pack_bf16x2(s[0], s[1]), pack_bf16x2(s[2], s[3]));
  }
  for (int w = 2 * pairs + threadIdx.x; w < words; w += 256) {
    const float2 r = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(a.resid + (size_t)t * a.hidden)[w]);
    float lo = r.x, hi = r.y;
    bool ok = true;
    for (int k = 0; k < a.top_k && ok; ++k) {
      uint32_t v;
      ok = wait_tagged(a.slots + ((size_t)(t * a.top_k + k)) * words + w, tag, v, deadline, a.status, kSiteMailbox | 0x80 | (uint32_t)k);
      const float p = a.topk_p[t * a.top_k + k];
      lo += p * bf16_lo(v);
      hi += p * bf16_hi(v);
    }
    reinterpret_cast<__nv_bfloat162*>(a.out + (size_t)t * a.hidden)[w] = __floats2bfloat162_rn(lo, hi);
  }
}

}  // namespace

#define S(stream) reinterpret_cast<cudaStream_t>(stream)
extern "C" int nrt_ep_args_size() { return (int)sizeof(EpArgs); }
extern "C" int nrt_ep_combine_args_size() { return (int)sizeof(EpCombineArgs); }
extern "C" int nrt_ep_count(const void* args, void* stream, int pdl) {
  EpArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.experts > kEpMaxExperts || a.x_args.tp * a.experts > kXchgMaxWords) return -3;
  return launch_pdl(ep_count_kernel, dim3(1), dim3(1024), 0, S(stream), pdl != 0, a);
}
extern "C" int nrt_ep_dispatch(const void* args, void* stream, int pdl) {
  EpArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.hidden % 256 || a.top_k > 32) return -3;
  return launch_pdl(ep_dispatch_kernel, dim3(a.tokens), dim3(256), 0, S(stream), pdl != 0, a);
}
extern "C" int nrt_ep_combine(const void* args, void* stream, int pdl) {
  EpCombineArgs a;
  memcpy(&a, args, sizeof(a));
  return launch_pdl(ep_combine_kernel, dim3(a.tokens), dim3(256), 0, S(stream), pdl != 0, a);
}
