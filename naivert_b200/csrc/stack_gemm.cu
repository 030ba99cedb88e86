// Token-chunk products of layer stacks.
//
// Tensor-core form (bf16): features are the M = 128 side of tcgen05.mma (weights = A operand), token rows the N side
// (64, 128, 192 or 256 per tile), both staged by TMA with 128-byte swizzle.  Persistent CTAs walk the (feature tile, item)
// list; two accumulators in TMEM let the products of the next tile run under the stores of the previous one.
//   warp 0    TMA producer        warp 1    UMMA issuer (and TMEM owner)
//   warps 2-9 epilogue: thread = feature x one half of the token columns
// An item is a row tile of one weight group (plain form: zcount groups, each reading its own columns of the token
// operand - heads or blocks with private weights) or a row segment of a routed expert (item form).  Sizes need no
// padding: the tensor maps carry the true extents and TMA fills the edges of a tile with zeros.
//
// Float form (`nrt_stack_gemm_f32`): the same products and epilogues on the CUDA cores in fp32.
#include "stack.cuh"
#include "launch.hpp"

#include <string.h>

using namespace nrt;

namespace {

constexpr int kFeat = 128;                    // features per tile
constexpr int kKStep = 64;                    // inner elements per stage (128 bytes of bf16)
constexpr int kATile = kFeat * 128;           // bytes
constexpr int kThreads = 320;

template <int NTOK, bool DUAL>
struct Cfg {
  static constexpr int kStage = (DUAL ? 2 : 1) * kATile + NTOK * 128;
  static constexpr int kStages = (200 * 1024) / kStage > 8 ? 8 : (200 * 1024) / kStage;
  static constexpr int kAccCols = (DUAL ? 2 : 1) * NTOK;
  static constexpr int kBufs = 2 * kAccCols <= 512 ? 2 : 1;      // two tiles in flight where they fit
  static constexpr int kTmem = kBufs * kAccCols <= 128 ? 128 : kBufs * kAccCols <= 256 ? 256 : 512;
  static constexpr int kSmem = kStages * kStage + 1024 + 512;
};
static_assert(Cfg<256, false>::kTmem == 512 && Cfg<128, true>::kTmem == 512 && Cfg<64, false>::kTmem == 128 && Cfg<192, true>::kBufs == 1, "TMEM columns");

struct Tail {
  uint64_t full[8], empty[8], acc_full[2], acc_empty[2];
  uint32_t tmem;
};

struct Item { int z, row0, rows; bool live; };              // rows: that count

__device__ __forceinline__ Item item_of(const StackGemmArgs& p, int item, int row_tiles, int ntok, int na) {
  Item it;
  if (p.n_items) {
    it.live = item < na;
    it.z = it.live ? p.item_z[item] : 0;
    it.row0 = it.live ? p.item_row[item] : 0;
    it.rows = it.live && p.item_live ? p.item_live[item] : ntok;
  } else {
    it.live = true;
    it.z = item / row_tiles;
    it.row0 = (item % row_tiles) * ntok;
    it.rows = min(ntok, p.rows - it.row0);
  }
  return it;
}

template <int EPI>
constexpr bool epi_has_bias() { return EPI == kSEpiBias || EPI == kSEpiDecaySoft || EPI == kSEpiDecayExp; }

template <int EPI>
__device__ __forceinline__ float epi_value(const StackGemmArgs& p, float a0, float a1, int n, float bias, float rate) {
  if (EPI == kSEpiBias) {
    const float v = a0 + bias;
    return n < p.act_cols ? gelu_tanh_f(v) : v;
  }
  if (EPI == kSEpiClampedGlu) return clamped_glu(a0, a1, p.limit, p.alpha);
  if (EPI == kSEpiSiluGlu) return silu_glu(a0, a1);
  if (EPI == kSEpiRelu2) return relu2_f(a0);
  if (EPI == kSEpiTanh) return tanhf(a0);
  if (EPI == kSEpiDecaySoft) return decay_soft(a0 + bias, rate);
  if (EPI == kSEpiDecayExp) return decay_exp(a0 + bias);
  return a0 * p.scale;
}

template <int NTOK, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
stack_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW2,
                  const __grid_constant__ CUtensorMap tmX, const StackGemmArgs p, const int n_tiles, const int items,
                  const int row_tiles, const int items_fastest) {
  constexpr bool DUAL = EPI == kSEpiClampedGlu || EPI == kSEpiSiluGlu;
  using C = Cfg<NTOK, DUAL>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Tail* tail = reinterpret_cast<Tail*>(smem + C::kStages * C::kStage);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kb_total = (p.k + kKStep - 1) / kKStep;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::kStages; ++i) { mbar_init(&tail->full[i], 1); mbar_init(&tail->empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tail->acc_full[i], 1); mbar_init(&tail->acc_empty[i], 256); }
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    if (DUAL) tma_prefetch_desc(&tmW2);
  }
  if (warp == 1) { tmem_alloc(&tail->tmem, C::kTmem); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tail->tmem;
  const int total = n_tiles * items;
#define NRT_TILE(w, tile, item)                                    \
  const int tile = items_fastest ? (w) / items : (w) % n_tiles;    \
  const int item = items_fastest ? (w) % items : (w) / n_tiles;

  // The weights of a CTA's first tile are on their way while the launch in front ends.
  int ahead = 0;                                           // stages whose weights have been asked for
  if (warp == 0 && elect_one() && !p.n_items && blockIdx.x < total) {
    NRT_TILE((int)blockIdx.x, tile, item)
    const Item it = item_of(p, item, row_tiles, NTOK, items);
    for (; ahead < C::kStages && ahead < kb_total; ++ahead) {
      uint8_t* s = smem + ahead * C::kStage;
      mbar_expect_tx(&tail->full[ahead], C::kStage);
      tma_load_3d(s, &tmW, &tail->full[ahead], ahead * kKStep, tile * kFeat, it.z);
      if (DUAL) tma_load_3d(s + kATile, &tmW2, &tail->full[ahead], ahead * kKStep, tile * kFeat, it.z);
    }
  }
  griddep_wait();
  griddep_launch();
  const int na = p.n_items ? min(min(*p.n_items, p.max_items), items) : items;

  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      int u = 0;
      for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
        NRT_TILE(w, tile, item)
        const Item it = item_of(p, item, row_tiles, NTOK, na);
        if (!it.live) continue;
        for (int kb = 0; kb < kb_total; ++kb, ++u) {
          const int st = u % C::kStages;
          if (u >= C::kStages && !mbar_wait(&tail->empty[st], ((u / C::kStages) & 1) ^ 1, p.status, kSiteStageEmpty | st)) { ok = false; break; }
          uint8_t* s = smem + st * C::kStage;
          if (u >= ahead) {
            mbar_expect_tx(&tail->full[st], C::kStage);
            tma_load_3d(s, &tmW, &tail->full[st], kb * kKStep, tile * kFeat, it.z);
            if (DUAL) tma_load_3d(s + kATile, &tmW2, &tail->full[st], kb * kKStep, tile * kFeat, it.z);
          }
          tma_load_3d(s + (DUAL ? 2 : 1) * kATile, &tmX, &tail->full[st], kb * kKStep, p.n_items ? 0 : it.z, it.row0);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      bool ok = true;
      int u = 0, t = 0;
      for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
        NRT_TILE(w, tile, item)
        (void)tile;
        const Item it = item_of(p, item, row_tiles, NTOK, na);
        if (!it.live) continue;
        // A tile with few rows is as many columns as it has rows: the rest of a 256-expert layer's second and third segments (8192 rows:
        // 640 segments of 128 for 65,536 pairs) took a fifth of its products (three layers of 4096 x 2048: gate and up 7.66 -> 7.16 ms,
        // down 4.56 -> 4.34).
        const uint32_t idesc = umma_idesc(1u, kFeat, (min(it.rows, NTOK) + 15) / 16 * 16);
        const int buf = t % C::kBufs;
        if (t >= C::kBufs && !mbar_wait(&tail->acc_empty[buf], ((t / C::kBufs) & 1) ^ 1, p.status, kSiteAccEmpty | buf)) { ok = false; break; }
        tc_fence_after();
        for (int kb = 0; kb < kb_total; ++kb, ++u) {
          const int st = u % C::kStages;
          if (!mbar_wait(&tail->full[st], (u / C::kStages) & 1, p.status, kSiteTmaFull | st)) { ok = false; break; }
          tc_fence_after();
          const uint32_t s = smem_u32(smem + st * C::kStage);
          const uint64_t da = umma_desc_sw128(s), da2 = umma_desc_sw128(s + kATile);
          const uint64_t db = umma_desc_sw128(s + (DUAL ? 2 : 1) * kATile);
          const uint32_t d = tmem + buf * C::kAccCols;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            umma_bf16(d, da + 2 * j, db + 2 * j, idesc, kb > 0 || j > 0);
            if (DUAL) umma_bf16(d + NTOK, da2 + 2 * j, db + 2 * j, idesc, kb > 0 || j > 0);
          }
          umma_commit(&tail->empty[st]);
          if (kb == kb_total - 1) umma_commit(&tail->acc_full[buf]);
        }
        ++t;
      }
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const int feat = quad * 32 + lane;
    constexpr int kHalf = NTOK / 2;
    bool ok = true;
    int t = 0;
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      NRT_TILE(w, tile, item)
      const Item it = item_of(p, item, row_tiles, NTOK, na);
      if (!it.live) continue;
      const int buf = t % C::kBufs;
      ok = __all_sync(0xffffffffu, mbar_wait(&tail->acc_full[buf], (t / C::kBufs) & 1, p.status, kSiteAccFull | buf));
      if (!ok) break;
      tc_fence_after();
      const int n = tile * kFeat + feat;
      const bool live = n < p.n;
      const float bias = (epi_has_bias<EPI>() && live) ? bf(p.bias + (size_t)it.z * p.n + n) : 0.f;
      const float rate = (EPI == kSEpiDecaySoft && live) ? p.rate[n] : 0.f;
      const long long zoff = p.n_items ? 0 : it.z * p.out_zstride;
      const uint32_t acc = tmem + (uint32_t(quad * 32) << 16) + buf * C::kAccCols + half * kHalf;
      const int row_end = it.row0 + it.rows, cols = min(kHalf, it.rows - half * kHalf);      // this half's rows
      if (cols <= 0) mbar_arrive(&tail->acc_empty[buf]);
#pragma unroll 1
      for (int c = 0; c < cols; c += 32) {
        uint32_t v0[32], v1[DUAL ? 32 : 1];
        __syncwarp();                               // the loads below are warp-collective
        tmem_ld16_nowait(acc + c, v0);
        tmem_ld16_nowait(acc + c + 16, v0 + 16);
        if (DUAL) {
          tmem_ld16_nowait(acc + NTOK + c, v1);
          tmem_ld16_nowait(acc + NTOK + c + 16, v1 + (DUAL ? 16 : 0));
        }
        tmem_ld_wait();
        if (c + 32 >= cols) {                       // last read of this accumulator: hand it back
          tc_fence_before();
          mbar_arrive(&tail->acc_empty[buf]);
        }
        const int row = it.row0 + half * kHalf + c;
        if (!live) {
        } else if (EPI == kSEpiTranspose) {
          // feature-major: the thread's 32 token columns are contiguous
          uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + zoff + (long long)n * p.out_ld + row);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (row + q * 8 < row_end) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v0[q * 8]), __uint_as_float(v0[q * 8 + 1]));
              o.y = pack_bf16x2(__uint_as_float(v0[q * 8 + 2]), __uint_as_float(v0[q * 8 + 3]));
              o.z = pack_bf16x2(__uint_as_float(v0[q * 8 + 4]), __uint_as_float(v0[q * 8 + 5]));
              o.w = pack_bf16x2(__uint_as_float(v0[q * 8 + 6]), __uint_as_float(v0[q * 8 + 7]));
              dst[q] = o;
            }
          }
        } else {
          const long long at = (long long)row * p.out_ld + zoff + n;
          if (p.out_f32) {
            float* o = reinterpret_cast<float*>(p.out) + at;
#pragma unroll
            for (int r = 0; r < 32; ++r)
              if (row + r < row_end)
                o[(long long)r * p.out_ld] = epi_value<EPI>(p, __uint_as_float(v0[r]), DUAL ? __uint_as_float(v1[DUAL ? r : 0]) : 0.f, n, bias, rate);
          } else {
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at;
#pragma unroll
            for (int r = 0; r < 32; ++r)
              if (row + r < row_end)
                o[(long long)r * p.out_ld] = __float2bfloat16_rn(
                    epi_value<EPI>(p, __uint_as_float(v0[r]), DUAL ? __uint_as_float(v1[DUAL ? r : 0]) : 0.f, n, bias, rate));
          }
        }
      }
      ++t;
    }
  }
#undef NRT_TILE
  drain_on_error(p.status);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, C::kTmem); }
}

int sm_count() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 148;
  }
  return sms;
}

template <int NTOK, int EPI>
int launch(const CUtensorMap& w, const CUtensorMap& w2, const CUtensorMap& x, const StackGemmArgs& a, int items_fastest,
           cudaStream_t stream, bool pdl) {
  constexpr bool DUAL = EPI == kSEpiClampedGlu || EPI == kSEpiSiluGlu;
  using C = Cfg<NTOK, DUAL>;
  auto* kern = stack_gemm_kernel<NTOK, EPI>;
  if (const int rc = allow_shared(kern, C::kSmem)) return rc;
  const int n_tiles = (a.n + kFeat - 1) / kFeat;
  const int row_tiles = (a.rows + NTOK - 1) / NTOK;
  const int items = a.n_items ? a.max_items : a.zcount * row_tiles;
  if (items < 1 || n_tiles < 1 || (long long)items * n_tiles > 0x7fffffffLL) return -3;
  const int total = items * n_tiles, sms = sm_count();
  return launch_pdl(kern, dim3(total < sms ? total : sms), dim3(kThreads), C::kSmem, stream, pdl, w, w2, x, a, n_tiles, items,
                    row_tiles, items_fastest);
}

// ------------------------------------------------------------------------------------ float form
// T x T tiles (features x rows), a thread has T / 16 rows x 4 features; inner steps of 32 through four stages of asynchronous
// copies, weights still bf16 in shared memory.  A product of a small model is a chain of a few steps on a few CTAs, so what counts
// is that no step waits for memory and that tiles are small enough to occupy the SMs: the products of 301 rows of a width of 320 take
// 7.3 us on average, 26 us with 64 x 64 tiles loaded element by element between two barriers.  Every output is one chain of fused multiply-adds in ascending k.
constexpr int kFK = 32, kFStages = 4;

__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {     // the rest of the 16 bytes becomes zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

template <int T, bool DUAL>
struct F32Stage {
  float x[T][kFK + 4];                        // odd strides in 16-byte words: rows fall into different banks
  __nv_bfloat16 w[DUAL ? 2 : 1][T][kFK + 8];
};

template <int T, int EPI>
__global__ void __launch_bounds__(T * 4) stack_gemm_f32_kernel(const StackGemmArgs p, const int row_tiles) {
  constexpr bool DUAL = EPI == kSEpiClampedGlu || EPI == kSEpiSiluGlu;
  constexpr int THREADS = T * 4, TX = T / 4, RT = T / 16;                // threads over features, rows per thread
  extern __shared__ __align__(16) uint8_t f32_smem[];
  using Stage = F32Stage<T, DUAL>;
  Stage* stages = reinterpret_cast<Stage*>(f32_smem);
  griddep_wait();
  griddep_launch();
  Item it;
  int row_lim;
  if (p.n_items) {
    // a segment may be taller than a tile: segments are cut into pieces of T rows
    const int per = (p.item_rows + T - 1) / T;
    const int item = blockIdx.y / per, part = blockIdx.y % per;
    it.live = item < min(*p.n_items, p.max_items);
    if (!it.live) return;
    it.z = p.item_z[item];
    row_lim = p.item_row[item] + (p.item_live ? p.item_live[item] : p.item_rows);
    it.row0 = p.item_row[item] + part * T;
    if (it.row0 >= row_lim) return;
  } else {
    it = item_of(p, blockIdx.y, row_tiles, T, 0);
    row_lim = p.rows;
  }
  const int n0 = blockIdx.x * T;
  const float* X = reinterpret_cast<const float*>(p.act) + (p.n_items ? 0 : it.z * p.act_zstride);
  const __nv_bfloat16* W[2] = {p.w + it.z * p.w_zstride, DUAL ? p.w2 + it.z * p.w_zstride : nullptr};
  const bool vec_x = (reinterpret_cast<uintptr_t>(X) & 15) == 0 && (p.act_ld & 3) == 0;
  const bool vec_w = ((reinterpret_cast<uintptr_t>(W[0]) | (DUAL ? reinterpret_cast<uintptr_t>(W[1]) : 0)) & 15) == 0 && (p.w_ld & 7) == 0;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int steps = (p.k + kFK - 1) / kFK;

  auto load = [&](int step) {
    Stage& st = stages[step % kFStages];
    const int k0 = step * kFK;
    if (vec_x) {
#pragma unroll
      for (int i = threadIdx.x; i < T * (kFK / 4); i += THREADS) {
        const int r = i / (kFK / 4), k = i % (kFK / 4) * 4;
        const int n = it.row0 + r < row_lim ? max(0, min(4, p.k - k0 - k)) : 0;
        copy16(&st.x[r][k], n ? X + (long long)(it.row0 + r) * p.act_ld + k0 + k : X, n * 4);
      }
    } else {
      for (int i = threadIdx.x; i < T * kFK; i += THREADS) {
        const int r = i / kFK, k = i % kFK;
        st.x[r][k] = it.row0 + r < row_lim && k0 + k < p.k ? X[(long long)(it.row0 + r) * p.act_ld + k0 + k] : 0.f;
      }
    }
#pragma unroll
    for (int d = 0; d < (DUAL ? 2 : 1); ++d) {
      if (vec_w) {
#pragma unroll
        for (int i = threadIdx.x; i < T * (kFK / 8); i += THREADS) {
          const int r = i / (kFK / 8), k = i % (kFK / 8) * 8;
          const int n = n0 + r < p.n ? max(0, min(8, p.k - k0 - k)) : 0;
          copy16(&st.w[d][r][k], n ? W[d] + (long long)(n0 + r) * p.w_ld + k0 + k : W[d], n * 2);
        }
      } else {
        for (int i = threadIdx.x; i < T * kFK; i += THREADS) {
          const int r = i / kFK, k = i % kFK;
          st.w[d][r][k] = n0 + r < p.n && k0 + k < p.k ? W[d][(long long)(n0 + r) * p.w_ld + k0 + k] : __float2bfloat16_rn(0.f);
        }
      }
    }
  };
  float acc[RT][4] = {}, acc2[RT][4] = {};
#pragma unroll 1
  for (int i = 0; i < kFStages - 1; ++i) {
    if (i < steps) load(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
#pragma unroll 1
  for (int i = 0; i < steps; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kFStages - 2) : "memory");
    __syncthreads();                                                     // step i has landed; everybody is done with step i - 1
    if (i + kFStages - 1 < steps) load(i + kFStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const Stage& st = stages[i % kFStages];
#pragma unroll
    for (int k = 0; k < kFK; k += 8) {
      float xv[RT][8];
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        *reinterpret_cast<float4*>(&xv[r][0]) = *reinterpret_cast<const float4*>(&st.x[ty * RT + r][k]);
        *reinterpret_cast<float4*>(&xv[r][4]) = *reinterpret_cast<const float4*>(&st.x[ty * RT + r][k + 4]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int d = 0; d < (DUAL ? 2 : 1); ++d) {
          const uint4 w = *reinterpret_cast<const uint4*>(&st.w[d][tx + TX * j][k]);
          const float wv[8] = {bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y), bf16_lo(w.z), bf16_hi(w.z), bf16_lo(w.w), bf16_hi(w.w)};
#pragma unroll
          for (int q = 0; q < 8; ++q)
#pragma unroll
            for (int r = 0; r < RT; ++r) {
              if (d == 0) acc[r][j] = fmaf(xv[r][q], wv[q], acc[r][j]);
              else acc2[r][j] = fmaf(xv[r][q], wv[q], acc2[r][j]);
            }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    const int row = it.row0 + ty * RT + i;
    if (row >= row_lim) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx + TX * j;
      if (n >= p.n) continue;
      const float bias = epi_has_bias<EPI>() ? bf(p.bias + (size_t)it.z * p.n + n) : 0.f;
      const float rate = EPI == kSEpiDecaySoft ? p.rate[n] : 0.f;
      const float v = epi_value<EPI>(p, acc[i][j], acc2[i][j], n, bias, rate);
      store_act(p.out, (long long)row * p.out_ld + (p.n_items ? 0 : it.z * p.out_zstride) + n, v, p.out_f32);
    }
  }
}

template <int T, int EPI>
int launch_f32_tile(const StackGemmArgs& a, cudaStream_t stream, bool pdl) {
  constexpr bool DUAL = EPI == kSEpiClampedGlu || EPI == kSEpiSiluGlu;
  constexpr int smem = kFStages * (int)sizeof(F32Stage<T, DUAL>);
  if (const int rc = allow_shared(stack_gemm_f32_kernel<T, EPI>, smem)) return rc;
  const int row_tiles = (a.rows + T - 1) / T;
  const long long items = a.n_items ? (long long)a.max_items * ((a.item_rows + T - 1) / T) : (long long)a.zcount * row_tiles;
  if (items < 1 || items > 65535) return -3;
  return launch_pdl(stack_gemm_f32_kernel<T, EPI>, dim3((a.n + T - 1) / T, (unsigned)items), dim3(T * 4), smem, stream, pdl, a, row_tiles);
}

// Tiles of 32 until tiles of 64 fill the SMs twice: below that the longest CTA is the time of the launch.
template <int EPI>
int launch_f32(const StackGemmArgs& a, cudaStream_t stream, bool pdl) {
  const long long rows = a.n_items ? (long long)a.max_items * a.item_rows : (long long)a.zcount * a.rows;
  const long long big = ((a.n + 63) / 64) * ((rows + 63) / 64);
  return big >= 2 * sm_count() || (rows + 31) / 32 > 32767 ? launch_f32_tile<64, EPI>(a, stream, pdl) : launch_f32_tile<32, EPI>(a, stream, pdl);
}

}  // namespace

extern "C" int nrt_stack_gemm_args_size() { return (int)sizeof(StackGemmArgs); }

// ntok: token rows per tile (64 to 256; two-product epilogues up to 192); the token map's box has that many rows.
extern "C" int nrt_stack_gemm(int epi, int ntok, const void* tmW, const void* tmW2, const void* tmX, const void* args,
                              int items_fastest, void* stream, int pdl) {
  CUtensorMap w, w2, x;
  memcpy(&w, tmW, sizeof(w));
  memcpy(&w2, tmW2 ? tmW2 : tmW, sizeof(w2));
  memcpy(&x, tmX, sizeof(x));
  StackGemmArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.n < 1 || a.k < 1 || a.rows < 1 || (a.n_items && a.item_rows != ntok)) return -3;
  if (((epi == kSEpiBias || epi == kSEpiDecaySoft || epi == kSEpiDecayExp) && !a.bias) || (epi == kSEpiDecaySoft && (!a.rate || a.zcount != 1))) return -3;
  if (epi == kSEpiTranspose && (a.out_f32 || a.out_ld % 8 || a.out_zstride % 8)) return -3;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
#define NRT_CASE(N, E) \
  if (ntok == N && epi == E) return launch<N, E>(w, w2, x, a, items_fastest, s, pdl != 0);
  NRT_CASE(64, kSEpiStore) NRT_CASE(128, kSEpiStore) NRT_CASE(192, kSEpiStore) NRT_CASE(256, kSEpiStore)
  NRT_CASE(64, kSEpiBias) NRT_CASE(128, kSEpiBias) NRT_CASE(192, kSEpiBias) NRT_CASE(256, kSEpiBias)
  NRT_CASE(64, kSEpiTranspose) NRT_CASE(256, kSEpiTranspose)
  NRT_CASE(64, kSEpiClampedGlu) NRT_CASE(128, kSEpiClampedGlu) NRT_CASE(192, kSEpiClampedGlu)
  NRT_CASE(64, kSEpiSiluGlu) NRT_CASE(128, kSEpiSiluGlu)
  NRT_CASE(64, kSEpiRelu2) NRT_CASE(128, kSEpiRelu2) NRT_CASE(192, kSEpiRelu2) NRT_CASE(256, kSEpiRelu2)
  NRT_CASE(64, kSEpiTanh) NRT_CASE(256, kSEpiTanh)
  NRT_CASE(64, kSEpiDecaySoft) NRT_CASE(256, kSEpiDecaySoft)
  NRT_CASE(64, kSEpiDecayExp) NRT_CASE(256, kSEpiDecayExp)
#undef NRT_CASE
  return -2;
}

extern "C" int nrt_stack_gemm_f32(int epi, const void* args, void* stream, int pdl) {
  StackGemmArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.n < 1 || a.k < 1 || a.rows < 1) return -3;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch (epi) {
    case kSEpiStore: return launch_f32<kSEpiStore>(a, s, pdl != 0);
    case kSEpiBias: return launch_f32<kSEpiBias>(a, s, pdl != 0);
    case kSEpiClampedGlu: return launch_f32<kSEpiClampedGlu>(a, s, pdl != 0);
    case kSEpiSiluGlu: return launch_f32<kSEpiSiluGlu>(a, s, pdl != 0);
    case kSEpiRelu2: return launch_f32<kSEpiRelu2>(a, s, pdl != 0);
    case kSEpiTanh: return launch_f32<kSEpiTanh>(a, s, pdl != 0);
    case kSEpiDecaySoft: return launch_f32<kSEpiDecaySoft>(a, s, pdl != 0);
    case kSEpiDecayExp: return launch_f32<kSEpiDecayExp>(a, s, pdl != 0);
  }
  return -2;
}
