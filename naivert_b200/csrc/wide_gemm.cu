// Chunk GEMM for prefill: the same swapped-operand tcgen05 engine as gemm.cuh with 64 token columns per tile.
//
// The 16-column engine re-reads every 16 KiB weight tile from L2 once per 16 tokens, which bounds a
// prefill chunk by L2 -> SM bandwidth (~18 KiB per 0.5 MFLOP).  Here a tile is 128 output features x
// 64 token rows of one work item (64 consecutive rows of the token operand that share one weight group: a row
// group of a prefill chunk, or a padded expert segment of the expert-parallel receive buffer), so a weight
// tile feeds four times the math; one CTA per SM walks the tiles.
//   warp 0     : TMA producer (weights 128 x 128 B, tokens 64 x 128 B, 128-byte swizzle, no multicast)
//   warp 1     : TMEM allocator + UMMA issuer (M = 128, N = 64; kind::f8f6f4 or kind::f16)
//   warps 2..17: epilogue; thread = output feature x a quarter (16) of the token columns: four warps per TMEM lane
//                quadrant, so that a thread has the registers to fetch the next accumulator while it adds the last one
// Block-scaled e4m3: one fresh TMEM accumulator per 128-wide K block (a ring of pairs), scaled by weight-block x
// activation-block scale and promoted in fp32 registers in ascending K order (the same arithmetic as the
// 16-column engine, so both produce identical values).  Scales of the item's rows times those of the weights are
// put into shared memory once per tile (after the first accumulator is ready, i.e. after the producer has seen
// the rows arrive).
// Epilogues: fp32 / bf16 store, SiLU(gate) * up with e4m3 re-quantisation, and the expert-parallel return
// (tagged bf16 pairs into the token owner's combine slots in peer memory).
//
// Reference counterpart: DeepGEMM contiguous grouped fp8 GEMM and cuBLAS bf16 GEMMs of the reference's prefill
// (naivert/kernels/naive_n0p5/prefill.py:1044-1146).
#include "gemm.cuh"
#include "launch.hpp"

#include <string.h>

using namespace nrt;

namespace {

constexpr int kWTok = 64;
constexpr int kWBTileBytes = kWTok * kKBytes;    // 8 KiB
constexpr int kMaxSmem = 227 * 1024;
// Row of a K block in the table of scales: lanes that hold consecutive K blocks of a token write to eight banks (to one at 64).
constexpr int kScaleLd = kWTok + 4;

template <bool FP8, bool DUAL>
struct WideCfg {
  static constexpr int kStageBytes = (DUAL ? 2 : 1) * kATileBytes + kWBTileBytes;
  static constexpr int kMaxStages = DUAL ? 4 : 6;
  static constexpr int kAccCols = DUAL ? 2 * kWTok : kWTok;
  // e4m3: accumulators change hands in pairs (two K blocks); bf16: one accumulator per tile, two tiles in flight
  static constexpr int kPair = FP8 ? 2 : 1;
  static constexpr int kAccBufs = FP8 ? 512 / (2 * kAccCols) : 2;
  static constexpr int kTmemCols = kAccCols * kPair * kAccBufs;    // 128 or 512
  static constexpr int kMaxKBlocks = 128;                          // K <= 16384 for e4m3
  static constexpr int kFixedBytes = 1024 /*align*/ + 2048 /*barriers + scratch*/;
  static constexpr int scale_bytes(int kb_total) { return FP8 ? (DUAL ? 2 : 1) * kb_total * kScaleLd * 4 : 0; }
  // as many stages as the scales leave room for: all of them, three of two products with K above 15,360
  static constexpr int stages(int kb_total) {
    const int fit = (kMaxSmem - kFixedBytes - scale_bytes(kb_total)) / kStageBytes;
    return fit < kMaxStages ? fit : kMaxStages;
  }
  static constexpr int smem_bytes(int kb_total) { return stages(kb_total) * kStageBytes + kFixedBytes + scale_bytes(kb_total); }
};

struct WideTail {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t acc_full[4];
  uint64_t acc_empty[4];
  uint32_t tmem_base;
  uint32_t pad;
  float red[4][kWTok];
};

constexpr int kWEpiWarps = 16, kWThreads = 64 + 32 * kWEpiWarps;
constexpr int kWCols = kWTok / (kWEpiWarps / 4);      // token columns per epilogue thread
static_assert(kWCols == 16, "one TMEM load per accumulator");

// two fp32 values in one register pair: one instruction for both, each rounded as by its scalar form
__device__ __forceinline__ uint64_t pack2u(uint32_t a, uint32_t b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float a, float b) { return pack2u(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// The wait for TMEM loads names their registers, so that nothing which reads them can be moved in front of it.
__device__ __forceinline__ void tmem_landed(uint32_t (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                 "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])::"memory");
}

// Persistent CTAs (one per SM) walk the (feature tile, item) work list with a fixed stride, so the TMA producer
// and the MMA issuer run ahead into the next tile while the epilogue warps still store the previous one; the
// stage ring and the accumulator ring simply continue across tiles.
// order 0: feature tiles vary fastest over the work list (consecutive CTAs share the item's token tile: grouped
// experts; or a weight matrix that fits the L2); order 1: items vary fastest (consecutive CTAs share a weight
// tile: one big weight matrix that must stream from HBM only once per chunk).
template <bool FP8, bool DUAL, int EPI>
__global__ void __launch_bounds__(kWThreads, 1)
wide_gemm_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                 const __grid_constant__ CUtensorMap tmB, const GemmArgs p, const int order, const int n_tiles, const int items,
                 const int stages) {
  using Cfg = WideCfg<FP8, DUAL>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  WideTail* tail = reinterpret_cast<WideTail*>(smem + stages * Cfg::kStageBytes);
  float* as_s = reinterpret_cast<float*>(smem + stages * Cfg::kStageBytes + 2048);   // [product][kb][kScaleLd]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kElemsPerStage = FP8 ? 128 : 64;
  const int kb_total = p.k_total / kElemsPerStage;

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) { mbar_init(&tail->full[i], 1); mbar_init(&tail->empty[i], 1); }
    for (int i = 0; i < Cfg::kAccBufs; ++i) { mbar_init(&tail->acc_full[i], 1); mbar_init(&tail->acc_empty[i], kWEpiWarps); }
    mbar_fence_init();
    tma_prefetch_desc(&tmA0);
    tma_prefetch_desc(&tmB);
    if (DUAL) tma_prefetch_desc(&tmA1);
  }
  if (warp == 1) { tmem_alloc(&tail->tmem_base, Cfg::kTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tail->tmem_base;
  griddep_wait();
  griddep_launch();

  const int na = min(min(*p.n_active, p.max_slots), items);
  const int total = n_tiles * items;
  // every role walks the same list: work w -> (feature tile, item); items >= na are skipped by all roles alike
#define NRT_WIDE_DECODE(w, n_tile, item)                               \
  const int n_tile = order ? (w) / items : (w) % n_tiles;              \
  const int item = order ? (w) % items : (w) / n_tiles;

  if (warp == 0) {
    if (elect_one()) {
      bool ready = !(p.fab.ag_call >= 0 && p.fab.tp > 1);
      bool ok = true;
      int st = 0;                                              // stage, over all tiles of this CTA
      uint32_t phase = 1;
      bool first = true;                                       // the ring has not been filled once
      for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
        NRT_WIDE_DECODE(w, n_tile, item)
        if (item >= na) continue;
        const int z = p.active_ids[item];
        const int brow = p.row_offsets ? p.row_offsets[item] : item * kWTok;
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!first && !mbar_wait(&tail->empty[st], phase, p.status, kSiteStageEmpty | st)) { ok = false; break; }
          uint8_t* sa = smem + st * Cfg::kStageBytes;
          const int kx = kb * kElemsPerStage;
          mbar_expect_tx(&tail->full[st], Cfg::kStageBytes);
          tma_load_3d(sa, &tmA0, &tail->full[st], kx, n_tile * kTileN, z);
          if (DUAL) tma_load_3d(sa + kATileBytes, &tmA1, &tail->full[st], kx, n_tile * kTileN, z);
          if (!ready) {
            // expert-parallel dispatch: the rows of every source rank must have landed before the first token tile
            const uint32_t tag = (*p.fab.epoch) * 1024u + (uint32_t)p.fab.ag_call + 1u;
            bool all = true;
            for (int s = 0; s < p.fab.tp && all; ++s) {
              uint32_t v;
              all = wait_tagged(p.fab.ag_flags + s, tag, v, globaltimer() + p.fab.timeout_ns, p.status, kSiteMailbox | 0x60 | s);
            }
            if (!all) { ok = false; break; }
            asm volatile("fence.acq_rel.sys;" ::: "memory");
            asm volatile("fence.proxy.async;" ::: "memory");
            ready = true;
          }
          tma_load_2d(sa + (DUAL ? 2 : 1) * kATileBytes, &tmB, &tail->full[st], kx, brow);
          if (++st == stages) { st = 0; phase ^= 1; first = false; }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // One thread runs this loop for every K block, so it is kept short: descriptors by addition, counters instead of remainders.
      constexpr uint32_t idesc = umma_idesc(FP8 ? 0u : 1u, kTileN, kWTok);
      const uint64_t desc = umma_desc_sw128(smem_u32(smem));
      bool ok = true;
      int st = 0, buf = 0, uses = 0;                           // stage, accumulator, accumulators handed out
      uint32_t phase = 0, acc_phase = 1;
      for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
        NRT_WIDE_DECODE(w, n_tile, item)
        (void)n_tile;
        if (item >= na) continue;
        for (int kb = 0; kb < kb_total; ++kb) {
          if (FP8 ? (kb & 1) == 0 : kb == 0) {
            if (uses >= Cfg::kAccBufs && !mbar_wait(&tail->acc_empty[buf], acc_phase, p.status, kSiteAccEmpty | buf)) { ok = false; break; }
            ++uses;
          }
          if (!mbar_wait(&tail->full[st], phase, p.status, kSiteTmaFull | st)) { ok = false; break; }
          tc_fence_after();
          const uint64_t da0 = desc + (uint32_t)(st * Cfg::kStageBytes >> 4);
          const uint64_t da1 = da0 + (kATileBytes >> 4), db = da0 + ((DUAL ? 2 : 1) * kATileBytes >> 4);
          const uint32_t d0 = tmem + (buf * Cfg::kPair + (FP8 ? kb & 1 : 0)) * Cfg::kAccCols;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t acc = FP8 ? (j > 0) : (kb > 0 || j > 0);
            if (FP8) {
              umma_f8(d0, da0 + 2 * j, db + 2 * j, idesc, acc);
              if (DUAL) umma_f8(d0 + kWTok, da1 + 2 * j, db + 2 * j, idesc, acc);
            } else {
              umma_bf16(d0, da0 + 2 * j, db + 2 * j, idesc, acc);
            }
          }
          umma_commit(&tail->empty[st]);
          if (kb == kb_total - 1 || (FP8 && (kb & 1))) {
            umma_commit(&tail->acc_full[buf]);
            if (++buf == Cfg::kAccBufs) { buf = 0; acc_phase ^= 1; }
          }
          if (++st == stages) { st = 0; phase ^= 1; }
        }
      }
    }
  } else {
    // e4m3: every K block is promoted - commit, load from TMEM, scale, add.  Per K block: o_proj (K 8192, 2048 rows, weights in L2)
    // 382 ns with accumulators in pairs, 500 ns with one accumulator per hand-over and eight warps that finished one block before they
    // asked for the next; gate and up of 256 experts of ~64 rows 767 ns (4.2 TB/s of weights), 1079 ns.  What bounds a block now is
    // several things that overlap: without additions, TMEM loads and products its copies alone take 0.7 of it (o_proj) to 0.9 (experts,
    // which stream from HBM), without the products 0.83, without the additions 0.88; the tensor cores are busy 29 %.
    const int quad = warp & 3;                       // TMEM lane quadrant this warp may read
    const int c0 = ((warp - 2) >> 2) * kWCols;       // first of its token columns
    const int row = quad * 32 + lane;                // feature within the tile
    const int e = threadIdx.x - 64;                  // 0..511 among the epilogue threads
    const uint32_t lane_addr = tmem + (uint32_t(quad * 32) << 16) + c0;
    const int nt_count = p.n_total / kTileN;
    bool ok = true;
    int v = 0, t = 0;                                // pairs of K blocks and tiles so far
    constexpr int kBars = FP8 ? (EPI == kEpiSiluQuant ? 4 : 2) : 0;       // barriers of a tile
    int w = blockIdx.x, owed = 0;                    // owed: of tile w when this warp's wait gave up there
    for (; w < total; w += gridDim.x) {
      NRT_WIDE_DECODE(w, n_tile, item)
      if (item >= na) continue;
      const int z = p.active_ids[item];
      const int brow = p.row_offsets ? p.row_offsets[item] : item * kWTok;
      const int n = n_tile * kTileN + row;
      float acc0[kWCols];
      float acc1[DUAL ? kWCols : 1];
      if (FP8) {
        uint32_t b0[16], b1[16];
        uint64_t sum0[kWCols / 2], sum1[DUAL ? kWCols / 2 : 1];       // two columns each
#pragma unroll
        for (int r = 0; r < kWCols / 2; ++r) {
          sum0[r] = 0;
          if (DUAL) sum1[DUAL ? r : 0] = 0;
        }
        const float* ws0 = p.w_scale0 + ((size_t)z * nt_count + n_tile) * kb_total;
        const float* ws1 = DUAL ? p.w_scale1 + ((size_t)z * nt_count + n_tile) * kb_total : nullptr;
        // wait for the pair of K blocks from `kb` on and request the first's accumulator
        auto ask = [&](int kb) {
          const int use = v + (kb >> 1), buf = use % Cfg::kAccBufs;
          if (!__all_sync(0xffffffffu, mbar_wait(&tail->acc_full[buf], (use / Cfg::kAccBufs) & 1, p.status, kSiteAccFull | buf))) return false;
          tc_fence_after();
          tmem_ld16_nowait(lane_addr + buf * 2 * Cfg::kAccCols, b0);
          return true;
        };
        auto acc_of = [&](int kb) { return lane_addr + ((v + (kb >> 1)) % Cfg::kAccBufs * 2 + (kb & 1)) * Cfg::kAccCols; };
        auto give_back = [&](int kb) {                                // the warp's values are in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tail->acc_empty[(v + (kb >> 1)) % Cfg::kAccBufs]);
        };
        auto add = [&](uint64_t* sum, const uint32_t (&b)[16], int kb) {                // kb: row of the table
          const float4* sc4 = reinterpret_cast<const float4*>(as_s + kb * kScaleLd + c0);
#pragma unroll
          for (int q = 0; q < kWCols / 4; ++q) {
            const float4 s = sc4[q];
            sum[q * 2] = fma2(pack2u(b[q * 4], b[q * 4 + 1]), pack2(s.x, s.y), sum[q * 2]);
            sum[q * 2 + 1] = fma2(pack2u(b[q * 4 + 2], b[q * 4 + 3]), pack2(s.z, s.w), sum[q * 2 + 1]);
          }
        };
        ok = ask(0);
        if (!ok) { owed = kBars; break; }
        // Scales of the item's 64 rows times the weights', once per tile instead of with every column of every block (the same product):
        // o_proj of 2048 rows 166 -> 159 us, gate and up of 256 experts of 64 rows 752 -> 735 us, down 389 -> 371 us.  Transposed to
        // [K block][row]; the rows' are read coherently after the first accumulator is ready (in the expert-parallel path peers wrote
        // them shortly before).  The first barrier keeps a fast warp from overwriting the table while a slow one still reads the previous
        // tile's scales.
        asm volatile("bar.sync 1, 512;" ::: "memory");
        const float* as = p.a_scale + (size_t)brow * kb_total;
        for (int i = e; i < kWTok * kb_total; i += 32 * kWEpiWarps) {
          const int r = i / kb_total, k = i - r * kb_total;
          const float s = __ldcv(as + i);
          as_s[k * kScaleLd + r] = s * __ldg(ws0 + k);
          if (DUAL) as_s[(kb_total + k) * kScaleLd + r] = s * __ldg(ws1 + k);
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
        // one accumulator is on its way while the one before it is added
        for (int kb = 0; kb < kb_total; kb += 2) {
          const bool two = kb + 1 < kb_total, more = kb + 2 < kb_total;
          tmem_landed(b0);
          if (DUAL) {
            tmem_ld16_nowait(acc_of(kb) + kWTok, b1);
            add(sum0, b0, kb);
            tmem_landed(b1);
            if (two) {
              tmem_ld16_nowait(acc_of(kb + 1), b0);
              add(sum1, b1, kb_total + kb);
              tmem_landed(b0);
              tmem_ld16_nowait(acc_of(kb + 1) + kWTok, b1);
              add(sum0, b0, kb + 1);
              tmem_landed(b1);
            }
            give_back(kb);
            if (more && !(ok = ask(kb + 2))) break;
            add(sum1, b1, kb_total + (two ? kb + 1 : kb));
          } else {
            if (two) {
              tmem_ld16_nowait(acc_of(kb + 1), b1);
              add(sum0, b0, kb);
              tmem_landed(b1);
              give_back(kb);
              if (more && !(ok = ask(kb + 2))) break;
              add(sum0, b1, kb + 1);
            } else {
              give_back(kb);
              add(sum0, b0, kb);
            }
          }
        }
        if (!ok) { owed = kBars - 2; break; }
        v += (kb_total + 1) / 2;
#pragma unroll
        for (int r = 0; r < kWCols / 2; ++r) {
          unpack2(sum0[r], acc0[2 * r], acc0[2 * r + 1]);
          if (DUAL) unpack2(sum1[DUAL ? r : 0], acc1[DUAL ? 2 * r : 0], acc1[DUAL ? 2 * r + 1 : 0]);
        }
      } else {
        const int buf = t % Cfg::kAccBufs;
        if (!__all_sync(0xffffffffu, mbar_wait(&tail->acc_full[buf], (t / Cfg::kAccBufs) & 1, p.status, kSiteAccFull | buf))) { ok = false; break; }
        tc_fence_after();
        uint32_t v0[16];
        tmem_ld16_nowait(lane_addr + buf * Cfg::kAccCols, v0);
        tmem_landed(v0);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tail->acc_empty[buf]);
#pragma unroll
        for (int r = 0; r < kWCols; ++r) acc0[r] = __uint_as_float(v0[r]);
      }
      ++t;

      const bool live = n < p.n_total;
      const size_t out_row0 = (size_t)brow + c0;
      if (EPI == kEpiStoreF32) {
        if (live)
#pragma unroll
          for (int r = 0; r < kWCols; ++r) p.out_f32[(out_row0 + r) * p.ld_out + n] = acc0[r] * p.out_scale;
      } else if (EPI == kEpiStoreBF16) {
        if (live)
#pragma unroll
          for (int r = 0; r < kWCols; ++r) p.out_bf16[(out_row0 + r) * p.ld_out + n] = __float2bfloat16_rn(acc0[r] * p.out_scale);
      } else if (EPI == kEpiSiluQuant) {
#pragma unroll
        for (int r = 0; r < kWCols; ++r) {
          acc0[r] = silu(acc0[r]) * acc1[DUAL ? r : 0];
          float m = fabsf(acc0[r]);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
          if (lane == 0) tail->red[quad][c0 + r] = m;
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
#pragma unroll
        for (int r = 0; r < kWCols; ++r) {
          const int c = c0 + r;
          const float am = fmaxf(fmaxf(tail->red[0][c], tail->red[1][c]), fmaxf(tail->red[2][c], tail->red[3][c]));
          const float s = pow2_scale(am);
          const __nv_fp8_e4m3 q(acc0[r] / s);
          p.out_q[(out_row0 + r) * p.n_total + n] = *reinterpret_cast<const uint8_t*>(&q);
          if (row == 0) p.out_qscale[(out_row0 + r) * nt_count + n_tile] = s;
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");      // the amax scratch is reused by the next tile
      } else if (EPI == kEpiReturn) {
        const uint32_t dtag = (*p.fab.epoch) * 1024u + (uint32_t)p.ep_dispatch_call + 1u;
        const uint32_t rtag = (*p.fab.epoch) * 1024u + (uint32_t)p.ep_return_call + 1u;
        const int words = p.n_total / 2;
#pragma unroll
        for (int r = 0; r < kWCols; ++r) {
          const int4 m = p.ep_meta[out_row0 + r];
          const float other = __shfl_down_sync(0xffffffffu, acc0[r], 1);
          if ((uint32_t)m.w == dtag && (lane & 1) == 0) {
            uint64_t* dst = p.ep_combine[m.x] + ((size_t)(m.y * p.ep_top_k + m.z)) * words + (n >> 1);
            st_tagged(dst, rtag, pack_bf16x2(acc0[r], other));
          }
        }
      }
    }
    // A warp whose wait gave up (its limit, or a fault recorded elsewhere on the device meanwhile) still takes the barriers of the tiles it
    // leaves: others may have seen the same accumulator in time, and would wait for it for good.
    if (FP8 && !ok) {
      for (;;) {
        for (int i = 0; i < owed; ++i) asm volatile("bar.sync 1, 512;" ::: "memory");
        if ((w += gridDim.x) >= total) break;
        NRT_WIDE_DECODE(w, n_tile, item)
        (void)n_tile;
        owed = item < na ? kBars : 0;
      }
    }
  }
#undef NRT_WIDE_DECODE

  drain_on_error(p.status);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, Cfg::kTmemCols); }
}

template <bool FP8, bool DUAL, int EPI>
int launch_wide(const CUtensorMap& a0, const CUtensorMap& a1, const CUtensorMap& b, const GemmArgs& args, int n_tiles, int items,
                int order, cudaStream_t stream, int pdl) {
  using Cfg = WideCfg<FP8, DUAL>;
  auto* kern = wide_gemm_kernel<FP8, DUAL, EPI>;
  if (const int rc = allow_shared(kern, kMaxSmem)) return rc;
  const int kb_total = args.k_total / 128;
  if (FP8 && kb_total > Cfg::kMaxKBlocks) return -6;                  // scale table size
  if (n_tiles < 1 || items < 1 || (long long)n_tiles * items > 0x7fffffffLL) return -3;
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms < 1) sms = 148;
  }
  const int total = n_tiles * items;
  const dim3 grid(total < sms ? total : sms, 1, 1);                    // persistent: one CTA per SM
  return launch_pdl(kern, grid, dim3(kWThreads, 1, 1), Cfg::smem_bytes(kb_total), stream, pdl != 0, a0, a1, b, args, order, n_tiles, items,
                    Cfg::stages(kb_total));
}

}  // namespace

extern "C" int nrt_wide_tok() { return kWTok; }

// variant = fp8 | dual<<1 | epi<<2 (item mode only; items of 64 rows).  The token tensor map must have 64-row
// boxes.  order: 0 = feature tiles vary fastest over the grid, 1 = items vary fastest.
extern "C" int nrt_wide_gemm_launch(int variant, const void* tmA0, const void* tmA1, const void* tmB, const void* args,
                                    int n_tiles, int items, int order, void* stream, int pdl) {
  CUtensorMap a0, a1, b;
  memcpy(&a0, tmA0, sizeof(a0));
  memcpy(&a1, tmA1 ? tmA1 : tmA0, sizeof(a1));
  memcpy(&b, tmB, sizeof(b));
  GemmArgs g;
  memcpy(&g, args, sizeof(g));
  if (!g.n_active || !g.active_ids) return -3;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
#define NRT_WCASE(FP8, DUAL, EPI)                    \
  case ((FP8) | ((DUAL) << 1) | ((EPI) << 2)):      \
    return launch_wide<(FP8) != 0, (DUAL) != 0, EPI>(a0, a1, b, g, n_tiles, items, order, s, pdl);
  switch (variant & 31) {
    NRT_WCASE(1, 1, kEpiSiluQuant)
    NRT_WCASE(1, 0, kEpiReturn)
    NRT_WCASE(1, 0, kEpiStoreBF16)
    // bf16 stores: for callers of this entry (64-row items with a row offset each); prompts multiply bf16 rows in stack_gemm.cu
    NRT_WCASE(0, 0, kEpiStoreF32)
    NRT_WCASE(0, 0, kEpiStoreBF16)
    default:
      return -2;
  }
#undef NRT_WCASE
}
