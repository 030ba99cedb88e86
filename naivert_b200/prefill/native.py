"""Chunked native prefill: whole chunks of prompt rows go through every layer in one pass.

A chunk of ``R`` rows (a multiple of 16, up to ``chunk``) is processed layer by layer with the same
kernels and caches as the decode/verify step, launched over row groups:

    RMSNorm -> q/k/v(/indexer) projection (tcgen05, tiles of up to 256 rows) -> RoPE / KV append /
    indexer keys -> [tcgen05 indexer sweep per row group -> exact top-k per row] -> row attention ->
    o_proj partials -> tensor-parallel reduction -> MoE -> draft feature ingest at the tap layers

On one GPU consecutive chunks of a prompt form a span (up to ``SPAN_ROWS`` rows): a layer's attention and routing take them in turn,
its experts together.

Parallel layout (``tp`` ranks, one process per GPU):

* attention is tensor parallel (heads split, KV caches of this rank's heads), the partial o_proj
  outputs are reduced with NCCL: all-reduce for dense layers, reduce-scatter for MoE layers;
* with expert-parallel weights (``ep_weights``) the MoE rows are sequence parallel (``R / tp`` rows per
  rank) and the experts are whole and split over the ranks: count / dispatch / grouped GEMMs / return /
  combine run inside the kernels of ``EPMoE`` over peer memory, then the residual rows are all-gathered;
* without them every rank runs all rows through its intermediate slice of every expert (the same
  grouped kernels on a single-rank exchange) and the partial sums are all-reduced.

The caches it fills are the decode caches, so decoding continues from the chunk boundary
(``SpeculativeRound.initialize(start_pos=...)`` replays what is left of the prompt).

Parity: ``NativePrefill`` (naivert/prefill/native/executor.py: chunk body :479-537, ``run``,
``warm_chunks``, ``resume_from_decode``, ``close``), ``TPMoE`` (naivert/prefill/native/moe_tp.py),
``DraftFeaturePrefillExecutor`` (naivert/prefill/draft_features.py:24-103), chunk planning
(naivert/prefill/planning.py).
"""
from __future__ import annotations

import os
from contextlib import contextmanager
from dataclasses import dataclass
from typing import Dict, List, Optional

import torch
import torch.distributed as dist

from ..models.spec import FULL_DSA, ModelSpec
from ..ops import kernels as K
from ..ops import stack_kernels as S
from ..runtime.target import LocalFabric, TargetRuntime
from .ep_moe import EPMoE, EPWeights
from .stack import StackPrefill

ROWS = K.K_TOK
SPAN_ROWS = 8192          # rows whose experts run together: 256 experts of top 8 see 256 rows each


@dataclass
class Chunk:
    pos0: int
    rows: int


def plan_chunks(start: int, end: int, chunk: int, quantum: int) -> List[Chunk]:
    """Split positions [start, end) into chunks of at most ``chunk`` rows; every chunk is a multiple of
    ``quantum`` rows, the remainder (< quantum) is left to the caller (prompt replay).
    Parity: naivert/prefill/planning.py (bucketed chunk plan)."""
    if chunk % quantum:
        raise ValueError(f"chunk {chunk} is not a multiple of {quantum}")
    out, p = [], start
    while end - p >= quantum:
        r = min(chunk, (end - p) // quantum * quantum)
        out.append(Chunk(p, r))
        p += r
    return out


class NativePrefill:
    V_BF16_F32 = K.gemm_variant(False, False, K.EPI_STORE_F32, K.GROUP_ITEM)
    V_BF16_BF16 = K.gemm_variant(False, False, K.EPI_STORE_BF16, K.GROUP_ITEM)
    V_FP8_BF16 = K.gemm_variant(True, False, K.EPI_STORE_BF16, K.GROUP_ITEM)
    V_FP8_GU = K.gemm_variant(True, True, K.EPI_SILU_QUANT, K.GROUP_ITEM)

    def __init__(self, spec: ModelSpec, target: TargetRuntime, draft=None, chunk: int = 4096,
                 ep_weights: Optional[list] = None, group=None):
        t = target
        self.spec, self.t, self.draft, self.group = spec, target, draft, group
        self.tp, self.rank, self.dev = t.fab.tp, t.fab.rank, t.dev
        if t.tp != t.fab.tp:
            raise ValueError("shape emulation has no peers to reduce with")
        self.ep = ep_weights is not None and self.tp > 1
        self.quantum = ROWS * (self.tp if self.ep else 1)
        if chunk % self.quantum or chunk < self.quantum:
            raise ValueError(f"chunk must be a multiple of {self.quantum}")
        if t.prefill_chunk < chunk:
            raise ValueError("the target's sliding-window rings were not sized for this chunk (prefill_chunk)")
        if FULL_DSA in spec.layer_kinds and not t.use_sweep:
            raise ValueError("the chunked indexer needs the tcgen05 sweep geometry (16 heads x 128)")
        self.C = C = chunk
        # 64-column chunk GEMM (a weight tile feeds 64 rows) unless NAIVERT_PREFILL_WIDE=0 or the chunk is not a
        # multiple of 64 rows; otherwise the step engine's 16-column tiles in item mode
        self.wide = os.environ.get("NAIVERT_PREFILL_WIDE", "1") == "1" and chunk % K.WIDE_TOK == 0
        self.step = K.WIDE_TOK if self.wide else ROWS
        s, dev = spec, self.dev
        H = s.hidden
        bf, f32, i32, u8 = torch.bfloat16, torch.float32, torch.int32, torch.uint8
        self.xn = torch.zeros(C, H, dtype=bf, device=dev)
        self.x8 = torch.zeros(C, H, dtype=u8, device=dev)
        self.xs = torch.ones(C, H // 128, dtype=f32, device=dev)
        self.part = torch.zeros(C, H, dtype=bf, device=dev)
        self.map_x8 = K.act_tmap(self.x8, self.step)
        self._bf16: Dict[tuple, tuple] = {}               # (weight, rows) -> argument block, tensor maps of the rows by tile height
        self.qkv = torch.zeros(C, t.qkv.shape[1], dtype=f32, device=dev)
        self.q = torch.zeros(C, t.q.shape[1], t.q.shape[2], dtype=bf, device=dev)
        self.o8 = torch.zeros(C, t.o8.shape[1], dtype=u8, device=dev)
        self.os = torch.ones(C, t.os.shape[1], dtype=f32, device=dev)
        self.map_o8 = K.act_tmap(self.o8, self.step)
        self.items = C // self.step
        self.row_offsets = (torch.arange(self.items, dtype=i32, device=dev) * self.step).contiguous()
        self.zero_ids = torch.zeros(self.items, dtype=i32, device=dev)
        self.n_items = torch.arange(self.items + 1, dtype=i32, device=dev)         # work items of a launch, by address
        ix = s.indexer
        if FULL_DSA in s.layer_kinds:
            self.iq8 = torch.zeros(C * ix.head_count, ix.head_dim, dtype=u8, device=dev)
            self.ihw = torch.zeros(C, ix.head_count, dtype=f32, device=dev)
            self.idx_logits = torch.zeros(C, t.capacity, dtype=f32, device=dev)
            self.sel = torch.zeros(C, ix.top_k, dtype=i32, device=dev)
            # the indexer is replicated, so ranks split the query rows of a chunk for the sweep and the top-k and
            # all-gather the selection lists (NAIVERT_PREFILL_SHARD_INDEX=0: every rank selects for every row)
            self.shard_index = self.tp > 1 and os.environ.get("NAIVERT_PREFILL_SHARD_INDEX", "1") == "1"
            self.sel_local = torch.zeros(C // self.tp, ix.top_k, dtype=i32, device=dev) if self.shard_index else None
            self.topk_state = torch.zeros(C * K.topk_grid_state_bytes() // 4, dtype=i32, device=dev) if t.topk_grid else None
        if s.dense_layer_count:
            Id = s.dense_inter_local(self.tp)
            self.yd8 = torch.zeros(C, Id, dtype=u8, device=dev)
            self.yds = torch.ones(C, Id // 128, dtype=f32, device=dev)
            self.map_yd8 = K.act_tmap(self.yd8, self.step)
        # ---- MoE
        rt = s.routing
        self.T = C // self.tp if self.ep else C                            # rows a rank routes
        self.scores = torch.zeros(self.T, rt.expert_count, dtype=f32, device=dev)
        self.tickets = torch.zeros(-(-self.T // ROWS), dtype=i32, device=dev)
        self.xl = torch.zeros(self.T, H, dtype=bf, device=dev)             # this rank's rows between scatter and gather
        self.rs = torch.zeros(self.T, H, dtype=bf, device=dev)
        self.zeros = torch.zeros(self.T, H, dtype=bf, device=dev) if (self.tp > 1 and not self.ep) else None
        has_moe = any("gate" in d for d in t.layers)
        self.moe_fab = t.fab if (self.ep or self.tp == 1) else LocalFabric(dev)
        self.moe: Optional[EPMoE] = None
        self.moe_w: List[Optional[EPWeights]] = []
        # Rows of several chunks go through a layer's experts together on one GPU: its weights are read once for all of them, and fewer
        # segments of 64 are padding.  16,001 tokens at 2048 rows a chunk, spans of one / four chunks: gate and up 42.3 -> 31.3 ms, down 24.4 -> 19.5 ms.
        self.span_limit = max(C, SPAN_ROWS // C * C) if has_moe and self.tp == 1 else C
        self._size_span(C)
        if has_moe:
            for L, d in enumerate(t.layers):
                if "gate" not in d:
                    self.moe_w.append(None)
                elif self.ep:
                    w = ep_weights[L]
                    self.moe_w.append(EPWeights(*({"w": w[n]["w"].to(dev), "s": w[n]["s"].to(dev)} for n in ("gate", "up", "down"))))
                else:
                    self.moe_w.append(EPWeights(*({"w": d[n].w, "s": d[n].s} for n in ("gate", "up", "down"))))
        # ---- draft feature ingest
        if draft is not None:
            Hd = s.draft.hidden
            self.dh = torch.zeros(C, Hd, dtype=bf, device=dev)
            self.dxn = torch.zeros(C, Hd, dtype=bf, device=dev)
            self.draw = torch.zeros(C, draft.wkv.shape[0], dtype=f32, device=dev)
        self.phases: dict = {}
        # grouped-head attention kernel; NAIVERT_PREFILL_GROUP_ATTN=0 keeps the per-head row kernel of the step
        # path (bitwise-comparable with replay)
        self.group_attn = os.environ.get("NAIVERT_PREFILL_GROUP_ATTN", "1") == "1"
        self.profile = False                         # per-stage CUDA-event timing (adds an event pair per stage)
        self._timed: Dict[str, list] = {}
        self._build_args()

    def _size_span(self, P: int) -> None:
        """Buffers of a span of ``P`` rows (whole chunks); an allocation that fails leaves the present ones."""
        s, t, C, dev, rt = self.spec, self.t, self.C, self.dev, self.spec.routing
        bf, f32, i32, H, T = torch.bfloat16, torch.float32, torch.int32, self.spec.hidden, P // self.tp if self.ep else P
        new = {
            "pos": torch.zeros(P // C, 4, dtype=i32, device=dev),           # [c][0] = position of chunk c's row 0
            "_steps": torch.arange(P // C, dtype=i32, device=dev)[:, None].expand(-1, 4) * C,
            "tokens": torch.zeros(P, dtype=i32, device=dev), "x": torch.zeros(P, H, dtype=bf, device=dev),
            "rope": {k: torch.zeros(P, v.shape[1], 2, dtype=f32, device=dev) for k, v in t.rope.items()},
            "idx_rope": torch.zeros(P, t.idx_rope.shape[1], 2, dtype=f32, device=dev),
            "topk_ids": torch.zeros(T, rt.top_k, dtype=i32, device=dev), "topk_p": torch.zeros(T, rt.top_k, dtype=f32, device=dev)}
        if any("gate" in d for d in t.layers):
            inter = rt.intermediate if self.ep else s.expert_inter_local(self.tp)
            new["moe"] = EPMoE(self.moe_fab, H, inter, rt.expert_count, rt.top_k, T, eps=s.norm_eps, item_rows=self.step)
        if self.draft is not None:
            kf = self.draft.kf
            new["feats"] = torch.zeros(P, max(1, len(s.draft.target_layer_ids)) * H, dtype=bf, device=dev)
            new["taps"] = new["feats"][:, self.rank * kf:(self.rank + 1) * kf]
            new["drope"] = torch.zeros(P, s.draft.head_dim // 2, 2, dtype=f32, device=dev)
        for name, v in new.items():
            setattr(self, name, v)
        self.span = P
        self._bf16.clear()

    def _fit_span(self, n: int) -> None:
        """Spans for ``n`` rows as far as the limit and the memory go: what a span needs beyond a chunk is taken when a prompt first asks
        for it, and without the memory chunks go on one by one."""
        P = min(self.span_limit, -(-n // self.C) * self.C)
        if P > self.span:
            torch.cuda.synchronize(self.dev)              # earlier calls may still use the buffers that go, on any stream
        while P > self.span:
            try:
                self._size_span(P)
            except torch.OutOfMemoryError:
                P -= self.C
                self.span_limit = P

    def _gemm(self, variant, a0, a1, b, args, n_tiles, items, pdl=False):
        """Plain projections share one weight matrix over all items.  A matrix that fits the L2 (126 MB) stays
        resident while feature tiles vary fastest (tokens stream once); a larger one is walked item-fastest so
        that each weight tile is fetched from HBM once and the (smaller) token operand stays resident instead."""
        args.n_active = self.n_items[items].data_ptr()
        if not self.wide:
            K.gemm(variant, a0, a1, b, args, n_tiles, items, pdl=pdl)
            return
        wbytes = a0.tensor.numel() * a0.tensor.element_size() * (2 if a1 is not None else 1)
        K.wide_gemm(variant, a0, a1, b, args, n_tiles, items, pdl=pdl, items_fastest=wbytes > (96 << 20))

    def _bf16_gemm(self, variant: int, weight: K.TensorMap, x: torch.Tensor, args: K.GemmArgs, n_tiles: int, R: int, items: int, pdl: bool) -> None:
        """Plain bf16 projections of R rows: up to 256 rows a tile, so that a weight tile in shared memory feeds as many (2048 rows of q/k/v,
        some 14,000 features of 4096 on average: 179 us, 282 us in tiles of 64)."""
        made = self._bf16.get((weight, x.data_ptr()))
        if made is None:
            a = S.StackGemmArgs()
            a.n, a.k, a.zcount, a.scale, a.status = args.n_total, args.k_total, 1, args.out_scale, args.status
            a.out, a.out_f32, a.out_ld = (args.out_f32, 1, args.ld_out) if args.out_f32 else (args.out_bf16, 0, args.ld_out)
            made = self._bf16[weight, x.data_ptr()] = (a, {})
        a, maps = made
        if not self.wide:
            if ROWS not in maps:
                maps[ROWS] = K.act_tmap(x, ROWS)
            self._gemm(variant, weight, None, maps[ROWS], args, n_tiles, items, pdl=pdl)
            return
        a.rows = R
        ntok = StackPrefill.tile_rows(S.EPI_STORE, n_tiles, R)
        if ntok not in maps:
            ld = x.stride(0) * 2
            maps[ntok] = K.TensorMap(x, (x.shape[1], 1, x.shape[0]), (ld, ld), (64, 1, ntok), 1)
        S.gemm(S.EPI_STORE, ntok, weight, None, maps[ntok], a, weight.tensor.numel() * 2 > (96 << 20), pdl, library=S.products())

    # ------------------------------------------------------------------ argument blocks
    def _item_args(self, n, k) -> K.GemmArgs:
        g = K.GemmArgs()
        g.n_total, g.k_total, g.rows, g.a_group, g.out_scale = n, k, self.step, 0, 1.0
        g.active_ids, g.max_slots = self.zero_ids.data_ptr(), self.items
        g.row_offsets = self.row_offsets.data_ptr()
        g.status = self.t.fab.status.data_ptr()
        return g

    def _build_args(self):
        s, t = self.spec, self.t
        H, ix = s.hidden, s.indexer
        self.L: List[dict] = []
        for L, d in enumerate(t.layers):
            a, nh, nkv, cols = d["a"], d["nh"], d["nkv"], d["cols"]
            e: dict = {}
            g = self._item_args(d["wqkv"].shape[0], H)
            g.out_f32, g.ld_out = self.qkv.data_ptr(), self.qkv.shape[1]
            e["qkv"] = g
            p = K.AttnPostArgs.from_buffer_copy(d["args_post"])
            p.qkv, p.ld, p.q_out = self.qkv.data_ptr(), self.qkv.shape[1], self.q.data_ptr()
            if d["kind"] == FULL_DSA:
                p.iq8, p.ihw = self.iq8.data_ptr(), self.ihw.data_ptr()
                # the step runtime keeps the query quantisation scale in a 16-row side buffer; a chunk has more rows,
                # so here the scale is folded into the head weights (the kernel's form without that buffer)
                p.iq_scale = None
                e["sweep_maps"] = K.sweep_maps(d["ik"], self.iq8)
                sw = K.SweepArgs()
                sw.ihw, sw.iks = self.ihw.data_ptr(), d["iks"].data_ptr()
                sw.heads, sw.top_k = ix.head_count, ix.top_k
                sw.logits, sw.ld, sw.status = self.idx_logits.data_ptr(), self.idx_logits.shape[1], t.fab.status.data_ptr()
                e["sweep"] = sw
            e["post"] = p
            q = K.AttnArgs.from_buffer_copy(d["args_attn"])
            q.q, q.o8, q.o_scale, q.part, q.tickets = self.q.data_ptr(), self.o8.data_ptr(), self.os.data_ptr(), None, None
            if d["kind"] == FULL_DSA:
                q.sel = self.sel.data_ptr()
            e["attn"] = q
            # one CTA per (KV head, row) shares every gathered key among the group's query heads
            e["group_attn"] = self.group_attn and a.head_dim == 192 and a.v_head_dim == 128 and nh // nkv <= 16
            g = self._item_args(H, d["wo"].k)
            g.w_scale0, g.a_scale = d["wo"].s.data_ptr(), self.os.data_ptr()
            g.out_bf16, g.ld_out = self.part.data_ptr(), H
            e["o"] = g
            if "dense" in d:
                dn = d["dense"]
                g = self._item_args(dn["gate"].n, H)
                g.w_scale0, g.w_scale1, g.a_scale = dn["gate"].s.data_ptr(), dn["up"].s.data_ptr(), self.xs.data_ptr()
                g.out_q, g.out_qscale = self.yd8.data_ptr(), self.yds.data_ptr()
                e["gu"] = g
                g = self._item_args(H, dn["down"].k)
                g.w_scale0, g.a_scale = dn["down"].s.data_ptr(), self.yds.data_ptr()
                g.out_bf16, g.ld_out = self.part.data_ptr(), H
                e["down"] = g
            else:
                rt = s.routing
                r = K.RouterArgs()
                r.w, r.bias, r.xn = None, d["router_b"].data_ptr(), self.xn.data_ptr()      # selection only (scores by torch.mm)
                if "router_wt" not in d:
                    d["router_wt"] = d["router_w"].float().t().contiguous()                 # [hidden][experts]
                r.hidden, r.experts, r.top_k = H, rt.expert_count, rt.top_k
                r.sigmoid, r.normalize, r.route_scale = int(rt.score_func == "sigmoid"), int(rt.normalize_top_k), rt.route_scale
                r.scores, r.ticket = self.scores.data_ptr(), self.tickets.data_ptr()
                r.max_slots = 0
                e["router"] = r
            self.L.append(e)
        if self.draft is not None:
            dr, dd = self.draft, s.draft
            g = self._item_args(dd.hidden, dr.kf)
            g.out_bf16, g.ld_out = self.dh.data_ptr(), dd.hidden
            self.args_fc = g
            g = self._item_args(dr.wkv.shape[0], dd.hidden)
            g.out_f32, g.ld_out = self.draw.data_ptr(), self.draw.shape[1]
            self.args_kv = g
            self.args_ingest = []
            for Ld in dr.layers:
                p = K.AttnPostArgs.from_buffer_copy(Ld["args_ingest_post"])
                p.qkv, p.ld = self.draw.data_ptr(), self.draw.shape[1]
                self.args_ingest.append(p)

    @contextmanager
    def _stage(self, name: str):
        if not self.profile:
            yield
            return
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        yield
        b.record()
        self._timed.setdefault(name, []).append((a, b))

    def stage_ms(self) -> Dict[str, float]:
        """Device milliseconds per stage since the last call (``profile`` must be on); waits for the stream."""
        torch.cuda.current_stream().synchronize()
        out = {k: round(sum(a.elapsed_time(b) for a, b in v), 3) for k, v in self._timed.items()}
        self._timed = {}
        return out

    # ------------------------------------------------------------------ collectives (NCCL on the current stream)
    def _all_reduce(self, buf: torch.Tensor) -> None:
        if self.tp > 1:
            dist.all_reduce(buf, group=self.group)

    # ------------------------------------------------------------------ chunks
    def _chunk(self, pos0: int, R: int) -> None:
        self._span(pos0, [R])

    def _span(self, start: int, sizes: List[int]) -> None:
        """Consecutive chunks of ``sizes`` rows (all but the last of ``chunk``) from position ``start`` on, layer by layer: attention and
        routing chunk by chunk, the experts for all of them."""
        s, t, tp = self.spec, self.t, self.tp
        pdl, n = False, sum(sizes)
        rows = [(c, c * self.C, R) for c, R in enumerate(sizes)]          # chunk, its first row, its rows
        torch.add(self._steps[:len(sizes)], start, out=self.pos[:len(sizes)])
        if getattr(self, "shard_index", False) and n % (ROWS * tp) == 0:   # ranks: spans of one chunk
            self.pos[0, 1:2].fill_(start + self.rank * (n // tp))
        x = self.x
        K.embed_rows(self.tokens, t.embed, x, n, pdl=pdl)
        for kind, tab in self.rope.items():
            a = s.attention[kind]
            K.rope_table(self.pos, n, a.rope_dim, a.rope_theta, tab, pdl=pdl)
        if FULL_DSA in self.rope:
            K.rope_table(self.pos, n, s.indexer.rope_dim, s.attention[FULL_DSA].rope_theta, self.idx_rope, pdl=pdl)
        T = n // tp if self.ep else n
        src = self.xl if self.ep else x
        xl = x[self.rank * T:(self.rank + 1) * T] if self.ep else x[:n]
        for L, (d, e) in enumerate(zip(t.layers, self.L)):
            for c, row0, R in rows:
                self._layer_rows(L, d, e, c, row0, start + row0, R, xl)
            if "dense" not in d:
                self.moe.stage = self._stage if self.profile else None
                with self._stage("moe"):
                    if self.ep or tp == 1:
                        self.moe.run(src, d["g_post"], self.topk_ids, self.topk_p, src, src, weights=self.moe_w[L], tokens=T)
                    else:
                        self.moe.run(src, d["g_post"], self.topk_ids, self.topk_p, self.zeros, self.part, weights=self.moe_w[L], tokens=T)
                with self._stage("tp_reduce"):
                    if self.ep:
                        dist.all_gather_into_tensor(x[:n], src[:T], group=self.group)
                    elif tp > 1:
                        self._all_reduce(self.part[:n])
                        torch.add(x[:n], self.part[:n], out=x[:n])
            tap = t.tap_of_layer.get(L)
            if tap is not None and self.draft is not None:
                H = s.hidden
                self.feats[:n, tap * H:(tap + 1) * H].copy_(x[:n])
        if self.draft is not None:
            with self._stage("draft_ingest"):
                K.rope_table(self.pos, n, s.draft.head_dim, s.draft.rope_theta, self.drope, pdl=pdl)
                for c, row0, R in rows:
                    self._ingest(c, row0, R)

    def _layer_rows(self, L: int, d: dict, e: dict, c: int, row0: int, pos0: int, R: int, xl: torch.Tensor) -> None:
        """One layer for the R rows of chunk ``c`` (rows ``row0`` on of the span) up to the choice of their experts, or through the dense MLP."""
        s, t, tp = self.spec, self.t, self.tp
        H, pdl, items = s.hidden, False, -(-R // self.step)
        x, xn, part, pos = self.x[row0:row0 + R], self.xn, self.part, self.pos[c]
        # ---- attention (tensor parallel)
        with self._stage("norm"):
            K.prep_norm(x, d["g_in"], R, s.norm_eps, xn=xn, pdl=pdl)
        with self._stage("qkv_gemm"):
            self._bf16_gemm(self.V_BF16_F32, d["map_qkv"], self.xn, e["qkv"], d["wqkv"].shape[0] // 128, R, items, pdl)
        p, q = e["post"], e["attn"]
        p.rows, p.pos0, p.rope = R, pos.data_ptr(), self.rope[d["kind"]][row0].data_ptr()
        if d["kind"] == FULL_DSA:
            p.idx_rope_tab = self.idx_rope[row0].data_ptr()
        with self._stage("attn_post"):
            K.attn_post(p, pdl=pdl)
        if d["kind"] == FULL_DSA and pos0 + R > s.indexer.top_k:
            sw = e["sweep"]
            sw.rows, sw.pos0 = R, pos.data_ptr()
            shard = self.shard_index and R % (ROWS * tp) == 0
            Rl = R // tp if shard else R                         # rows this rank selects for
            first = self.rank * Rl if shard else 0
            sw.group0, sw.ngroups = first // ROWS, Rl // ROWS
            tiles = -(-(pos0 + R) // 128)
            with self._stage("index_sweep"):
                K.index_sweep(*e["sweep_maps"], sw, max(1, min(tiles, 592 // (Rl // ROWS))), pdl=pdl)
            with self._stage("topk"):
                logits, pos_l = self.idx_logits[first:first + Rl], pos[1:]             # pos[1] = pos0 + first
                sel = self.sel_local if shard else self.sel
                if t.topk_grid:
                    K.topk_rows_grid(logits, pos_l, Rl, s.indexer.top_k, sel, self.topk_state, 16, pdl=pdl)
                else:
                    K.topk_rows(logits, pos_l, Rl, s.indexer.top_k, sel, pdl=pdl)
                if shard:
                    dist.all_gather_into_tensor(self.sel[:R], self.sel_local[:Rl], group=self.group)
        q.rows, q.pos0 = R, pos.data_ptr()
        with self._stage("attn_dsa" if d["kind"] == FULL_DSA else "attn_swa"):
            if e["group_attn"]:
                K.attn_group(q, pdl=pdl)
            else:
                K.attn_rows(q, 1, pdl=pdl)
        with self._stage("o_gemm"):
            self._gemm(self.V_FP8_BF16, d["wo"].map, None, self.map_o8, e["o"], H // 128, items, pdl=pdl)
        moe = "dense" not in d
        T = R // tp if self.ep else R
        with self._stage("tp_reduce"):
            if self.ep and moe:
                # sequence parallel from here to the end of the layer: this rank keeps rows [rank*T, (rank+1)*T)
                dist.reduce_scatter_tensor(self.rs[:T], part[:R], group=self.group)
                torch.add(xl, self.rs[:T], out=self.xl[:T])
            else:
                self._all_reduce(part[:R])
                torch.add(x, part[:R], out=x)
        if not moe:
            dn = d["dense"]
            with self._stage("dense_mlp"):
                K.prep_norm(x, d["g_post"], R, s.norm_eps, x8=self.x8, xs=self.xs, pdl=pdl)
                self._gemm(self.V_FP8_GU, dn["gate"].map, dn["up"].map, self.map_x8, e["gu"], dn["gate"].n // 128, items, pdl=pdl)
                self._gemm(self.V_FP8_BF16, dn["down"].map, None, self.map_yd8, e["down"], H // 128, items, pdl=pdl)
            with self._stage("tp_reduce"):
                self._all_reduce(part[:R])
                torch.add(x, part[:R], out=x)
            return
        with self._stage("router"):
            K.prep_norm(self.xl if self.ep else x, d["g_post"], T, s.norm_eps, xn=xn, pdl=pdl)
            # scores of all chunk rows as one fp32 matrix product (library GEMM, no TF32: the same products as
            # the step's FMA loop, summed in another order), selection by the router kernel per 16 rows
            tf32 = torch.backends.cuda.matmul.allow_tf32
            torch.backends.cuda.matmul.allow_tf32 = False
            torch.mm(xn[:T].float(), d["router_wt"], out=self.scores[:T])
            torch.backends.cuda.matmul.allow_tf32 = tf32
            r = e["router"]
            r.rows, r.topk_ids, r.topk_p = T, self.topk_ids[row0].data_ptr(), self.topk_p[row0].data_ptr()
            K.router(r, pdl=pdl)

    def _ingest(self, c: int, row0: int, R: int) -> None:
        """Draft context for a chunk's rows: fc over this rank's feature taps (reduced over the ranks),
        RMSNorm, every draft layer's k/v projection in one GEMM, k-norm + RoPE + append."""
        dr, dd, pdl, items = self.draft, self.spec.draft, False, -(-R // self.step)
        self._bf16_gemm(self.V_BF16_BF16, dr.map_fc, self.taps[row0:row0 + self.C], self.args_fc, dd.hidden // 128, R, items, pdl)
        self._all_reduce(self.dh[:R])
        K.prep_norm(self.dh, dr.hidden_norm, R, dd.norm_eps, xn=self.dxn, pdl=pdl)
        self._bf16_gemm(self.V_BF16_F32, dr.map_kv, self.dxn, self.args_kv, dr.wkv.shape[0] // 128, R, items, pdl)
        for p in self.args_ingest:
            p.rows, p.pos0, p.rope = R, self.pos[c].data_ptr(), self.drope[row0].data_ptr()
            K.attn_post(p, pdl=pdl)

    # ------------------------------------------------------------------ public API
    def run(self, prompt: torch.Tensor, start: int = 0, end: Optional[int] = None) -> int:
        """Ingest prompt positions [start, end) in whole chunks on the current stream; returns the first
        position that was *not* ingested (the remainder, fewer than ``quantum`` rows, is left to replay).
        ``prompt`` may live in pinned host memory.  Caches before ``start`` must be valid."""
        n = int(prompt.numel())
        end = n if end is None else end
        if not 0 <= start <= end <= n or end > self.t.capacity:
            raise ValueError(f"prefill range [{start}, {end}) outside the prompt / cache capacity")
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        p = start
        chunks = plan_chunks(start, end, self.C, self.quantum)
        self._fit_span(sum(c.rows for c in chunks))
        ev0.record()
        each = self.span // self.C
        for i in range(0, len(chunks), each):
            sizes = [c.rows for c in chunks[i:i + each]]
            first, p = chunks[i].pos0, chunks[i].pos0 + sum(sizes)
            self.tokens[:p - first].copy_(prompt[first:p].to(torch.int32), non_blocking=True)
            self._span(first, sizes)
        ev1.record()
        self.phases = {"chunks": len(chunks), "rows": p - start, "events": (ev0, ev1)}
        return p

    def executor_ms(self) -> float:
        """Device time of the last ``run`` (waits for it)."""
        ev0, ev1 = self.phases["events"]
        ev1.synchronize()
        return ev0.elapsed_time(ev1)

    def warm_chunks(self, sizes=None) -> None:
        """Run row counts once on scratch positions so that module loading, kernel attributes, NCCL channels and span buffers are paid
        before the first request.  The default ends with the longest span.  The rows it writes into the caches start at position 0 and
        are overwritten by the next request."""
        for r in sorted(set(sizes or [self.quantum, self.C, self.span_limit])):
            rows = [r] if r <= self.C else [c.rows for c in plan_chunks(0, min(r, self.t.capacity), self.C, self.quantum)]
            self._fit_span(sum(rows))
            self.tokens.zero_()
            self._span(0, rows[:self.span // self.C])
        torch.cuda.current_stream().synchronize()
        self.check()

    def resume_from_decode(self, position: int) -> int:
        """A session that was decoding continues with a long new turn: every cache is position indexed (or a
        ring keyed by position), so chunks simply resume at ``position``; returns it for symmetry with the
        reference's executor (which rebuilds its swizzled shadows here)."""
        if not 0 <= position <= self.t.capacity:
            raise ValueError("resume position outside the cache")
        return position

    def check(self) -> None:
        self.t.fab.check()
        if self.moe_fab is not self.t.fab:
            self.moe_fab.check()

    def close(self) -> None:
        if self.moe_fab is not self.t.fab:
            self.moe_fab.close()
