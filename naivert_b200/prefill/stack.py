"""Chunk path of layer-stack models: R prompt rows go through every layer in one pass over the step's own caches.

    rows (stream update + norms)
    token mixer        one class per mechanism in ``prefill/stack_mixers.py``
    feed-forward       two-product GLU -> down, or squared ReLU -> down; routed experts: scores -> choice -> rows sorted by
                       expert -> grouped products -> weighted sum inside the next row kernel

A chunk may start and end anywhere and has any length up to ``chunk`` rows; the caches and states it leaves are those
the step continues from.  Where the chunks are too short to fill the routed experts, several go through the layers side by side
(a span): mixers and dense feed-forwards take them one after the other with the scratch of one, the experts' products all at once.
"""
from __future__ import annotations

from bisect import bisect_left
from contextlib import contextmanager, nullcontext
from functools import lru_cache
from typing import Callable, Dict, List, Optional, Sequence, Tuple

import torch

from ..ops import kernels as K
from ..ops import stack_kernels as S
from ..runtime.packing import Packed, pad
from ..runtime.stack import StackRuntime
from .stack_mixers import MIXERS

SMS = 148
# tile sizes of the chunk products by epilogue (the others: 64 and 256)
TILE_ROWS = {S.EPI_STORE: (64, 128, 192, 256), S.EPI_RELU2: (64, 128, 192, 256), S.EPI_BIAS: (64, 128, 192, 256), S.EPI_CLAMPED_GLU: (64, 128, 192),
             S.EPI_SILU_GLU: (64, 128)}
FUNCTION_EPI = (S.EPI_TANH, S.EPI_DECAY_SOFT, S.EPI_DECAY_EXP)
# Pairs (token, choice) per expert that a span is filled up to, and its most rows.  Below, an expert's product is bound by the read of its
# weights (12.9 GB a layer at 256 experts of 4096 x 2048), which a span does once: with three such layers, 8192 rows in chunks of 2048 take
# 30.1 ms, 47.0 ms when every chunk went through the experts by itself (their products: 28.3 -> 11.0 ms).  A span's rows cost 2 GB there.
SPAN_PAIRS, SPAN_ROWS = 256, 8192


_UNTIMED = nullcontext()


class StackPrefill:
    quantum = 1

    def __init__(self, runtime: StackRuntime, chunk: int = 2048, kv_block: int = 16384):
        self.t, self.spec, self.C, self.dev = runtime, runtime.spec, chunk, runtime.dev
        self.f32, self.act = runtime.f32, runtime.act
        self.kv_block = pad(min(kv_block, runtime.capacity), 64)
        s, dev, C = self.spec, self.dev, chunk
        f32, i32 = torch.float32, torch.int32
        L = runtime.layers
        ffs = [d["spec"].mlp for d in L if d["spec"].mlp is not None]
        moe = [f for f in ffs if f.kind == "moe"]
        self.h_ld = pad(s.hidden, 8)
        # Argument blocks by launch: a prompt of a small model is some 70 launches of a few microseconds, and filling some twenty fields anew for
        # each took longer.  What changes from prompt to prompt - rows, positions, segments - is set every time.  (Buffers that are taken
        # anew clear it.)
        self._kept: Dict[tuple, object] = {}
        self.maps: Dict[tuple, object] = {}
        filled = min([-(-SPAN_PAIRS * f.routing.expert_count // f.routing.top_k) for f in moe], default=0)
        self.span_limit = max(C, min(SPAN_ROWS, filled, runtime.capacity) // C * C)
        self._size_span(C)
        # buffers of the mixers, one per role, shared by the layers (sizes differ from layer to layer)
        sizes: Dict[tuple, int] = {}
        for d in L:
            for name, (n, t) in MIXERS[d["kind"]].scratch(self, d["spec"].mixer, d).items():
                sizes[name, t] = max(n, sizes.get((name, t), 0))
        self.buf = {name: self._zeros(n, t) for (name, t), n in sizes.items()}
        self.ff = self._zeros(C * max([pad(f.ff, 8) for f in ffs if f.kind != "moe"], default=0), self.act)
        self.head_rows = 256
        self.pdl = False
        self.hw = torch.zeros(self.head_rows, self.h_ld, dtype=self.act, device=dev)
        self.tensor_cores = not self.f32              # attention of chunk rows on tcgen05 (else the plain kernel)
        self.phases: dict = {}
        self.profile = False                          # per-stage CUDA-event timing (adds an event pair per stage)
        self._timed: Dict[str, list] = {}

    def _zeros(self, n: int, t=torch.float32) -> torch.Tensor:
        return torch.zeros(max(8, n), dtype=t, device=self.dev)

    def _size_span(self, P: int) -> None:
        """Buffers for spans of ``P`` rows (whole chunks); an allocation that fails leaves the present ones."""
        s, C, L, z, f32, i32 = self.spec, self.C, self.t.layers, self._zeros, torch.float32, torch.int32
        moe = [d["spec"].mlp for d in L if d["spec"].mlp is not None and d["spec"].mlp.kind == "moe"]

        def rows(width: int, t=f32) -> torch.Tensor:
            return torch.zeros(P, width, dtype=t, device=self.dev)

        # position of each chunk, stream, input and output rows of the sublayers
        rows_of = {"pos": torch.zeros(P // C, dtype=i32, device=self.dev), "x": rows(s.hidden), "h": rows(self.h_ld, self.act), "y": rows(s.hidden),
                   "y2": rows(s.hidden) if any(d["kind"] == "parallel" for d in L) else None}
        new = {"tokens": torch.zeros(P, dtype=i32, device=self.dev)}
        if moe:
            E, T = max(f.routing.expert_count for f in moe), max(f.routing.top_k for f in moe)
            items, cap = -(-P * T // 64) + E, max(self._segment_rows(P, f.routing) for f in moe)
            new.update(scores=z(P * E), ids=z(P * T, i32), probs=z(P * T), slot_of=z(P * T, i32), n_items=z(1, i32), seg_rows=z(E, i32),
                       max_items=items, item_z=z(items, i32), item_row=z(items, i32), item_live=z(items, i32), cap=cap, sorted=z(cap * self.h_ld, self.act),
                       ea=z(cap * max(pad(f.ff, 8) for f in moe), self.act), ey=z(cap * s.hidden))
        self.rows_of, self.span = rows_of, P
        self._kept.clear()
        for key in [k for k in self.maps if k[0] == "x"]:      # maps hold the tensors they describe, and these go
            del self.maps[key]
        for name, v in new.items():
            setattr(self, name, v)
        self._window()

    def _fit_span(self, n: int) -> None:
        """Spans for ``n`` rows as far as the limit and the memory go.  What a span needs beyond a chunk is taken when a prompt first asks
        for it: an engine that sees short prompts only never holds it, and without the memory chunks go on one by one."""
        P = min(self.span_limit, -(-n // self.C) * self.C)
        if P > self.span:
            torch.cuda.synchronize(self.dev)              # earlier calls may still use the buffers that go, on any stream
        while P > self.span:
            try:
                self._size_span(P)
            except torch.OutOfMemoryError:
                P -= self.C
                self.span_limit = P

    def kept(self, key: tuple, build: Callable[[], object]):
        """The argument block that ``build`` made for ``key`` (its launch, layer run and whatever else its fixed fields hang on)."""
        a = self._kept.get(key)
        if a is None:
            a = self._kept[key] = build()
        return a

    def stage(self, name: str):
        return self._stage(name) if self.profile else _UNTIMED

    @contextmanager
    def _stage(self, name: str):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        yield
        b.record()
        self._timed.setdefault(name, []).append((a, b))

    def stage_ms(self) -> Dict[str, Tuple[float, int]]:
        """(device milliseconds, calls) per stage since the last call (``profile`` must be on); waits for the stream."""
        torch.cuda.current_stream().synchronize()
        out = {k: (sum(a.elapsed_time(b) for a, b in v), len(v)) for k, v in self._timed.items()}
        self._timed = {}
        return out

    @staticmethod
    def _item_rows(rows: int, routing, f32: bool = False) -> int:
        """Rows of a segment of the expert list: 128 where the experts are well filled."""
        return 128 if not f32 and rows * routing.top_k >= 96 * routing.expert_count else 64

    def _items(self, rows: int, routing, item_rows: int) -> int:
        """Most segments the choices of ``rows`` tokens can need."""
        pairs = rows * routing.top_k
        return pairs // item_rows + min(pairs, routing.expert_count)

    def _segment_rows(self, rows: int, routing) -> int:
        """Rows the sorted buffers need for chunks of at most ``rows`` tokens."""
        return max(self._items(rows, routing, i) * i for i in (64, 128))

    # ------------------------------------------------------------------ products
    def _wmap(self, p: Packed) -> K.TensorMap:
        key = ("w", p.w.data_ptr(), p.z, p.n)
        if key not in self.maps:
            self.maps[key] = S.weight_map(p.w, p.k)
        return self.maps[key]

    @staticmethod
    @lru_cache(maxsize=4096)
    def tile_rows(epi: int, tiles: int, rows: int) -> int:
        """Token rows per tile of a product with ``tiles`` feature tiles.  Few rows are one tile where the feature tiles occupy more than
        half of the SMs: every weight is then fetched by one CTA only, and what is in flight - which bounds a product that streams
        its weights - is all different: 152,576 features of 4096 x 1 row 419 -> 212 us, 10,240 x 187 rows 49 -> 38 us, and 16,384 x 187
        rows of two products 90 -> 87 us against the widest tile that fills the SMs, which larger products take.  With fewer feature
        tiles two rows of tiles are still one wave (8,192 features of 4096: 100 rows in tiles of 64 / 128 21.1 / 22.5 us, of two products
        34.6 / 40.0; feature-major stores of 512, 100 / 200 rows in tiles of 64 / 256 6.6 / 7.9 and 8.5 / 9.2).  Tanh and the decays are
        bound by their special functions, a thread's share of which grows with the tile (12,288 features of 128, 100 rows: 12.5 / 16.1)."""
        sizes = TILE_ROWS.get(epi, (64, 256))
        whole = next((t for t in sizes if t >= rows), None)
        if whole is not None and 2 * tiles > SMS and (whole == 64 or epi not in FUNCTION_EPI):
            return whole
        return next((t for t in reversed(sizes) if t != 192 and tiles * -(-rows // t) >= SMS - 20), 64)

    def _xmap(self, t: torch.Tensor, k: int, zcount: int, zstride: int, rows: int, ld: int, box: int, offset: int) -> K.TensorMap:
        key = ("x", t.data_ptr(), k, zcount, zstride, rows, ld, box, offset)
        if key not in self.maps:
            self.maps[key] = S.token_map(t, k, zcount, zstride, rows, ld, box, offset)
        return self.maps[key]

    def gemm(self, epi: int, w: Packed, x: torch.Tensor, x_ld: int, rows: int, out: torch.Tensor, out_ld: int, *, w2: Optional[Packed] = None,
              z: int = 1, x_z: int = 0, out_z: int = 0, x_off: int = 0, x_rows: Optional[int] = None, items: Optional[tuple] = None,
              bias: Optional[torch.Tensor] = None, rate: Optional[torch.Tensor] = None, act_cols: int = 0, scale: float = 1.0, limit: float = 0.0, alpha: float = 0.0,
             keep: bool = False) -> None:
        """out[row, z, :] = epilogue(W_z x[row, z, :]) for every token row; ``items`` = (segment rows, most segments).  ``keep``: weights
        and buffers are the engine's own, which stay, and so does the argument block (a weight and an epilogue have one caller)."""
        def build():
            a = S.StackGemmArgs()
            a.n, a.k, a.zcount = w.n, w.k, z
            a.out, a.out_ld, a.out_zstride, a.out_f32 = out.data_ptr(), out_ld, out_z, int(out.dtype == torch.float32)
            a.bias = None if bias is None else bias.data_ptr()
            a.rate = None if rate is None else rate.data_ptr()
            a.act_cols, a.scale, a.limit, a.alpha, a.status = act_cols, scale, limit, alpha, self.t.fab.status.data_ptr()
            if items is not None:
                a.n_items, a.item_z, a.item_row, a.item_live = (self.n_items.data_ptr(), self.item_z.data_ptr(), self.item_row.data_ptr(),
                                                                self.item_live.data_ptr())
            if self.f32:
                a.act, a.act_ld, a.act_zstride = x.data_ptr() + 4 * x_off, x_ld, x_z
                a.w, a.w2 = w.w.data_ptr(), None if w2 is None else w2.w.data_ptr()
                a.w_ld, a.w_zstride = w.ld, w.n * w.ld
            return a, w, {}                              # (the weight's name in the key stays its own)

        key = ("gemm", epi, id(w), x.data_ptr(), x_off, out.data_ptr(), out_ld, items is None)
        a, _, maps = self.kept(key, build) if keep else build()
        a.rows = rows
        if items is not None:
            a.item_rows, a.max_items = items
        if self.f32:
            S.gemm_f32(epi, a, self.pdl)
            return
        dual = w2 is not None
        if items is not None:
            ntok = items[0]
        else:
            ntok = self.tile_rows(epi, -(-w.n // 128) * z, rows)
        live = x_rows if x_rows is not None else x.numel() // x_ld
        made = maps.get((ntok, live))
        if made is None:
            made = maps[ntok, live] = (self._wmap(w), self._wmap(w2) if dual else None, self._xmap(x, w.k, z, x_z, live, x_ld, ntok, x_off),
                                       items is None and w.nbytes * (2 if dual else 1) > (96 << 20))
        S.gemm(epi, ntok, *made[:3], a, made[3], self.pdl)

    def early(self, rows: int) -> bool:
        """Whether the launches of ``rows`` rows begin under the end of the one in front.  That takes 2 us off a launch: 32 / 187 / 800 rows of
        the bench models 1.06 / 1.03 / 1.01 times as fast, of the small models 1.03 / 1.05 / 1.15, of their 32-bit form 1.19 / 1.16 / 0.95
        (2048 of the routed bench model: 0.97).  Long launches lose by it: CTAs that start while others of the last launch hold their SMs
        stand closer than one to an SM, and two kernels whose grids are about an SM each never begin early for that (attention on the tensor
        cores, matrix-state recurrence: with them 400 / 1200 rows of the matrix-state model were 0.95 / 0.89)."""
        return self.t.pdl and (rows <= 512 if self.f32 else rows * self.spec.hidden <= 1 << 22)

    def product(self, *args, **more) -> None:
        """``gemm`` of the engine's own weights and buffers."""
        self.gemm(*args, keep=True, **more)

    # ------------------------------------------------------------------ one span
    def _window(self, chunk: Optional[int] = None) -> None:
        """``pos``, ``x``, ``h``, ``y`` and ``y2`` become those of one chunk of the span, or of the whole of it (``at``: which, -1 all)."""
        self.at = -1 if chunk is None else chunk

        def build():
            if chunk is None:
                return self.rows_of
            return {name: None if t is None else t[chunk:chunk + 1] if name == "pos" else t[chunk * self.C:(chunk + 1) * self.C] for name, t in self.rows_of.items()}

        self.__dict__.update(self.kept(("window", chunk), build))

    def _chunks(self, R: int, pos0: int):
        """(rows, first position) of the chunks of a span of R rows, each with its own rows in place."""
        for i in range(-(-R // self.C)):
            self._window(i)
            yield min(self.C, R - i * self.C), pos0 + i * self.C
        self._window()

    def _rows(self, R: int, *, embed: bool = False, y: Optional[torch.Tensor] = None, post=None, y2: Optional[torch.Tensor] = None, join=None,
              moe=None, add=None, pre=None, copy: bool = False) -> None:
        """Stream update; then the input rows ``h`` of the next sublayer: normed by ``pre``, or the stream itself (``copy``)."""
        s = self.spec

        def build():
            a = S.StackRowArgs()
            if embed:
                a.tokens, a.table, a.vocab, a.embed_scale = self.tokens.data_ptr(), self.t.embed.data_ptr(), s.vocab, s.embed_scale
            if y is not None:
                a.y, a.y_ld, a.post_w = y.data_ptr(), s.hidden, post.data_ptr()
                if join is not None:
                    a.y2, a.join_w, a.join_w2 = y2.data_ptr(), join[0].data_ptr(), join[1].data_ptr()
                if moe is not None:
                    a.slot_of, a.probs, a.top_k = self.slot_of.data_ptr(), self.probs.data_ptr(), moe.top_k
            a.add = None if add is None else add.data_ptr()
            a.x, a.width, a.eps = self.x.data_ptr(), s.hidden, s.norm_eps
            a.pre_w = None if pre is None else pre.data_ptr()
            a.norm, a.copy_h = S.NORM[s.norm], int(copy)
            a.h, a.h_f32, a.h_ld = self.h.data_ptr(), int(self.f32), self.h_ld
            return a

        # (norms and vectors belong to the layers, whose addresses stay)
        key = ("rows", embed, y is not None and y.data_ptr(), post is not None and post.data_ptr(), join is not None, moe is not None,
               add is not None and add.data_ptr(), pre is not None and pre.data_ptr(), copy)
        a = self.kept(key, build)
        a.rows = R
        with self.stage("rows"):
            S.rows(a, self.pdl)

    def _feed_forward(self, d: dict, R: int) -> torch.Tensor:
        """Returns the buffer that holds the result rows (sorted by expert for routed layers)."""
        f, W = d["spec"].mlp, self.spec.hidden
        fp = pad(f.ff, 8)
        if f.kind == "relu2":
            for n, _ in self._chunks(R, 0):
                with self.stage("ff_up"):
                    self.product(S.EPI_RELU2, d["up"], self.h, self.h_ld, n, self.ff, fp)
                with self.stage("ff_down"):
                    self.product(S.EPI_STORE, d["down"], self.ff, fp, n, self.y, W)
            return self.y
        if f.kind == "dense":
            for n, _ in self._chunks(R, 0):
                with self.stage("dense_gate_up"):
                    self.product(S.EPI_CLAMPED_GLU, d["gate"], self.h, self.h_ld, n, self.ff, fp, w2=d["up"], limit=f.limit, alpha=f.alpha)
                with self.stage("dense_down"):
                    self.product(S.EPI_STORE, d["down"], self.ff, fp, n, self.y, W)
            return self.y
        rt = f.routing
        with self.stage("router"):
            self.product(S.EPI_STORE, d["router"], self.h, self.h_ld, R, self.scores, rt.expert_count)
        ir = self._item_rows(R, rt, self.f32)
        items = self._items(R, rt, ir)

        def build():
            q = K.RouterArgs()
            q.bias, q.hidden, q.experts, q.top_k = d["correction"].data_ptr(), W, rt.expert_count, rt.top_k
            q.sigmoid, q.normalize, q.route_scale = 1, int(rt.normalize_top_k), rt.route_scale
            q.scores, q.topk_ids, q.topk_p = self.scores.data_ptr(), self.ids.data_ptr(), self.probs.data_ptr()
            e = K.EpArgs()
            e.topk_ids, e.topk_p, e.top_k = self.ids.data_ptr(), self.probs.data_ptr(), rt.top_k
            e.experts = e.experts_local = rt.expert_count
            e.slot_of, e.n_items, e.item_expert, e.item_row = (self.slot_of.data_ptr(), self.n_items.data_ptr(), self.item_z.data_ptr(),
                                                               self.item_row.data_ptr())
            e.seg_rows, e.item_live, e.x_args = self.seg_rows.data_ptr(), self.item_live.data_ptr(), self.t.fab.xchg_args()
            g = S.MoeGatherArgs()
            eb = self.h.element_size()
            g.h, g.h_ld, g.sorted, g.slot_of = self.h.data_ptr(), self.h_ld * eb, self.sorted.data_ptr(), self.slot_of.data_ptr()
            g.top_k, g.row_bytes, g.cap = rt.top_k, self.h_ld * eb, self.cap
            return q, e, g

        q, e, g = self.kept(("experts", d["correction"].data_ptr()), build)
        q.rows = e.tokens = g.rows = R
        e.max_items, e.item_rows = items, ir
        with self.stage("choice"):
            S.route(q, rt.group_count, rt.limited_group_count, self.pdl)
        with self.stage("expert_count"):
            S.moe_count(e, self.pdl)
        with self.stage("expert_gather"):
            S.moe_gather(g, self.pdl)
        seg = dict(items=(ir, items))
        with self.stage("expert_gate_up"):
            self.product(S.EPI_SILU_GLU, d["gate"], self.sorted, self.h_ld, ir, self.ea, fp, w2=d["up"], x_rows=self.cap, **seg)
        with self.stage("expert_down"):
            self.product(S.EPI_STORE, d["down"], self.ea, fp, ir, self.ey, W, x_rows=self.cap, **seg)
        return self.ey

    def _chunk(self, pos0: int, R: int, want: Sequence[int] = (), trace: Optional[list] = None) -> Optional[torch.Tensor]:
        """Rows [0, R) of ``tokens`` at positions pos0 ..: fills caches and states; logits of the rows in ``want``.
        ``trace`` collects the stream after every layer run."""
        t, s = self.t, self.spec
        self.pdl = self.early(R)
        self._window()
        for i in range(-(-R // self.C)):
            self.pos[i:i + 1].fill_(pos0 + i * self.C)
        wait = dict(embed=True)                         # what the next row kernel adds to the stream first
        for r in t.runs:
            d, run = r["layer"], r["run"]
            add = None if run.pass_start is None else t.loop_step[run.pass_start]
            self._rows(R, add=add, pre=d["norm1"], copy=d["norm1"] is None and d["kind"] != "wkv", **wait)
            for n, p in self._chunks(R, pos0):
                MIXERS[d["kind"]].run(self, r, n, p)
            wait = dict(y=self.y, post=d["norm1b"])
            if d["kind"] == "parallel":
                wait.update(y2=self.y2, join=(d["out"], d["out2"]))
            f = d["spec"].mlp
            if f is not None:
                self._rows(R, pre=d["norm2"], copy=d["norm2"] is None, **wait)
                wait = dict(y=self._feed_forward(d, R), post=d["norm2b"], moe=f.routing if f.kind == "moe" else None)
            if trace is not None:
                self._rows(R, **wait)
                wait = {}
                trace.append(self.x[:R].clone())
        if not len(want):
            return None
        self._rows(R, pre=t.g_final, **wait)
        out = torch.empty(len(want), s.vocab, dtype=torch.float32, device=self.dev)
        straight = want == list(range(want[0], want[0] + len(want)))             # rows that follow one another
        idx = None if straight else torch.as_tensor(want, dtype=torch.long, device=self.dev)
        for i in range(0, len(want), self.head_rows):
            n = min(self.head_rows, len(want) - i)
            rows = self.h[want[0] + i:want[0] + i + n] if idx is None else self.h.index_select(0, idx[i:i + n])
            if not self.f32:                             # (one tensor map for all prompts)
                rows = self.hw[:n].copy_(rows)
            self.gemm(S.EPI_STORE, t.head, rows if self.f32 else self.hw, self.h_ld, n, out[i:i + n], s.vocab, scale=s.logit_scale)
        return out

    # ------------------------------------------------------------------ public API (that of ``NativePrefill``)
    def extend(self, tokens: torch.Tensor, pos0: int, want: Sequence[int] = (), trace: Optional[list] = None) -> torch.Tensor:
        """Feed ``tokens`` (host or device) at positions pos0 .. in spans of chunks; logits [len(want), vocab] of the rows in ``want``.
        ``trace`` collects, chunk by chunk, the stream after every layer run."""
        n = int(tokens.numel())
        if not 0 <= pos0 <= pos0 + n <= self.t.capacity:
            raise ValueError(f"rows [{pos0}, {pos0 + n}) outside the cache capacity {self.t.capacity}")
        out: List[torch.Tensor] = []
        order = list(want)
        if order != sorted(order):
            raise ValueError("wanted rows must ascend")
        self._fit_span(n)
        for c0 in range(0, n, self.span):
            R = min(self.span, n - c0)
            self.tokens[:R].copy_(tokens[c0:c0 + R].to(torch.int32), non_blocking=True)
            seen: Optional[list] = None if trace is None else []
            rows = map(int, order[bisect_left(order, c0):bisect_left(order, c0 + R)])
            got = self._chunk(pos0 + c0, R, [w - c0 for w in rows] if c0 else list(rows), seen)
            for i in range(0, R if seen else 0, self.C):
                trace.extend(x[i:i + self.C] for x in seen)
            if got is not None:
                out.append(got)
        return out[0] if len(out) == 1 else torch.cat(out) if out else torch.empty(0, self.spec.vocab, dtype=torch.float32, device=self.dev)

    def run(self, prompt: torch.Tensor, start: int = 0, end: Optional[int] = None) -> int:
        n = int(prompt.numel())
        end = n if end is None else end
        if not 0 <= start <= end <= n or end > self.t.capacity:
            raise ValueError(f"prefill range [{start}, {end}) outside the prompt / cache capacity")
        ev = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        self._fit_span(end - start)
        ev[0].record()
        self.extend(prompt[start:end], start)
        ev[1].record()
        self.phases = {"chunks": -(-(end - start) // self.C), "rows": end - start, "events": ev}
        return end

    def executor_ms(self) -> float:
        a, b = self.phases["events"]
        b.synchronize()
        return a.elapsed_time(b)

    def warm_chunks(self, sizes=None) -> None:
        """Run row counts once at position 0 (module loading, kernel attributes, scratch); the next request overwrites the rows.  The
        default ends with the longest span: its products of the routed experts are others than a chunk's."""
        for r in sorted(set(sizes or [1, self.C, self.span_limit])):
            self._fit_span(min(r, self.t.capacity))
            self.tokens.zero_()
            self._chunk(0, min(r, self.span, self.t.capacity))
        torch.cuda.current_stream().synchronize()
        self.check()

    def check(self) -> None:
        self.t.fab.check()

    def close(self) -> None:
        self.maps.clear()
        self._kept.clear()
