"""Layer-stack models without a GPU: configuration, tensor lists, order of runs, refusals, the plain implementation's own
invariants, the trace replay logic."""
import io
import json
import math
import os
import struct
from types import SimpleNamespace

import pytest
import torch

import tumatar_oracle as oracle
from naivert_b200.models import tumatar
from naivert_b200.models.blocks import LoopSpec, StackSpec
from naivert_b200.models.registry import MODELS, design_of, resolve_checkpoint_model, resolve_model, spec_from_config


def small():
    spec = tumatar.small_spec()
    return spec, tumatar.config_from_spec(spec)


def test_configuration_round_trip_and_registry():
    spec, cfg = small()
    again = spec_from_config(json.loads(json.dumps(cfg)), spec.name)
    assert again == spec and resolve_model("tumatar-small") == spec and design_of(spec) is tumatar
    assert {"tumatar-small", "tumatar-bench", "tumatar-bench-dense"} <= set(MODELS)
    with pytest.raises(KeyError, match="no registered model"):
        spec_from_config({"architecture": "Nobody"})
    for name in ("naive-n0.5", "small-w8a8"):
        assert not isinstance(resolve_model(name), StackSpec)


def test_speculative_target_is_found_by_its_config():
    from naivert_b200.models.checkpoint import target_config
    spec = resolve_model("naive-n0.5")
    assert spec_from_config(target_config(spec)) is spec


def test_order_of_layer_runs():
    spec, cfg = small()
    got = [(r.layer, r.pass_start) for r in spec.runs()]
    assert got == [(0, None), (1, 0), (2, None), (1, 1), (2, None), (3, None)] == oracle.layer_order(cfg)
    assert [r.run for r in spec.runs()] == list(range(6))
    assert [r.layer for r in spec.with_layers(2).runs()] == [0, 1]            # a loop that would be cut is dropped
    no_loop = dict(cfg, loop=None)
    assert [r.layer for r in spec_from_config(no_loop).runs()] == [0, 1, 2, 3]


@pytest.mark.parametrize("change,message", [
    (lambda c: c["layers"][0]["mixer"].update(blocks=7), "does not split into blocks"),
    (lambda c: c["layers"][0].update(type="other"), "unknown layer type"),
    (lambda c: c["layers"][0]["mlp"].update(kind="other"), "unknown feed-forward"),
    (lambda c: c["layers"][0]["mlp"]["router"].update(experts=300), "router of 300 experts"),
    (lambda c: c["layers"][0]["mlp"]["router"].update(groups={"count": 5, "keep": 1}), "expert groups"),
    (lambda c: c["layers"][0]["mlp"]["router"].update(top=13, groups={"count": 4, "keep": 2}), "fewer eligible experts"),
    (lambda c: c["layers"][1]["mixer"].update(dim=600), "head width"),
    (lambda c: c.update(loop={"start": 2, "stop": 2, "times": 1}), "loop bounds"),
])
def test_what_the_kernels_cannot_run_is_refused_by_name(change, message):
    _, cfg = small()
    change(cfg)
    with pytest.raises(ValueError, match=message):
        spec_from_config(cfg)


def test_checkpoint_files(tmp_path):
    from naivert_b200.models.checkpoint import CheckpointError, load_stack_weights, write_stack_checkpoint
    spec, cfg = small()
    sd = tumatar.init_state_dict(spec, seed=3)
    write_stack_checkpoint(str(tmp_path), spec, state_dict=sd)
    found = resolve_checkpoint_model(str(tmp_path))
    assert found.layers == spec.layers and found.loop == spec.loop
    w = load_stack_weights(found, str(tmp_path))
    assert torch.equal(w["layers"][0]["mlp"]["gate"][5], sd["l0.mlp.e5.gate"]) and torch.equal(w["loop"], sd["loop.step"])
    assert torch.equal(w["layers"][3]["mix"]["dkv.norm"], sd["l3.mix.dkv.norm"]) and w["layers"][2]["mlp"] is None
    cfg["layers"][1]["mixer"]["kv_rank"] += 8
    with pytest.raises(CheckpointError, match="the configuration needs"):
        load_stack_weights(spec_from_config(cfg), str(tmp_path))
    cfg2 = tumatar.config_from_spec(spec)
    cfg2["layers"].append(cfg2["layers"][0])
    with pytest.raises(CheckpointError, match="lacks"):
        load_stack_weights(spec_from_config(cfg2), str(tmp_path))


def test_engine_refuses_what_the_family_has_not():
    from naivert_b200.runtime.engine import Engine, RuntimeContractError
    spec, _ = small()
    with pytest.raises(RuntimeContractError, match="one GPU"):
        Engine.build(spec, tp=2)
    with pytest.raises(RuntimeContractError, match="no draft"):
        Engine.build(spec, draft_ckpt="somewhere")
    with pytest.raises(RuntimeContractError, match="32-bit"):
        Engine.build(resolve_model("small-w8a8"), dtype="fp32")
    assert spec.kv_bytes_per_token() == 3 * 112 * 2                          # three attention runs


def test_head_padding_keeps_the_products():
    from naivert_b200.runtime.packing import head_rows, pack
    w = torch.randn(3 * 5, 7)
    p = head_rows(w, 3, 5, 8)
    assert p.shape == (24, 7) and torch.equal(p.view(3, 8, 7)[:, :5], w.view(3, 5, 7)) and not p.view(3, 8, 7)[:, 5:].any()
    k = pack(w, "cpu")
    assert (k.z, k.n, k.ld, k.k) == (1, 15, 8, 7) and not k.w[:, :, 7].any()


def test_segment_bound_covers_every_distribution():
    """Segments needed by any split of the choices over the experts stay inside the list the chunk path allocates."""
    from naivert_b200.prefill.stack import StackPrefill
    rt = tumatar.small_spec().layers[0].mlp.routing
    g = torch.Generator().manual_seed(0)
    for rows in (1, 2, 7, 64, 300):
        for ir in (64, 128):
            bound = StackPrefill._items(None, rows, rt, ir)
            worst = 0
            for trial in range(40):
                p = torch.rand(rt.expert_count, generator=g) ** (trial % 9)
                ids = torch.multinomial(p.expand(rows, -1), rt.top_k, generator=g).flatten()
                n = torch.bincount(ids, minlength=rt.expert_count)
                worst = max(worst, int((-(-n // ir)).sum()))
            assert worst <= bound


def test_server_chooses_the_model_by_the_checkpoint(tmp_path):
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "examples"))
    import serve_sessions
    spec, cfg = small()
    (tmp_path / "config.json").write_text(json.dumps(cfg))
    assert serve_sessions.choose_model(None, str(tmp_path)).layers == spec.layers
    assert serve_sessions.choose_model("tumatar-small", None) is resolve_model("tumatar-small")
    assert serve_sessions.choose_model(None, None).name == "naive-n0.5"
    assert serve_sessions.parse_args(["--dtype", "fp32"]).dtype == "fp32"
    with pytest.raises(SystemExit):
        serve_sessions.main(["--model", "tumatar-small", "--log-level", "error"])          # neither a checkpoint nor --random-init


# --------------------------------------------------------------------------- the plain implementation
def test_plain_convolution_and_recurrence_by_hand():
    x = torch.tensor([[1.0], [2.0], [3.0]], dtype=torch.float64)
    k, b = torch.tensor([[10.0, 1.0]], dtype=torch.float64), torch.tensor([0.5], dtype=torch.float64)
    assert oracle.causal_conv(x, k, b).flatten().tolist() == [1.5, 12.5, 23.5]
    w = {"y": torch.zeros(1, 1), "y.b": torch.tensor([1.0]), "x": torch.ones(1, 1), "x.b": torch.zeros(1), "conv": torch.ones(1, 1),
         "conv.b": torch.zeros(1), "ra": torch.zeros(1, 1, 1), "ra.b": torch.zeros(1, 1), "ri": torch.zeros(1, 1, 1), "ri.b": torch.zeros(1, 1),
         "lam": torch.zeros(1), "o": torch.ones(1, 1)}
    w = {n: t.double() for n, t in w.items()}
    out = oracle.rglru(torch.tensor([[1.0], [2.0]]).double(), w, "", {"width": 1, "blocks": 1})
    a = math.exp(-8 * 0.5 * math.log(2.0))
    y = float(oracle.gelu_tanh(torch.tensor(1.0, dtype=torch.float64)))
    drive = math.sqrt(1 - a * a) * 0.5
    assert torch.allclose(out.flatten(), torch.tensor([drive * y, (a * drive + 2 * drive) * y], dtype=torch.float64))


def test_plain_choice_by_hand():
    eye = torch.eye(6).double()
    w = {"router": eye, "correction": torch.tensor([0.0, 0.0, -3.0, -3.0, 0.4, -2.0]).double()}
    z = torch.tensor([[0.0, 0.1, 5.0, 4.0, 0.0, 0.2]]).double()
    r = {"experts": 6, "top": 2, "groups": {"count": 3, "keep": 1}}
    ids, ws = oracle.route(z, w, "", r)
    assert ids == [[1, 0]]                                                   # pair scores: 1.02, about -4, about -0.5
    assert [round(float(v), 6) for v in ws[0]] == [round(1 / (1 + math.exp(-0.1)), 6), 0.5]      # weights without the correction
    ids, _ = oracle.route(z, w, "", dict(r, groups={"count": 3, "keep": 3}))
    assert ids == [[4, 1]]


def test_plain_model_is_causal():
    spec, cfg = small()
    sd = tumatar.init_state_dict(spec, seed=1)
    g = torch.Generator().manual_seed(2)
    toks = torch.randint(0, spec.vocab, (9,), generator=g).tolist()
    full = oracle.forward(cfg, sd, toks)
    assert torch.allclose(full[:6], oracle.forward(cfg, sd, toks[:6]))
    assert torch.isfinite(full).all() and full.std() > 1e-3


# --------------------------------------------------------------------------- tiles and spans of prompt chunks
def test_token_rows_per_tile():
    """One tile for few rows only where it was the faster one; everywhere else the widest tile that fills the SMs."""
    from naivert_b200.ops import stack_kernels as S
    from naivert_b200.prefill.stack import StackPrefill
    rule = StackPrefill.tile_rows
    functions = (S.EPI_TANH, S.EPI_DECAY_SOFT, S.EPI_DECAY_EXP)
    for epi in (S.EPI_STORE, S.EPI_BIAS, S.EPI_RELU2, S.EPI_CLAMPED_GLU, S.EPI_TRANSPOSE) + functions:
        for rows in (1, 64):
            assert [rule(epi, tiles, rows) for tiles in (1, 64, 75, 128, 1192)] == [64] * 5
    for epi in (S.EPI_TRANSPOSE,) + functions:                   # no sizes between: 64 feature tiles keep tiles of 64
        assert [rule(epi, 64, rows) for rows in (65, 128, 129, 256)] == [64] * 4
        assert [rule(epi, 96, rows) for rows in (65, 256)] == ([256] * 2 if epi == S.EPI_TRANSPOSE else [64] * 2)
        assert [rule(epi, 128, rows) for rows in (65, 256)] == [256] * 2
    for epi in (S.EPI_STORE, S.EPI_BIAS, S.EPI_RELU2):
        assert [rule(epi, 64, rows) for rows in (65, 128, 129, 187, 256)] == [64, 64, 128, 128, 128]
        assert [rule(epi, 80, rows) for rows in (65, 128, 129, 187, 256)] == [128, 128, 192, 192, 256]
    assert [rule(S.EPI_CLAMPED_GLU, 64, rows) for rows in (100, 187)] == [64, 128]
    assert [rule(S.EPI_CLAMPED_GLU, 128, rows) for rows in (100, 187, 256)] == [128, 192, 128]


@pytest.mark.parametrize("want", [[3, 3, 5], torch.tensor([3, 3, 5]), (torch.tensor(3), 3, 5), torch.tensor([0, 4, 4, 4, 9, 11]), torch.tensor([[2], [2], [4]])])
def test_wanted_rows_of_any_kind_are_plain_numbers(want):
    """Rows equal as numbers count as repeated whatever holds them: elements of a tensor hash by identity."""
    from naivert_b200.prefill.stack import StackPrefill
    seen = []

    class Fake(StackPrefill):
        def __init__(self):
            self.t, self.C, self.span, self.tokens = SimpleNamespace(capacity=64), 8, 8, torch.zeros(8, dtype=torch.int32)

        def _fit_span(self, n):
            pass

        def _chunk(self, pos0, R, want, trace):
            seen.append(want)
            return torch.tensor([float(pos0 + w) for w in want]).view(-1, 1) if want else None

    got = Fake().extend(torch.zeros(12, dtype=torch.int32), 0, want)
    assert got.flatten().tolist() == [float(w) for w in want]
    assert all(type(w) is int for rows in seen for w in rows)


def test_buffers_of_a_shorter_span_are_given_back(monkeypatch):
    """Tensor maps of token rows hold their tensors: those of buffers that a longer span replaces go with them, weights' stay."""
    import weakref
    from naivert_b200.ops import stack_kernels as S
    from naivert_b200.prefill.stack import StackPrefill
    spec = tumatar.small_spec()
    monkeypatch.setattr(S, "token_map", lambda t, *shape: SimpleNamespace(tensor=t))
    pf = object.__new__(StackPrefill)
    pf.__dict__.update(spec=spec, C=8, dev="cpu", act=torch.bfloat16, h_ld=spec.hidden, _kept={}, maps={("w", 1): "weight"},
                       t=SimpleNamespace(layers=[{"spec": layer, "kind": layer.mixer.kind} for layer in spec.layers]))
    pf._size_span(8)
    old = []
    for chunks in (2, 3):
        for t in (pf.h, pf.sorted, pf.ea):
            pf._xmap(t, 8, 1, 0, 8, 8, 64, 0)
        old += [weakref.ref(t) for t in (pf.h, pf.sorted, pf.ea, pf.ey, pf.x)]
        del t
        pf._size_span(8 * chunks)
        assert all(r() is None for r in old) and list(pf.maps) == [("w", 1)]


def test_spans_grow_with_the_prompt_as_far_as_memory_goes(monkeypatch):
    from naivert_b200.prefill.stack import StackPrefill
    sized = []

    class Fake(StackPrefill):
        def __init__(self, room):
            self.C, self.span, self.span_limit, self.dev, self.room = 4, 4, 16, "cuda", room

        def _size_span(self, P):
            sized.append(P)
            if P > self.room:
                raise torch.OutOfMemoryError("no room")
            self.span = P

    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    pf = Fake(100)
    for n, span in ((1, 4), (4, 4), (5, 8), (3, 8), (1000, 16)):
        pf._fit_span(n)
        assert pf.span == span
    assert sized == [8, 16]
    sized.clear()
    pf = Fake(8)
    for n, span in ((3, 4), (13, 8), (1000, 8)):                # what does not fit is tried once
        pf._fit_span(n)
        assert pf.span == span
    assert sized == [16, 12, 8]


# --------------------------------------------------------------------------- trace replay
class FakeEngine:
    def __init__(self):
        self.log, self.seq = [], []

    def reset(self):
        self.log.append("reset")
        self.seq = []

    def extend(self, tokens, want=()):
        base = len(self.seq)
        self.seq += list(tokens)
        self.log.append((tuple(tokens), tuple(want)))
        return torch.tensor([[float(base + w), float(self.seq[base + w])] for w in want]).view(len(want), 2)

    def close(self):
        self.log.append("close")


def test_trace_steps_map_to_engine_calls(tmp_path, monkeypatch, capsys):
    from naivert_b200.runtime import trace_run
    fake = FakeEngine()
    monkeypatch.setattr(trace_run, "build_engine", lambda model, dtype, n: fake)
    lines = [{"step": 0, "entries": [{"id": "a", "tokens": [4, 5, 6], "want": [2, 0]}], "end": []},
             {"step": 1, "entries": [{"id": "a", "tokens": [7], "want": []}], "end": ["a"]},
             {"step": 2, "entries": [{"id": "b", "tokens": [8, 9], "want": [1]}], "end": ["b"]}]
    monkeypatch.setattr("sys.stdin", io.StringIO("\n".join(json.dumps(x) for x in lines) + "\n"))
    assert trace_run.main(["--model", "m", "--out", str(tmp_path / "o"), "--max-tokens", "8"]) == 0
    assert capsys.readouterr().out.splitlines() == ["done 0", "done 1", "done 2"]
    assert fake.log[-1] == "close" and [x for x in fake.log if isinstance(x, tuple)] == [((4, 5, 6), (0, 2)), ((7,), ()), ((8, 9), (1,))]
    assert struct.unpack("<4f", (tmp_path / "o" / "0.f32").read_bytes()) == (2.0, 6.0, 0.0, 4.0)
    assert struct.unpack("<2f", (tmp_path / "o" / "2.f32").read_bytes()) == (1.0, 9.0)
    assert sorted(os.listdir(tmp_path / "o")) == ["0.f32", "2.f32"]


def test_trace_refuses_a_second_live_request(tmp_path):
    from naivert_b200.runtime.trace_run import TraceError, TraceRunner
    r = TraceRunner(FakeEngine(), str(tmp_path))
    r.step({"step": 0, "entries": [{"id": "a", "tokens": [1], "want": []}], "end": []})
    with pytest.raises(TraceError, match="one sequence"):
        r.step({"step": 1, "entries": [{"id": "b", "tokens": [1], "want": []}], "end": []})
