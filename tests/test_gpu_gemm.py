"""tcgen05 skinny GEMM engine vs the fp32 torch oracle of the same op (single GPU, tp=1)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup():
    from naivert_b200.ops import kernels as K
    K.lib()
    return K


def _status():
    return torch.zeros(4, dtype=torch.int32, device="cuda")


def _packet(x, K):
    from naivert_b200.ops.quant import quantize_act_pow2
    r, k = x.shape
    x8 = torch.zeros(16, k, dtype=torch.uint8, device="cuda")
    xs = torch.ones(16, k // 128, dtype=torch.float32, device="cuda")
    q, s = quantize_act_pow2(x)
    x8[:r] = q.view(torch.uint8)
    xs[:r] = s
    return x8, xs


def _fab(K, status, epoch, features):
    f = K.FabricArgs()
    f.epoch = epoch.data_ptr()
    f.status = status.data_ptr()
    f.tp, f.rank, f.call_idx, f.features = 1, 0, 0, features
    f.timeout_ns = 1_000_000_000
    return f


@pytest.mark.parametrize("rows,n,k", [(8, 512, 1024), (1, 256, 256), (16, 1024, 4096)])
def test_fp8_linear_store(rows, n, k):
    K = _setup()
    from naivert_b200.ops.quant import quantize_fp8_block, w8a8_linear_ref
    g = torch.Generator(device="cuda").manual_seed(1)
    w = torch.randn(n, k, device="cuda", generator=g) * 0.05
    x = (torch.randn(rows, k, device="cuda", generator=g)).bfloat16().float()
    w8, ws = quantize_fp8_block(w)
    x8, xs = _packet(x, K)
    out = torch.zeros(rows, n, device="cuda")
    st = _status()
    a = K.GemmArgs()
    a.n_total, a.k_total, a.rows, a.a_group = n, k, rows, 0
    a.w_scale0, a.a_scale = ws.data_ptr(), xs.data_ptr()
    a.out_f32, a.ld_out, a.out_scale = out.data_ptr(), n, 1.0
    a.status = st.data_ptr()
    tmA, tmB = K.weight_tmap(w8.view(torch.uint8)), K.act_tmap(x8)
    K.gemm(K.gemm_variant(True, False, K.EPI_STORE_F32, K.GROUP_NONE), tmA, None, tmB, a, n // 128)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    ref = w8a8_linear_ref(x, w8, ws)
    err = (out - ref).abs().max().item()
    assert err <= 1e-4 * ref.abs().max().item() + 1e-6, err


def test_bf16_linear_store():
    K = _setup()
    g = torch.Generator(device="cuda").manual_seed(2)
    rows, n, k = 8, 640, 1024                       # 640 = 5 tiles
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    x = torch.zeros(16, k, device="cuda", dtype=torch.bfloat16)
    x[:rows] = torch.randn(rows, k, device="cuda", generator=g).bfloat16()
    out = torch.zeros(rows, n, device="cuda")
    st = _status()
    a = K.GemmArgs()
    a.n_total, a.k_total, a.rows = n, k, rows
    a.out_f32, a.ld_out, a.out_scale = out.data_ptr(), n, 1.0
    a.status = st.data_ptr()
    K.gemm(K.gemm_variant(False, False, K.EPI_STORE_F32, K.GROUP_NONE), K.weight_tmap(w), None, K.act_tmap(x), a, n // 128)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    ref = x[:rows].float() @ w.float().T
    assert (out - ref).abs().max().item() <= 2e-3 * ref.abs().max().item()


def test_fp8_allreduce_tp1_residual():
    K = _setup()
    from naivert_b200.ops.quant import quantize_fp8_block, w8a8_linear_ref
    g = torch.Generator(device="cuda").manual_seed(3)
    rows, n, k = 8, 1024, 512
    w8, ws = quantize_fp8_block(torch.randn(n, k, device="cuda", generator=g) * 0.05)
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16().float()
    resid = torch.randn(rows, n, device="cuda", generator=g).bfloat16()
    x8, xs = _packet(x, K)
    out = torch.zeros(rows, n, device="cuda", dtype=torch.bfloat16)
    st, epoch = _status(), torch.ones(1, dtype=torch.int32, device="cuda")
    a = K.GemmArgs()
    a.n_total, a.k_total, a.rows = n, k, rows
    a.w_scale0, a.a_scale = ws.data_ptr(), xs.data_ptr()
    a.out_bf16, a.ld_out, a.resid = out.data_ptr(), n, resid.data_ptr()
    a.fab = _fab(K, st, epoch, n)
    a.status = st.data_ptr()
    K.gemm(K.gemm_variant(True, False, K.EPI_ALLREDUCE, K.GROUP_NONE), K.weight_tmap(w8.view(torch.uint8)), None,
           K.act_tmap(x8), a, n // 128)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    ref = (resid.float() + w8a8_linear_ref(x, w8, ws).bfloat16().float()).bfloat16()
    diff = (out.float() - ref.float()).abs()
    assert diff.max().item() <= 0.02 * ref.float().abs().max().item()
    assert (diff > 0).float().mean().item() < 0.01       # at most rare 1-ulp flips


def test_moe_gate_up_down_grouped():
    """Grouped gate/up (SiLU + e4m3 requantisation) followed by the probability-weighted down
    projection, against the W8A8 recipe evaluated in torch."""
    K = _setup()
    from naivert_b200.ops.quant import quantize_act_pow2, quantize_fp8_block, w8a8_linear_ref
    g = torch.Generator(device="cuda").manual_seed(4)
    E, H, I, rows, slots = 8, 512, 256, 8, 5
    gate = torch.randn(E, I, H, device="cuda", generator=g) * 0.05
    up = torch.randn(E, I, H, device="cuda", generator=g) * 0.05
    down = torch.randn(E, H, I, device="cuda", generator=g) * 0.05
    g8, gs = quantize_fp8_block(gate)
    u8, us = quantize_fp8_block(up)
    d8, ds = quantize_fp8_block(down)
    x = torch.randn(rows, H, device="cuda", generator=g).bfloat16().float()
    x8, xs = _packet(x, K)
    active = torch.tensor([1, 2, 4, 6, 7, 0, 0, 0], dtype=torch.int32, device="cuda")
    n_active = torch.tensor([slots], dtype=torch.int32, device="cuda")
    probs = torch.zeros(8, 16, device="cuda")
    probs[:slots, :rows] = torch.rand(slots, rows, device="cuda", generator=g)
    probs[1, 3] = 0.0
    y8 = torch.zeros(8 * 16, I, dtype=torch.uint8, device="cuda")
    ys = torch.ones(8 * 16, I // 128, device="cuda")
    st, epoch = _status(), torch.ones(1, dtype=torch.int32, device="cuda")

    a = K.GemmArgs()
    a.n_total, a.k_total, a.rows = I, H, rows
    a.n_active, a.active_ids, a.max_slots = n_active.data_ptr(), active.data_ptr(), 8
    a.w_scale0, a.w_scale1, a.a_scale = gs.data_ptr(), us.data_ptr(), xs.data_ptr()
    a.out_q, a.out_qscale = y8.data_ptr(), ys.data_ptr()
    a.status = st.data_ptr()
    K.gemm(K.gemm_variant(True, True, K.EPI_SILU_QUANT, K.GROUP_ITEM), K.weight_tmap(g8.view(torch.uint8)),
           K.weight_tmap(u8.view(torch.uint8)), K.act_tmap(x8), a, I // 128, 8)

    resid = torch.randn(rows, H, device="cuda", generator=g).bfloat16()
    out = torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16)
    b = K.GemmArgs()
    b.n_total, b.k_total, b.rows = H, I, rows
    b.n_active, b.active_ids, b.probs, b.max_slots = n_active.data_ptr(), active.data_ptr(), probs.data_ptr(), 8
    b.n_experts = E
    b.w_scale0, b.a_scale = ds.data_ptr(), ys.data_ptr()
    b.out_bf16, b.ld_out, b.resid = out.data_ptr(), H, resid.data_ptr()
    b.fab = _fab(K, st, epoch, H)
    b.status = st.data_ptr()
    K.gemm(K.gemm_variant(True, False, K.EPI_ALLREDUCE, K.GROUP_LOOP), K.weight_tmap(d8.view(torch.uint8)), None,
           K.act_tmap(y8), b, H // 128, 1)
    torch.cuda.synchronize()
    assert int(st[0]) == 0

    mix = torch.zeros(rows, H, device="cuda")
    for s in range(slots):
        e = int(active[s])
        gg = w8a8_linear_ref(x, g8[e], gs[e])
        uu = w8a8_linear_ref(x, u8[e], us[e])
        y = torch.nn.functional.silu(gg) * uu
        yq, ysc = quantize_act_pow2(y)
        got_q = y8[s * 16:s * 16 + rows].view(torch.float8_e4m3fn).float() * ys[s * 16:s * 16 + rows].repeat_interleave(128, 1)
        want_q = yq.float() * ysc.repeat_interleave(128, 1)
        assert (got_q - want_q).abs().max().item() <= 0.07 * want_q.abs().max().item()   # one e4m3 step
        assert ((got_q - want_q).abs() > 0).float().mean().item() < 0.02
        mix += probs[s, :rows, None] * w8a8_linear_ref(y, d8[e], ds[e])
    ref = (resid.float() + mix.bfloat16().float()).bfloat16().float()
    assert (out.float() - ref).abs().max().item() <= 0.02 * ref.abs().max().item()


def test_prep_norm_packet():
    K = _setup()
    from naivert_b200.ops.quant import quantize_act_pow2
    g = torch.Generator(device="cuda").manual_seed(5)
    rows, H = 8, 1024
    x = torch.randn(16, H, device="cuda", generator=g).bfloat16()
    gamma = (1 + 0.05 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    xn = torch.empty(16, H, device="cuda", dtype=torch.bfloat16)
    x8 = torch.empty(16, H, device="cuda", dtype=torch.uint8)
    xs = torch.empty(16, H // 128, device="cuda")
    K.prep_norm(x, gamma, rows, 1e-5, xn, x8, xs, pdl=False)
    torch.cuda.synchronize()
    xf = x[:rows].float()
    ref = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * gamma.float()).bfloat16()
    d = (xn[:rows].float() - ref.float()).abs()
    assert d.max().item() <= 0.01 * ref.float().abs().max().item()
    q, s = quantize_act_pow2(xn[:rows].float())
    assert torch.equal(xs[:rows], s)
    assert torch.equal(x8[:rows], q.view(torch.uint8))
    assert int(xn[rows:].abs().sum()) == 0 and int(x8[rows:].sum()) == 0


def _items(n_items, step=64):
    off = (torch.arange(n_items, dtype=torch.int32, device="cuda") * step).contiguous()
    ids = torch.zeros(n_items, dtype=torch.int32, device="cuda")
    cnt = torch.tensor([n_items], dtype=torch.int32, device="cuda")
    return off, ids, cnt


@pytest.mark.parametrize("order", [False, True])
def test_chunk_gemm_bf16_matches_torch(order):
    """64-column persistent chunk GEMM (bf16, fp32 store) against torch on 320 rows x 640 features x K 1024."""
    K = _setup()
    g = torch.Generator(device="cuda").manual_seed(3)
    rows, n, k = 320, 640, 1024
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16()
    out = torch.zeros(rows, n, device="cuda")
    st = _status()
    off, ids, cnt = _items(rows // 64)
    a = K.GemmArgs()
    a.n_total, a.k_total, a.rows, a.out_scale = n, k, 64, 1.0
    a.n_active, a.active_ids, a.max_slots, a.row_offsets = cnt.data_ptr(), ids.data_ptr(), rows // 64, off.data_ptr()
    a.out_f32, a.ld_out, a.status = out.data_ptr(), n, st.data_ptr()
    K.wide_gemm(K.gemm_variant(False, False, K.EPI_STORE_F32, K.GROUP_ITEM), K.weight_tmap(w), None, K.act_tmap(x, 64), a,
                n // 128, rows // 64, items_fastest=order)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    ref = x.float() @ w.float().T
    assert (out - ref).abs().max().item() <= 2e-3 * ref.abs().max().item()


@pytest.mark.parametrize("n,k", [(640, 1024), (9600, 192), (18944, 64)])
@pytest.mark.parametrize("rows", [1, 63, 64, 65, 187, 320])
def test_chunk_projection(rows, n, k):
    """bf16 projections of a chunk (rows of a wider buffer, fp32 and bf16 stores) at the edges of 64- and 256-row tiles; rows past the
    chunk's are left alone.  Products are exact in fp32: a sum of k of them is off by at most k half steps of 2^-24, doubled for the
    tensor unit's truncation."""
    from types import SimpleNamespace
    from naivert_b200.prefill.native import NativePrefill
    K = _setup()
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).bfloat16()
    x = torch.randn(384, k + 64, device="cuda", generator=g).bfloat16()[:, 64:]
    st, wm = _status(), K.weight_tmap(w)
    owner = SimpleNamespace(wide=True, _bf16={})
    ref, size = x[:rows].double() @ w.double().T, x[:rows].double().abs() @ w.double().abs().T
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.full((384, n), 7.0, device="cuda", dtype=dtype)
        a = K.GemmArgs()
        a.n_total, a.k_total, a.out_scale, a.ld_out, a.status = n, k, 1.0, n, st.data_ptr()
        setattr(a, "out_f32" if dtype == torch.float32 else "out_bf16", out.data_ptr())
        owner._bf16 = {}
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            NativePrefill._bf16_gemm(owner, 0, wm, x, a, n // 128, rows, 0, False)
        torch.cuda.synchronize()
        assert int(st[0]) == 0
        bound = 2 * k * 2.0 ** -24 * size + (0 if dtype == torch.float32 else 2.0 ** -8 * ref.abs())
        assert bool(((out[:rows].double() - ref).abs() <= bound).all())
        assert bool((out[rows:] == 7).all())


def test_chunk_gemm_fp8_gate_up_matches_torch():
    """e4m3 block-scaled gate/up with SiLU and e4m3 re-quantisation on the chunk engine vs the torch recipe."""
    K = _setup()
    from naivert_b200.ops.quant import dequant_act, quantize_act_pow2, quantize_fp8_block, w8a8_linear_ref
    g = torch.Generator(device="cuda").manual_seed(4)
    rows, n, k = 192, 256, 1024
    wg = torch.randn(n, k, device="cuda", generator=g) * 0.05
    wu = torch.randn(n, k, device="cuda", generator=g) * 0.05
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16().float()
    g8, gs = quantize_fp8_block(wg)
    u8, us = quantize_fp8_block(wu)
    xq, xs = quantize_act_pow2(x)
    x8 = xq.view(torch.uint8).contiguous()
    xs = xs.float().contiguous()
    y8 = torch.zeros(rows, n, dtype=torch.uint8, device="cuda")
    ys = torch.zeros(rows, n // 128, device="cuda")
    st = _status()
    off, ids, cnt = _items(rows // 64)
    a = K.GemmArgs()
    a.n_total, a.k_total, a.rows, a.out_scale = n, k, 64, 1.0
    a.n_active, a.active_ids, a.max_slots, a.row_offsets = cnt.data_ptr(), ids.data_ptr(), rows // 64, off.data_ptr()
    a.w_scale0, a.w_scale1, a.a_scale = gs.data_ptr(), us.data_ptr(), xs.data_ptr()
    a.out_q, a.out_qscale, a.status = y8.data_ptr(), ys.data_ptr(), st.data_ptr()
    K.wide_gemm(K.gemm_variant(True, True, K.EPI_SILU_QUANT, K.GROUP_ITEM), K.weight_tmap(g8.view(torch.uint8)),
                K.weight_tmap(u8.view(torch.uint8)), K.act_tmap(x8, 64), a, n // 128, rows // 64)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    gg, uu = w8a8_linear_ref(x, g8, gs), w8a8_linear_ref(x, u8, us)
    want = torch.nn.functional.silu(gg) * uu
    got = dequant_act(y8.view(torch.float8_e4m3fn), ys)
    # one e4m3 rounding of the reference value (relative step 2^-3, half of it as error) plus accumulation noise
    assert (got - want).abs().max().item() <= 0.07 * want.abs().max().item()
    wq, wsc = quantize_act_pow2(want)
    assert torch.equal(ys, wsc.float()) or (ys - wsc.float()).abs().max().item() <= ys.max().item()


@pytest.mark.parametrize("k,n,rows", [(128, 128, 64), (256, 384, 64), (384, 256, 192), (1152, 128, 128), (4224, 256, 64), (640, 2048, 1024)])
def test_chunk_gemm_fp8_pairs_of_k_blocks(k, n, rows):
    """One, two, odd and many K blocks (accumulators change hands in pairs), more tiles than CTAs: e4m3 products against the torch
    recipe.  fp32 sums of k products of bf16-rounded outputs: 2^-8 of the value and k 2^-24 of the magnitudes."""
    K = _setup()
    from naivert_b200.ops.quant import dequant_act, quantize_act_pow2, quantize_fp8_block, w8a8_linear_ref
    g = torch.Generator(device="cuda").manual_seed(k + n)
    ws = [quantize_fp8_block(torch.randn(n, k, device="cuda", generator=g) * 0.05) for _ in range(2)]
    x = torch.randn(rows, k, device="cuda", generator=g).bfloat16().float()
    xq, xs = quantize_act_pow2(x)
    x8, xs = xq.view(torch.uint8).contiguous(), xs.float().contiguous()
    off, ids, cnt = _items(rows // 64)
    maps = [K.weight_tmap(w.view(torch.uint8)) for w, _ in ws]
    for dual in (False, True):
        out = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
        y8, ys, st = torch.zeros(rows, n, dtype=torch.uint8, device="cuda"), torch.zeros(rows, n // 128, device="cuda"), _status()
        a = K.GemmArgs()
        a.n_total, a.k_total, a.rows, a.out_scale = n, k, 64, 1.0
        a.n_active, a.active_ids, a.max_slots, a.row_offsets = cnt.data_ptr(), ids.data_ptr(), rows // 64, off.data_ptr()
        a.w_scale0, a.w_scale1, a.a_scale = ws[0][1].data_ptr(), ws[1][1].data_ptr(), xs.data_ptr()
        a.out_q, a.out_qscale, a.out_bf16, a.ld_out, a.status = y8.data_ptr(), ys.data_ptr(), out.data_ptr(), n, st.data_ptr()
        K.wide_gemm(K.gemm_variant(True, dual, K.EPI_SILU_QUANT if dual else K.EPI_STORE_BF16, K.GROUP_ITEM), maps[0], maps[1] if dual else None,
                    K.act_tmap(x8, 64), a, n // 128, rows // 64)
        torch.cuda.synchronize()
        assert int(st[0]) == 0
        gate, up = (w8a8_linear_ref(x, w, s) for w, s in ws)
        if dual:
            want = torch.nn.functional.silu(gate) * up
            assert (dequant_act(y8.view(torch.float8_e4m3fn), ys) - want).abs().max().item() <= 0.07 * want.abs().max().item()
        else:
            slack = k * 2.0 ** -24 * dequant_act(xq, xs).abs().max() * k ** 0.5
            assert ((out.float() - gate).abs() <= 2.0 ** -8 * gate.abs() + slack).all()


@pytest.mark.parametrize("k", [15360, 15488, 16384])
def test_chunk_gemm_fp8_longest_rows(k):
    """The table of scales takes the room of a stage from two products of more than 15,360 channels."""
    test_chunk_gemm_fp8_pairs_of_k_blocks(k, 128, 64)
