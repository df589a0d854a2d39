"""tcgen05 / TMA GEMM and the fused LM-head statistics epilogue against PyTorch references."""
import math

import pytest
import torch

from mindspeed_rl_b200.ops import gemm as G
from mindspeed_rl_b200.ops import _lib
from mindspeed_rl_b200.ops._lib import c_float, c_int, c_ll, ptr, stream

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (300, 520, 192), (1024, 3584, 3584), (77, 1000, 4096)])
def test_gemm_bf16_tn(m, n, k):
    torch.manual_seed(0)
    a = (torch.randn(m, k, device=DEV) * 0.5).bfloat16()
    b = (torch.randn(n, k, device=DEV) * 0.5).bfloat16()
    c = G.gemm_bf16_tn(a, b)
    G.check_status(DEV)
    _assert_close(c, a.float() @ b.float().t(), k)


def _assert_close(c, ref, k, scale=0.25):
    """bf16 output of an fp32-accumulated product of entries of magnitude ~``sqrt(scale)``: the result
    has standard deviation ``scale * sqrt(k)`` and carries one bf16 rounding (relative 2^-8), so the
    band is 1 % relative plus 1 % of that standard deviation."""
    err = (c.float() - ref).abs()
    tol = 1e-2 * ref.abs() + 1e-2 * scale * (k ** 0.5)
    assert bool((err <= tol).all()), f"max err {err.max().item()} ref max {ref.abs().max().item()}"


PAIR_SHAPES = [(256, 256, 64), (128, 256, 128), (300, 520, 192), (1024, 3584, 3584), (77, 1000, 4096), (640, 72, 200)]


@pytest.mark.parametrize("m,n,k", PAIR_SHAPES)
def test_gemm_pair_forward_and_bias(m, n, k):
    torch.manual_seed(0)
    a = (torch.randn(m, k, device=DEV) * 0.5).bfloat16()
    b = (torch.randn(n, k, device=DEV) * 0.5).bfloat16()
    bias = torch.randn(n, device=DEV).bfloat16()
    ref = a.float() @ b.float().t()
    _assert_close(G.gemm_pair(a, b), ref, k)
    _assert_close(G.gemm_pair(a, b, bias=bias), ref + bias.float(), k)
    G.check_status(DEV)


@pytest.mark.parametrize("m,n,k,splits", [(256, 512, 2048, 4), (200, 1000, 4096, 5), (256, 3584, 18944, 5),
                                          (130, 264, 1536, 3), (64, 256, 640, 16)])
def test_gemm_pair_split_reduction(m, n, k, splits):
    """Small-M form: the reduction cut into pieces (including pieces of unequal length and more pieces
    asked for than the planner would give), partial tiles added in a fixed order, optional bias."""
    torch.manual_seed(2)
    a = (torch.randn(m, k, device=DEV) * 0.5).bfloat16()
    b = (torch.randn(n, k, device=DEV) * 0.5).bfloat16()
    bias = torch.randn(n, device=DEV).bfloat16()
    ref = a.float() @ b.float().t()
    out1 = G.gemm_pair_splitk(a, b, splits)
    _assert_close(out1, ref, k)
    _assert_close(G.gemm_pair_splitk(a, b, splits, bias=bias), ref + bias.float(), k)
    assert torch.equal(out1, G.gemm_pair_splitk(a, b, splits))      # fixed summation order
    G.check_status(DEV)


def test_linear_fwd_routes_decode_shapes():
    """256-token decode shapes: wide outputs on the plain pair kernel, long reductions on the split
    form, the rest on the library; all three agree with the fp32 product."""
    torch.manual_seed(3)
    for n, k in [(37888 // 8, 3584), (3584, 18944), (4608, 3584)]:
        x = (torch.randn(256, k, device=DEV) * 0.5).bfloat16()
        w = (torch.randn(n, k, device=DEV) * 0.5).bfloat16()
        _assert_close(G.linear_fwd(x, w), x.float() @ w.float().t(), k)
    assert G.splitk_plan(256, 3584, 18944) >= 2 and G.splitk_plan(256, 4608, 3584) == 0
    G.check_status(DEV)


@pytest.mark.parametrize("m,n,k", PAIR_SHAPES)
def test_gemm_pair_data_and_weight_gradient_forms(m, n, k):
    """``dy @ w`` with ``w`` as an MN-major B operand, and ``dy.T @ x`` with both operands MN-major,
    stored and accumulated into fp32 / bf16 gradient buffers."""
    torch.manual_seed(1)
    dy = (torch.randn(m, k, device=DEV) * 0.5).bfloat16()         # [T, N_lin] : reduction over its columns
    w = (torch.randn(k, n, device=DEV) * 0.5).bfloat16()          # [N_lin, K_lin] read as stored
    _assert_close(G.gemm_pair(dy, w, b_mn=True), dy.float() @ w.float(), k)
    t = k                                                          # tokens are the reduction of the weight gradient
    t8 = (t + 7) // 8 * 8
    g_out = (torch.randn(t8, m // 8 * 8 or 8, device=DEV) * 0.5).bfloat16()
    x_in = (torch.randn(t8, n // 8 * 8 or 8, device=DEV) * 0.5).bfloat16()
    ref = g_out.float().t() @ x_in.float()
    _assert_close(G.gemm_pair(g_out, x_in, a_mn=True, b_mn=True), ref, t8)
    for dt in (torch.float32, torch.bfloat16):
        base = torch.randn(ref.shape, device=DEV).to(dt)
        grad = base.clone()
        mode = "acc_f32" if dt == torch.float32 else "acc_bf16"
        G.gemm_pair(g_out, x_in, a_mn=True, b_mn=True, out=grad, mode=mode)
        G.gemm_pair(g_out, x_in, a_mn=True, b_mn=True, out=grad, mode=mode)
        _assert_close(grad, base.float() + 2 * ref, 4 * t8)
    G.check_status(DEV)


@pytest.mark.parametrize("m,f,k", [(129, 6144, 64), (256, 6200, 200), (300, 6168, 192), (1025, 8, 264), (2000, 1544, 1096)])
def test_gemm_pair_swiglu(m, f, k):
    """SwiGLU in the epilogue of the first MLP linear: the bits of the plain kernel followed by the SwiGLU kernel, with widths
    that end inside a tile of 128 and of 64 columns, and rows that end inside a tile."""
    from mindspeed_rl_b200 import ops
    torch.manual_seed(4)
    x = torch.randn(m, k, device=DEV).bfloat16()
    w = (0.2 * torch.randn(2 * f, k, device=DEV)).bfloat16()
    gate_up = G.gemm_pair(x, w)
    want = ops.swiglu_fwd(gate_up)
    L = _lib.load()
    for keep in (False, True):
        act = torch.full((m, f), 7.0, device=DEV).bfloat16()
        gu = torch.full((m, 2 * f), 7.0, device=DEV).bfloat16() if keep else None
        assert L.msrl_gemm_pair_swiglu(ptr(x), c_ll(k), ptr(w), c_ll(k), ptr(act), ptr(gu), c_int(m), c_int(f), c_int(k),
                                       ptr(G._status_word(x.device)), stream()) == 0
        G.check_status(DEV)
        assert torch.equal(act, want)
        if keep:
            assert torch.equal(gu, gate_up)
        got, got_gu = G.linear_swiglu(x, w, keep)
        assert (got_gu is None) == (not keep)
        _assert_close(got, torch.nn.functional.silu(gate_up[:, :f].float()) * gate_up[:, f:].float(), k)


@pytest.mark.parametrize("m,f,k,keep,launches", [(300, 6144, 896, False, 1), (300, 6144, 896, True, 2), (300, 6144, 1536, True, 1),
                                                 (256, 6144, 1536, True, 2), (256, 6144, 1536, False, 1)])
def test_linear_swiglu_in_one_kernel_where_it_is_the_faster_one(m, f, k, keep, launches):
    torch.manual_seed(4)
    x, w = torch.randn(m, k, device=DEV).bfloat16(), (k ** -0.5 * torch.randn(2 * f, k, device=DEV)).bfloat16()
    before = _lib.launch_count()
    act, gate_up = G.linear_swiglu(x, w, keep)
    assert _lib.launch_count() - before == launches and (gate_up is not None) == keep
    both = G.gemm_pair(x, w)
    assert not keep or torch.equal(gate_up, both)
    _assert_close(act, torch.nn.functional.silu(both[:, :f].float()) * both[:, f:].float(), 16)
    G.check_status(DEV)


@pytest.mark.parametrize("m", [1, 127, 128, 129, 256, 257, 300, 384, 385, 1409])
@pytest.mark.parametrize("v,k", [(1000, 264), (2500, 1800)])
def test_lmhead_stats_forms(m, v, k):
    """Row tiles of 256 on CTA pairs and of 128 on single CTAs write the same records, and the rule takes the latter where the
    last 256 rows are at most half full."""
    torch.manual_seed(6)
    h = torch.randn(m, k, device=DEV).bfloat16()
    w = (torch.randn(v, k, device=DEV) * k ** -0.5).bfloat16()
    labels = torch.randint(-5, v + 5, (m,), device=DEV)
    got, tiles = G.lmhead_stats(h, w, labels, 0.7)
    L = _lib.load()
    for kernel in (L.msrl_lmhead_stats, L.msrl_lmhead_stats_rows128):
        st = torch.full_like(got, 7.0)
        assert kernel(ptr(h), c_ll(k), ptr(w), c_ll(k), ptr(labels), c_int(0), c_float(0.7), ptr(st), c_int(m), c_int(v), c_int(k),
                      ptr(G._status_word(h.device)), stream()) == 0
        assert torch.equal(st, got)
    G.check_status(DEV)
    z = (h.float() @ w.float().t()).bfloat16().float() * 0.7
    pad = torch.full((m, tiles * 256 - v), -math.inf, device=DEV)
    # a logit that lies between two bf16 values may round either way: 2^-8 of it
    torch.testing.assert_close(got[:, :, 0].t(), torch.cat([z, pad], 1).view(m, tiles, 256).amax(-1), rtol=2 ** -7, atol=1e-3)
    assert [G._lmhead_rows128(n, 3584) for n in (1, 128, 129, 256, 300, 640, 1664)] == [True, True, False, False, True, True, False]


@pytest.mark.parametrize("n", [1, 4, 5, 32, 33, 600])
@pytest.mark.parametrize("t", [1, 31, 128, 129, 700])
def test_logprob_finish_record_counts(n, t):
    """One, four and sixteen warps to the records of 32 rows, on both sides of their borders, from records on a 16-byte boundary and
    beside one."""
    torch.manual_seed(7)
    st = torch.rand(n, t, 4, device=DEV) + 0.5
    st[..., 0] *= 5
    for base in (st, torch.cat([torch.zeros(1, device=DEV), st.view(-1)])[1:]):
        logp, ent, lse = (torch.full((t,), 9.0, device=DEV) for _ in range(3))
        assert _lib.load().msrl_logprob_finish(ptr(base), c_int(n), c_ll(t), ptr(logp), ptr(ent), ptr(lse), stream()) == 0
        d = st.double()
        c = torch.exp(d[..., 0] - d[..., 0].amax(0))
        s = (d[..., 1] * c).sum(0)
        want = d[..., 0].amax(0) + torch.log(s)
        # fp32 sums of up to 600 terms of one sign, exponentials and logarithm on the fast units
        torch.testing.assert_close(lse, want.float(), rtol=2e-6, atol=2e-6)
        torch.testing.assert_close(logp, (d[..., 2].sum(0) - want).float(), rtol=1e-5, atol=1e-5)
        torch.testing.assert_close(ent, (want - (d[..., 3] * c).sum(0) / s).float(), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("t,v,h", [(200, 1000, 256), (513, 5000, 896)])
def test_lmhead_stats_fused(t, v, h):
    torch.manual_seed(1)
    x = torch.randn(t, h, device=DEV).bfloat16()
    w = (0.05 * torch.randn(v, h, device=DEV)).bfloat16()
    y = torch.randint(0, v, (t,), device=DEV)
    stats, tiles = G.lmhead_stats(x, w, y, 1 / 0.7)
    G.check_status(DEV)
    logp = torch.empty(t, device=DEV)
    ent = torch.empty(t, device=DEV)
    lse = torch.empty(t, device=DEV)
    L = _lib.load()
    assert L.msrl_logprob_finish(ptr(stats), c_int(tiles), c_ll(t), ptr(logp), ptr(ent), ptr(lse), stream()) == 0
    z = (x.float() @ w.float().t()).bfloat16().float() / 0.7
    ls = torch.log_softmax(z, -1)
    ref_lp = ls.gather(-1, y[:, None])[:, 0]
    ref_ent = -(ls.exp() * ls).sum(-1)
    assert (logp - ref_lp).abs().max() < 3e-2, (logp - ref_lp).abs().max()
    assert (ent - ref_ent).abs().max() < 3e-2, (ent - ref_ent).abs().max()


@pytest.mark.parametrize("ml,k,n", [(128, 256, 256), (384, 512, 776), (1024, 1024, 1536)])
def test_fused_comm_gemm_single_rank(ml, k, n):
    """World size 1 exercises the comm warps, counters and tile order of both fused variants
    (self-gather, push to the own staging area) without a second GPU."""
    from mindspeed_rl_b200.parallel.fused_tp import FusedTP
    from mindspeed_rl_b200.parallel.symm import SymmetricArena

    torch.manual_seed(3)
    arena = SymmetricArena(8 * ml * max(k, n) * 2 + (8 << 20))
    try:
        f = FusedTP(arena, [0], ml, k, n)
        for call in range(3):
            x = (torch.randn(ml, k, device=DEV) * 0.5).bfloat16()
            w = (torch.randn(n, k, device=DEV) * 0.5).bfloat16()
            assert f.fits_ag(x, w) and f.fits_rs(x, w)
            y, xg = f.ag_gemm(x, w)
            G.check_status(x.device)
            assert torch.equal(xg, x)
            ref = x.float() @ w.float().t()
            assert bool(((y.float() - ref).abs() <= 2e-2 * ref.abs() + 0.25).all()), call
            out = f.gemm_rs(x, w)
            G.check_status(x.device)
            assert bool(((out.float() - ref).abs() <= 2e-2 * ref.abs() + 0.25).all()), call
        arena.check()
    finally:
        arena.close()


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("nh,nkv,interleaved", [(4, 2, True), (7, 1, False)])
def test_flash_attention_fwd_tcgen05(nh, nkv, interleaved, causal, monkeypatch):
    """tcgen05 forward attention against the fp32 oracle and the mma.sync kernel: ragged packed
    sequences that end inside a key tile, one longer than several tiles, a single token."""
    from mindspeed_rl_b200 import ops
    from mindspeed_rl_b200.ops.layouts import QKVLayout
    torch.manual_seed(11)
    lay = QKVLayout(nh, nkv, 128, interleaved)
    lens = [1, 129, 640, 77, 1000, 256]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    t = int(cu[-1])
    qkv = (0.7 * torch.randn(t, lay.width, device="cuda")).bfloat16()
    monkeypatch.setenv("MSRL_ATTN_TCGEN05", "1")
    out, lse = ops.attn_varlen_fwd(qkv, lay, cu.cuda(), max(lens), causal=causal)
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "tcgen05 attention")
    monkeypatch.setenv("MSRL_ATTN_TCGEN05", "0")
    out_m, lse_m = ops.attn_varlen_fwd(qkv, lay, cu.cuda(), max(lens), causal=causal)
    out_r, lse_r = ops.attn_varlen_fwd(qkv.cpu(), lay, cu, max(lens), causal=causal)
    torch.testing.assert_close(out.float().cpu(), out_r.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(lse.cpu(), lse_r, rtol=1e-2, atol=2e-2)
    torch.testing.assert_close(out.float(), out_m.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(lse, lse_m, rtol=1e-2, atol=2e-2)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("nh,nkv,ql,kl", [
    (3, 1, [127, 128, 129, 1], [127, 128, 129, 1]),              # few tiles: one query tile to a block
    (3, 1, [64], [64 + 2000]),                                   # a short portion behind many cached keys
    (6, 2, [255, 256, 257, 385, 1, 900], [255, 256, 257, 385, 1, 900]),   # pairs across row tiles (three heads a group), odd counts
    (2, 2, [1300] * 9, [1300, 1301, 1427, 1428, 1429, 3000, 2000, 1400, 1556]),   # pairs of row tiles, ends inside and on a tile
    (16, 2, [300, 700, 128], [100, 701, 1]),                     # rows that see nothing when causal
])
def test_flash_attention_fwd_query_tile_pairs(nh, nkv, ql, kl, causal, monkeypatch):
    """Blocks of one and of two query tiles at the borders of tiles and pairs, against the mma.sync kernel and, where every row
    sees a key, the fp32 formulation.  Scores of several tens (q scaled by 6) move the running maximum."""
    from mindspeed_rl_b200 import ops
    from mindspeed_rl_b200.ops.layouts import QKVLayout
    torch.manual_seed(13)
    lay = QKVLayout(nh, nkv, 128, True)
    cu_q, cu_k = (torch.tensor([0] + list(torch.tensor(x).cumsum(0)), dtype=torch.int32) for x in (ql, kl))
    tk = int(cu_k[-1])
    qkv = (6.0 * torch.randn(int(cu_q[-1]), lay.width, device=DEV)).bfloat16()
    k, v = (torch.randn(tk, nkv, 128, device=DEV).bfloat16() for _ in range(2))
    runs = []
    for on in "10":
        monkeypatch.setenv("MSRL_ATTN_TCGEN05", on)
        runs.append(ops.attn_varlen_fwd(qkv, lay, cu_q.to(DEV), max(ql), causal=causal, kv=(k, v), cu_seqlens_k=cu_k.to(DEV)))
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "tcgen05 attention")
    (out, lse), (out_m, lse_m) = runs
    # P and the output are rounded to bf16 (2^-9 each) over values of order one; the two kernels round P against different
    # running maxima
    torch.testing.assert_close(out.float(), out_m.float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(lse, lse_m, rtol=1e-4, atol=1e-3)
    if not causal or all(b >= a for a, b in zip(ql, kl)):
        out_r, lse_r = ops.attn_varlen_fwd(qkv.cpu(), lay, cu_q, max(ql), causal=causal, kv=(k.cpu(), v.cpu()), cu_seqlens_k=cu_k)
        torch.testing.assert_close(out.float().cpu(), out_r.float(), rtol=2e-2, atol=2e-2)
        torch.testing.assert_close(lse.cpu(), lse_r, rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("window", [1, 65, 128, 129, 300, None])
@pytest.mark.parametrize("nh,nkv,form", [(4, 4, "plain"), (6, 2, "plain"), (4, 4, "all"), (6, 2, "all"), (6, 2, "cap"), (6, 2, "sink"),
                                         (4, 4, "gate")])
def test_flash_attention_fwd_pairs_with_windows_and_score_forms(nh, nkv, form, window):
    """Two query tiles to a block whose key ranges start and end at different tiles (every pair crosses row tiles without groups,
    some do with three heads to a group), soft caps, sinks and gates, more keys than queries; against the fp32 formulation."""
    from mindspeed_rl_b200 import ops
    from mindspeed_rl_b200.ops.window import GroupedHeads, window_prefill_attention
    torch.manual_seed(17)
    ql, more = [700, 1, 127, 129, 385, 640, 250], [0, 300, 1, 77, 128, 200, 515]
    kl = [a + b for a, b in zip(ql, more)]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (max(ql) + 127) // 128 * nh * len(ql) > sms            # below that a block takes one query tile
    cu_q, cu_k = (torch.tensor([0] + list(torch.tensor(x).cumsum(0)), dtype=torch.int32, device=DEV) for x in (ql, kl))
    lay = GroupedHeads(nh, nkv, 128, 128, 128, 128, 0, nh * 128, (nh + nkv) * 128)
    proj = (4.0 * torch.randn(sum(ql), (nh + 2 * nkv) * 128, device=DEV)).bfloat16()
    k, v = (torch.randn(sum(kl), nkv, 128, device=DEV).bfloat16() for _ in range(2))
    f = ops.ScoreForm(softcap=6.0 if form in ("cap", "all") else 0.0,
                      gate=torch.randn(sum(ql), nh, device=DEV).bfloat16() if form in ("gate", "all") else None,
                      sink=2.0 * torch.randn(nh, device=DEV) if form in ("sink", "all") else None)
    got = window_prefill_attention(proj, lay, cu_q, cu_k, max(ql), 128 ** -0.5, window, kv=(k, v), form=f)
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "tcgen05 attention")
    host = ops.ScoreForm(f.softcap, *(None if x is None else x.cpu() for x in (f.gate, f.sink)))
    want = window_prefill_attention(proj.cpu(), lay, cu_q.cpu(), cu_k.cpu(), max(ql), 128 ** -0.5, window, kv=(k.cpu(), v.cpu()),
                                    form=host)
    # P and the output are rounded to bf16 (2^-9 each) over values of order one
    torch.testing.assert_close(got.float().cpu(), want.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("nh,nkv,interleaved", [(4, 2, True), (7, 1, False)])
def test_flash_attention_bwd_tcgen05(nh, nkv, interleaved, causal, monkeypatch):
    """tcgen05 backward (dQ kernel, dK/dV kernel, delta) against autograd through the fp32
    formulation and against the mma.sync kernels."""
    from mindspeed_rl_b200 import ops
    from mindspeed_rl_b200.ops.layouts import QKVLayout
    torch.manual_seed(12)
    lay = QKVLayout(nh, nkv, 128, interleaved)
    lens = [1, 129, 640, 77, 1000, 256]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    t = int(cu[-1])
    qkv = (0.7 * torch.randn(t, lay.width, device="cuda")).bfloat16()
    dout = (0.5 * torch.randn(t, nh * 128, device="cuda")).bfloat16()
    monkeypatch.setenv("MSRL_ATTN_TCGEN05", "1")
    out, lse = ops.attn_varlen_fwd(qkv, lay, cu.cuda(), max(lens), causal=causal)
    dqkv = ops.attn_varlen_bwd(dout, qkv, out, lse, lay, cu.cuda(), max(lens), causal=causal)
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "tcgen05 attention")
    monkeypatch.setenv("MSRL_ATTN_TCGEN05", "0")
    dqkv_m = ops.attn_varlen_bwd(dout, qkv, out, lse, lay, cu.cuda(), max(lens), causal=causal)
    out_r, lse_r = ops.attn_varlen_fwd(qkv.cpu(), lay, cu, max(lens), causal=causal)
    dqkv_r = ops.attn_varlen_bwd(dout.cpu(), qkv.cpu(), out_r, lse_r, lay, cu, max(lens), causal=causal)
    torch.testing.assert_close(dqkv.float().cpu(), dqkv_r.float(), rtol=3e-2, atol=5e-2)
    torch.testing.assert_close(dqkv.float(), dqkv_m.float(), rtol=3e-2, atol=5e-2)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("nh,nkv,ql,kl", [
    (3, 1, [127, 128, 129, 1], [127, 128, 129, 1]),              # borders of a tile; odd heads
    (7, 1, [700], [700]),                                        # key tiles shared by two blocks, odd number of steps
    (2, 1, [2], [2]),                                            # one step to each of the two blocks
    (8, 8, [385, 130, 900, 513] * 8, [385, 130, 900, 513] * 8),  # many key tiles: one block each
    (4, 2, [130, 64, 500], [1500, 64, 257]),                     # more keys than queries, and fewer
])
def test_flash_attention_bwd_key_tiles(nh, nkv, ql, kl, causal, monkeypatch):
    """Backward with one and with two blocks to a key tile, at the borders of 128-row tiles, against the formulas in fp32 with
    the log-sum-exp of the forward (where rows see no key at all, which the formulas answer with nan, against the mma.sync
    kernels).  Run twice: the same bits."""
    from mindspeed_rl_b200 import ops
    torch.manual_seed(14)
    cu_q, cu_k = (torch.tensor([0] + list(torch.tensor(x).cumsum(0)), dtype=torch.int32) for x in (ql, kl))
    tq, tk = int(cu_q[-1]), int(cu_k[-1])
    q = torch.randn(tq, nh, 128, device=DEV).bfloat16()
    k, v = (torch.randn(tk, nkv, 128, device=DEV).bfloat16() for _ in range(2))
    do = torch.randn(tq, nh * 128, device=DEV).bfloat16()
    out, lse = ops.attn_kv_fwd(q, k, v, cu_q.to(DEV), cu_k.to(DEV), max(ql), causal)
    got, again = (ops.attn_kv_bwd(do, q, k, v, out, lse, cu_q.to(DEV), cu_k.to(DEV), max(ql), max(kl), causal) for _ in range(2))
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "tcgen05 attention")
    if causal and any(a > b for a, b in zip(ql, kl)):
        monkeypatch.setenv("MSRL_ATTN_TCGEN05", "0")
        ref = ops.attn_kv_bwd(do, q, k, v, out, lse, cu_q.to(DEV), cu_k.to(DEV), max(ql), max(kl), causal)
    else:
        ref = ops.attn_kv_bwd(do.cpu().float(), q.cpu().float(), k.cpu().float(), v.cpu().float(), out.cpu().float(), lse.cpu(),
                              cu_q, cu_k, max(ql), max(kl), causal)
    for a, b, c in zip(got, again, ref):
        assert torch.equal(a, b)
        a, c = a.float().cpu(), c.float().cpu()
        # P and dS are rounded to bf16 (2^-9 of each term, averaged over the sum) and so is the result
        assert ((a - c).norm() / c.norm()).item() < 6e-3
        torch.testing.assert_close(a, c, rtol=2e-2, atol=2e-2 * c.abs().max().item())


@pytest.mark.parametrize("bad", [math.inf, math.nan])
@pytest.mark.parametrize("ql,kl,causal,poison", [
    ([144, 100], [144, 100], True, 144),          # the next sequence from its first row on
    ([130, 100], [130, 100], True, 144),          # from the next sixteen rows on
    ([130, 100], [130, 100], False, 144),
    ([1030, 90, 300] * 3, [1030, 90, 300] * 3, True, 1040),
    ([200, 40], [264, 140], True, 272),           # more keys than queries
])
def test_flash_attention_does_not_read_the_next_sequence(ql, kl, causal, poison, bad):
    """What follows a sequence in the packed rows takes part in its last tile with weights of exact zeros, which an inf or nan turns
    into nan: no sixteen rows that lie wholly behind the sequence are multiplied."""
    from mindspeed_rl_b200 import ops
    torch.manual_seed(15)
    nh, nkv = 4, 2
    cu_q, cu_k = (torch.tensor([0] + list(torch.tensor(x).cumsum(0)), dtype=torch.int32, device=DEV) for x in (ql, kl))
    q, do = (torch.randn(sum(ql), nh, 128, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(sum(kl), nkv, 128, device=DEV).bfloat16() for _ in range(2))

    def run():
        o, lse = ops.attn_kv_fwd(q, k, v, cu_q, cu_k, max(ql), causal)
        dq, dk, dv = ops.attn_kv_bwd(do.view(sum(ql), -1), q, k, v, o, lse, cu_q, cu_k, max(ql), max(kl), causal)
        return o[:ql[0]], lse[:, :ql[0]], dq[:ql[0]], dk[:kl[0]], dv[:kl[0]]

    clean = [x.clone() for x in run()]
    for x, n in ((q, poison - kl[0] + ql[0]), (do, poison - kl[0] + ql[0]), (k, poison), (v, poison)):
        x[n:] = bad
    for a, b in zip(run(), clean):
        assert bool(a.isfinite().all()) and torch.equal(a, b)
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "tcgen05 attention")


@pytest.mark.parametrize("bad", [math.inf, math.nan])
def test_flash_attention_reads_what_some_row_of_a_tile_sees(bad):
    """Keys behind the last and before the first that a tile of 128 query rows sees, and queries that see none of 128 keys, do not
    reach it across a border of sixteen."""
    from mindspeed_rl_b200 import ops
    from mindspeed_rl_b200.ops.window import GroupedHeads, window_prefill_attention
    torch.manual_seed(16)
    nh, nkv, ql, kl = 4, 2, 200, 264
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device=DEV) for n in (ql, kl))
    q, do = (torch.randn(ql, nh, 128, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(kl, nkv, 128, device=DEV).bfloat16() for _ in range(2))
    o, lse = ops.attn_kv_fwd(q, k, v, cu_q, cu_k, ql, True)
    clean = ops.attn_kv_bwd(do.view(ql, -1), q, k, v, o, lse, cu_q, cu_k, ql, kl, True)
    v2 = v.clone()
    v2[192:] = bad                                            # row r sees keys up to r + 64: rows 0 to 127 none of these
    assert torch.equal(ops.attn_kv_fwd(q, k, v2, cu_q, cu_k, ql, True)[0][:128], o[:128])
    do[:64] = bad                                             # these rows see no key from 128 on
    for a, b in zip(ops.attn_kv_bwd(do.view(ql, -1), q, k, v, o, lse, cu_q, cu_k, ql, kl, True)[1:], clean[1:]):
        assert torch.equal(a[128:], b[128:])
    lay = GroupedHeads(4, 2, 128, 128, 128, 128, 0, 512, 768)
    t, cu = 500, torch.tensor([0, 500], dtype=torch.int32, device=DEV)
    proj = torch.randn(t, 1024, device=DEV).bfloat16()
    want = window_prefill_attention(proj, lay, cu, cu, t, 128 ** -0.5, 150)
    proj[:96, 768:] = bad                                     # rows from 256 on see keys from 107 on
    assert torch.equal(window_prefill_attention(proj, lay, cu, cu, t, 128 ** -0.5, 150)[256:], want[256:])
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "tcgen05 attention")


@pytest.mark.parametrize("causal", [False, True])
def test_block_attention_with_separate_kv(causal):
    """The block primitives of ring attention (queries against a separate K/V block, log-sum-exp of the
    whole row given to the backward) against the fp32 formulation: ragged query and key lengths,
    non-causal and bottom-right causal."""
    from mindspeed_rl_b200 import ops
    torch.manual_seed(21)
    nh, nkv, hd = 6, 2, 128
    ql, kl = [130, 64, 500], [257, 64, 900]
    cu_q = torch.tensor([0] + list(torch.tensor(ql).cumsum(0)), dtype=torch.int32)
    cu_k = torch.tensor([0] + list(torch.tensor(kl).cumsum(0)), dtype=torch.int32)
    tq, tk = int(cu_q[-1]), int(cu_k[-1])
    q = (0.7 * torch.randn(tq, nh, hd, device="cuda")).bfloat16()
    k = (0.7 * torch.randn(tk, nkv, hd, device="cuda")).bfloat16()
    v = (0.7 * torch.randn(tk, nkv, hd, device="cuda")).bfloat16()
    do = (0.5 * torch.randn(tq, nh * hd, device="cuda")).bfloat16()
    out, lse = ops.attn_kv_fwd(q, k, v, cu_q.cuda(), cu_k.cuda(), max(ql), causal)
    dq, dk, dv = ops.attn_kv_bwd(do, q, k, v, out, lse, cu_q.cuda(), cu_k.cuda(), max(ql), max(kl), causal)
    G.check_status(torch.device("cuda", torch.cuda.current_device()), "block attention")
    out_r, lse_r = ops.attn_kv_fwd(q.cpu().float(), k.cpu().float(), v.cpu().float(), cu_q, cu_k, max(ql), causal)
    dq_r, dk_r, dv_r = ops.attn_kv_bwd(do.cpu().float(), q.cpu().float(), k.cpu().float(), v.cpu().float(), out_r, lse_r,
                                       cu_q, cu_k, max(ql), max(kl), causal)
    torch.testing.assert_close(out.float().cpu(), out_r, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(lse.cpu(), lse_r, rtol=1e-2, atol=2e-2)
    for a, b in ((dq, dq_r), (dk, dk_r), (dv, dv_r)):
        torch.testing.assert_close(a.float().cpu(), b, rtol=3e-2, atol=5e-2)
