"""GPU parity: the CUDA kernels, called through the C ABI, against the reference's golden vectors
and against the CPU oracle (which tests/test_oracle.py pins to those vectors).

Tolerances (stated by the target for bf16 kernels vs the fp32 reference on bf16-rounded inputs):
max-abs <= 2e-2 on O, relative L2 <= 1e-2 on each gradient.  fp32 tensors through the general
kernels are held to 1e-4.
"""
import ctypes
import math

import pytest
import torch

import simplical_attn_b200 as sab
from oracle import c_oracle, simplicial_oracle as so
from simplical_attn_b200 import _abi
from simplical_attn_b200 import simplicial_attn as host
from tests import golden_util as gu

pytestmark = pytest.mark.gpu

TOL_O_BF16 = 2e-2
TOL_G_BF16 = 1e-2
TOL_F32 = 1e-4
DEV = "cuda"
TC_BWD_READY = True


def _grad_err(a, b):
    """Relative L2 against the reference gradient.  Where the reference gradient is zero (one
    (j,k) pair per query: softmax weight 1, no logit gradient) the error is absolute and scaled by
    0.1: a bf16 kernel then returns scale * (dO.(V1*V2) - dO.O) * K, which is the rounding of the
    stored O (2^-9 relative) times values of order 10, not zero."""
    if float(b.abs().max()) < 1e-5:
        return 0.1 * float((a.float().cpu() - b).abs().max())
    return so.rel_l2(a.float().cpu(), b)


def _run(ins, cfg, algo, dtype=torch.bfloat16, need=(True,) * 5, halo1=0, halo2=0):
    t = {k: v.to(DEV).to(dtype) for k, v in ins.items()}
    o, lse = sab.two_simplicial_attn_fwd_kernel(t["q"], t["k1"], t["k2"], t["v1"], t["v2"], cfg["w1"], cfg["w2"],
                                                cfg["scale"], cfg["k2_bias"], cfg["v2_bias"], halo1, halo2, algo=algo)
    grads = sab.two_simplicial_attn_bwd(t["q"], t["k1"], t["k2"], t["v1"], t["v2"], o, lse, t["do"], cfg["w1"], cfg["w2"],
                                        cfg["scale"], cfg["k2_bias"], cfg["v2_bias"], halo1, halo2, need,
                                        algo=algo if (algo != "tcgen05" or TC_BWD_READY) else "auto")
    torch.cuda.synchronize()
    return o, lse, grads


def _tc_supported(cfg):
    return cfg["D"] in (64, 128) and min(cfg["w2"], cfg["N"]) <= 1024


@pytest.mark.parametrize("name", gu.names())
def test_general_bf16_vs_reference_golden(name):
    cfg, ins, outs = gu.load(name)
    o, _, grads = _run(ins, cfg, "general")
    assert float((o.float().cpu() - outs["o"]).abs().max()) <= TOL_O_BF16
    for nm, g in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads):
        assert _grad_err(g, outs[nm]) <= TOL_G_BF16, nm


@pytest.mark.parametrize("name", gu.names())
def test_general_fp32_vs_reference_golden(name):
    cfg, ins, outs = gu.load(name)
    o, _, grads = _run(ins, cfg, "general", dtype=torch.float32)
    assert float((o.cpu() - outs["o"]).abs().max()) <= TOL_F32
    for nm, g in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads):
        assert _grad_err(g, outs[nm]) <= TOL_F32, nm


@pytest.mark.parametrize("name", [n for n in gu.names() if _tc_supported(gu.load(n)[0])])
def test_tensor_core_vs_reference_golden(name):
    cfg, ins, outs = gu.load(name)
    o, _, grads = _run(ins, cfg, "tcgen05")
    assert float((o.float().cpu() - outs["o"]).abs().max()) <= TOL_O_BF16
    for nm, g in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads):
        assert _grad_err(g, outs[nm]) <= TOL_G_BF16, nm


# B, N, H, Hkv, D, w1, w2, k2_bias, v2_bias, halo1, halo2
ORACLE_CASES = [
    (1, 300, 2, 1, 128, 100, 32, 0.0, 0.0, 0, 0),      # grouped heads, ragged N
    (2, 200, 2, 2, 128, 512, 32, 0.0, 0.0, 0, 0),      # w1 > N
    (1, 260, 2, 2, 128, 130, 16, 0.0, 0.0, 0, 0),      # two column tiles, 16 delta slots
    (1, 150, 1, 1, 128, 40, 64, 0.0, 0.0, 0, 0),       # 64 delta slots: a query spans two warps
    (1, 140, 2, 2, 64, 33, 5, 0.1, -0.2, 0, 0),        # odd windows, biases
    (1, 96, 2, 1, 128, 48, 12, 0.0, 0.0, 47, 11),      # a sequence shard with halo rows
    (1, 520, 1, 1, 64, 24, 1, 0.0, 0.0, 0, 0),         # w2 = 1: 128 queries per row tile
    (1, 130, 2, 2, 128, 300, 128, 0.0, 0.0, 0, 0),     # widest K2 window: one query per row tile
    (1, 210, 2, 1, 64, 70, 14, 0.05, 0.0, 0, 0),       # D = 64 with 16 delta slots, two of them masked
    (1, 300, 2, 2, 64, 90, 50, 0.0, 0.1, 0, 0),        # D = 64 with 64 delta slots
    (1, 333, 4, 2, 64, 100, 32, 0.0, 0.0, 0, 0),       # D = 64 with 32 delta slots, grouped heads
    (1, 200, 2, 2, 64, 70, 24, 0.1, 0.0, 69, 23),      # D = 64, 32 delta slots (8 masked), bias, halo rows
]


@pytest.mark.parametrize("case", ORACLE_CASES)
@pytest.mark.parametrize("algo", ["general", "tcgen05"])
def test_vs_cpu_oracle(case, algo):
    B, N, H, Hkv, D, w1, w2, kb, vb, h1, h2 = case
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=3, seed_do=4, halo1=h1, halo2=h2)
    scale = 1.0 / math.sqrt(D)
    cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=kb, v2_bias=vb)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    o, lse, grads = _run(ins, cfg, algo, halo1=h1, halo2=h2)
    ref = so.forward_backward(q, k1, k2, v1, v2, do, w1, w2, scale, kb, vb, h1, h2)
    assert float((o.float().cpu() - ref[0]).abs().max()) <= TOL_O_BF16
    assert float((lse.cpu() - ref[1]).abs().max()) <= 2e-2
    for nm, g, r in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads, ref[2:]):
        assert _grad_err(g, r) <= TOL_G_BF16, nm


# K2 windows wider than one pass of the tensor-core kernels (128 positions): the library chains passes over
# 128-position chunks of the window.  B, N, H, Hkv, D, w1, w2, k2_bias, v2_bias, halo1, halo2
WIDE_K2_CASES = [
    (1, 400, 2, 1, 128, 64, 256, 0.0, 0.0, 0, 0),      # two full chunks, grouped heads
    (1, 330, 2, 2, 128, 40, 160, 0.0, 0.0, 0, 0),      # a full chunk and a 32-position one
    (1, 300, 1, 1, 64, 48, 300, 0.1, -0.1, 0, 0),      # window wider than the sequence is long, D = 64, biases, three chunks
    (1, 200, 2, 2, 128, 30, 200, 0.0, 0.0, 29, 199),   # a sequence shard with halo rows in front
]


@pytest.mark.parametrize("case", WIDE_K2_CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def test_wide_k2_window_vs_cpu_oracle(case, dtype):
    B, N, H, Hkv, D, w1, w2, kb, vb, h1, h2 = case
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=5, seed_do=6, halo1=h1, halo2=h2)
    scale = 1.0 / math.sqrt(D)
    cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=kb, v2_bias=vb)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    o, lse, grads = _run(ins, cfg, "tcgen05", dtype=dtype, halo1=h1, halo2=h2)
    if dtype == torch.float16:
        q, k1, k2, v1, v2, do = (t.to(torch.float16).float() for t in (q, k1, k2, v1, v2, do))
    ref = so.forward_backward(q, k1, k2, v1, v2, do, w1, w2, scale, kb, vb, h1, h2)
    assert float((o.float().cpu() - ref[0]).abs().max()) <= TOL_O_BF16
    assert float((lse.cpu() - ref[1]).abs().max()) <= 2e-2
    for nm, g, r in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads, ref[2:]):
        assert _grad_err(g, r) <= TOL_G_BF16, nm


@pytest.mark.parametrize("shape", [(260, 128, 130, 16), (300, 128, 100, 32), (150, 128, 40, 64), (210, 64, 70, 14), (333, 64, 100, 32),
                                   (130, 128, 300, 128), (330, 128, 40, 160)])
@pytest.mark.parametrize("algo", ["tcgen05", "general"])
def test_nothing_behind_the_tensors_is_read_into_the_results(shape, algo):
    """The last 128-row tile of a sequence has rows for queries past the end; their K2 / V2 window rows lie
    past the end of K2 / V2.  Whatever is in memory there (here: NaN, the tensors are views of larger buffers)
    must not reach any result."""
    N, D, w1, w2 = shape
    B, H, Hkv = 1, 2, 2
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=21, seed_do=22)
    scale = 1.0 / math.sqrt(D)

    def padded(t):
        big = torch.full((B, N + 192, t.shape[2], D), float("nan"), dtype=torch.bfloat16, device=DEV)
        big[:, :N] = t.to(DEV).to(torch.bfloat16)
        return big[:, :N]

    clean = [t.to(DEV).to(torch.bfloat16) for t in (q, k1, k2, v1, v2, do)]
    dirty = [padded(t) for t in (q, k1, k2, v1, v2, do)]
    outs = []
    for ts in (clean, dirty):
        o, lse = sab.two_simplicial_attn_fwd_kernel(*ts[:5], w1, w2, scale, algo=algo)
        grads = sab.two_simplicial_attn_bwd(*ts[:5], o, lse, ts[5], w1, w2, scale, algo=algo)
        outs.append((o, lse) + tuple(grads))
    torch.cuda.synchronize()
    for nm, a, b in zip(("o", "lse", "dq", "dk1", "dk2", "dv1", "dv2"), *outs):
        assert bool(torch.isfinite(b.float()).all()), nm
        assert torch.equal(a, b), nm


@pytest.mark.parametrize("shape", [(1, 700, 4, 2, 128, 200, 32, 0, 0), (2, 260, 2, 2, 128, 130, 16, 0, 0), (1, 150, 2, 1, 128, 40, 64, 0, 0),
                                   (1, 130, 2, 2, 128, 300, 128, 0, 0), (1, 330, 2, 2, 128, 40, 160, 0, 0), (1, 333, 4, 2, 64, 100, 32, 0, 0),
                                   (1, 96, 2, 1, 128, 48, 12, 47, 11)])
def test_workspace_contents_do_not_matter(shape, monkeypatch):
    """The kernels write every partial sum of the workspace before they read it: a workspace full of NaN
    bit patterns (behind the status word, which must start at zero) gives the same results, bit for bit."""
    B, N, H, Hkv, D, w1, w2, h1, h2 = shape
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=31, seed_do=32, halo1=h1, halo2=h2)
    cfg = dict(w1=w1, w2=w2, scale=1.0 / math.sqrt(D), k2_bias=0.0, v2_bias=0.0)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    clean = _run(ins, cfg, "tcgen05", halo1=h1, halo2=h2)

    def nan_workspace(nbytes, device):
        ws = torch.full((max(int(nbytes), 256),), 0xFF, dtype=torch.uint8, device=device)
        ws[:256].zero_()
        return ws

    monkeypatch.setattr(host, "_workspace", nan_workspace)
    dirty = _run(ins, cfg, "tcgen05", halo1=h1, halo2=h2)
    for nm, a, b in zip(("o", "lse"), clean[:2], dirty[:2]):
        assert torch.equal(a, b), nm
    for nm, a, b in zip(("dq", "dk1", "dk2", "dv1", "dv2"), clean[2], dirty[2]):
        assert bool(torch.isfinite(b.float()).all()) and torch.equal(a, b), nm


def test_tensor_core_vs_general_medium():
    """Same bf16 inputs through both kernel families at a size the CPU oracle would take minutes for."""
    B, N, H, Hkv, D, w1, w2 = 1, 2048, 4, 2, 128, 512, 32
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D)
    cfg = dict(w1=w1, w2=w2, scale=1.0 / math.sqrt(D), k2_bias=0.0, v2_bias=0.0)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    o_t, lse_t, g_t = _run(ins, cfg, "tcgen05")
    o_g, lse_g, g_g = _run(ins, cfg, "general")
    assert float((o_t.float() - o_g.float()).abs().max()) <= 3e-2      # two bf16-rounded results
    assert float((lse_t - lse_g).abs().max()) <= 1e-2
    for nm, a, b in zip(("dq", "dk1", "dk2", "dv1", "dv2"), g_t, g_g):
        assert so.rel_l2(a.float().cpu(), b.float().cpu()) <= TOL_G_BF16, nm


def test_full_size_forward_row_slices_vs_oracle():
    """The forward configuration quoted for one GPU (B2 H8 N8192 D128 w 512/32, storage [B,H,N,D]):
    row slices at the start, across a window boundary, in the middle and at the end are compared
    with the C loop oracle; the whole output is checked finite and against the general kernels on
    one (batch, head)."""
    B, N, H, D, w1, w2 = 2, 8192, 8, 128, 512, 32
    scale = 1.0 / math.sqrt(D)
    q, k1, k2, v1, v2, _ = so.make_inputs(B, N, H, H, D)
    dev = [t.to(DEV).to(torch.bfloat16).permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3) for t in (q, k1, k2, v1, v2)]
    assert dev[0].stride(2) == N * D                                    # [B,H,N,D] storage
    o, lse = sab.two_simplicial_attn_fwd_kernel(*dev, w1, w2, scale, algo="tcgen05")
    torch.cuda.synchronize()
    assert bool(torch.isfinite(o.float()).all()) and bool(torch.isfinite(lse).all())
    for lo, hi in ((0, 40), (500, 530), (4090, 4100), (8180, 8192)):
        ro, rl = c_oracle.forward(q, k1, k2, v1, v2, w1, w2, scale, row_begin=lo, row_end=hi)
        assert float((o[:, lo:hi].float().cpu() - ro[:, lo:hi]).abs().max()) <= TOL_O_BF16
        assert float((lse[:, :, lo:hi].cpu() - rl[:, :, lo:hi]).abs().max()) <= 2e-2
    sl = [t[1:2, :, 3:4].contiguous() for t in dev]
    og, lg = sab.two_simplicial_attn_fwd_kernel(*sl, w1, w2, scale, algo="general")
    assert float((o[1:2, :, 3:4].float() - og.float()).abs().max()) <= 3e-2
    assert float((lse[1:2, 3:4] - lg).abs().max()) <= 1e-2


def _module_inputs(B=1, N=96, H=2, D=64, dtype=torch.bfloat16, seed=11, scale_in=1.0):
    g = torch.Generator().manual_seed(seed)
    return [(scale_in * torch.randn(B, N, H, D, generator=g)).to(DEV).to(dtype).requires_grad_(True) for _ in range(5)]


def test_module_autograd_and_accumulation():
    """Public call: gradients exist for every input, None-gating follows requires_grad, and a second
    backward doubles .grad (the reference's test_gradient_accumulation, test_correctness.py:290-318)."""
    ins = _module_inputs()
    attn = sab.TwoSimplicialAttention(64, w1=16, w2=8)
    attn(*ins).sum().backward()
    first = [t.grad.clone() for t in ins]
    assert all(bool(torch.isfinite(g.float()).all()) and float(g.float().abs().sum()) > 0 for g in first)
    attn(*ins).sum().backward()
    for t, g in zip(ins, first):
        assert torch.allclose(t.grad.float(), 2 * g.float(), atol=1e-2, rtol=1e-2)
    ins2 = _module_inputs()
    ins2[1].requires_grad_(False)
    ins2[4].requires_grad_(False)
    attn(*ins2).sum().backward()
    assert ins2[1].grad is None and ins2[4].grad is None and ins2[0].grad is not None


@pytest.mark.parametrize("algo", ["general", "tcgen05"])
def test_deterministic(algo):
    host.default_algo = algo
    try:
        outs = []
        for _ in range(2):
            ins = _module_inputs(N=200, D=128)
            o = sab.TwoSimplicialAttention(128, w1=64, w2=16)(*ins)
            o.backward(torch.ones_like(o))
            outs.append([o.detach().clone()] + [t.grad.clone() for t in ins])
        for a, b in zip(*outs):
            assert torch.equal(a, b)
    finally:
        host.default_algo = "auto"


@pytest.mark.parametrize("algo", ["general", "tcgen05"])
def test_edge_cases_finite(algo):
    """The reference's TestEdgeCases (test_correctness.py:321-396): w=1, w > N, zeros, large inputs."""
    host.default_algo = algo
    try:
        for (N, w1, w2, fill) in ((32, 1, 1, None), (32, 100, 100, None), (32, 8, 8, 0.0), (32, 8, 8, 10.0)):
            ins = _module_inputs(N=N, D=64)
            if fill is not None:
                ins = [torch.full_like(t, fill).requires_grad_(True) for t in ins]
            o = sab.TwoSimplicialAttention(64, w1=w1, w2=w2)(*ins)
            o.sum().backward()
            assert o.shape == ins[0].shape and bool(torch.isfinite(o.float()).all())
            assert all(bool(torch.isfinite(t.grad.float()).all()) for t in ins)
            if fill == 0.0:
                assert float(o.float().abs().max()) == 0.0
            if fill == 10.0:
                assert float((o.float() - 100.0).abs().max()) <= 1.0     # softmax of equal logits: mean of v1*v2
    finally:
        host.default_algo = "auto"


def test_fp16_and_fp32_through_auto():
    """The reference's dtype matrix (test_correctness.py:39,154): fp16 runs on the tensor-core kernels (where they
    cover the shape), fp32 on the general kernels."""
    for dtype, tol in ((torch.float16, 1e-2), (torch.float32, 1e-4)):
        cfg, ins, outs = gu.load("tiny_sym")
        o, _, _ = _run(ins, cfg, "auto", dtype=dtype)
        assert float((o.float().cpu() - outs["o"]).abs().max()) <= tol


@pytest.mark.parametrize("name", [n for n in gu.names() if _tc_supported(gu.load(n)[0])])
def test_tensor_core_fp16_vs_reference_golden(name):
    """IEEE half through the tensor-core kernels (the golden inputs are bf16 values, exact in half)."""
    cfg, ins, outs = gu.load(name)
    o, _, grads = _run(ins, cfg, "tcgen05", dtype=torch.float16)
    assert o.dtype == torch.float16
    assert float((o.float().cpu() - outs["o"]).abs().max()) <= TOL_O_BF16
    for nm, g in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads):
        assert g.dtype == torch.float16
        assert _grad_err(g, outs[nm]) <= TOL_G_BF16, nm


@pytest.mark.parametrize("case", [ORACLE_CASES[0], ORACLE_CASES[2], ORACLE_CASES[3], ORACLE_CASES[4], ORACLE_CASES[5], ORACLE_CASES[8]])
def test_tensor_core_fp16_vs_cpu_oracle(case):
    B, N, H, Hkv, D, w1, w2, kb, vb, h1, h2 = case
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=3, seed_do=4, halo1=h1, halo2=h2)
    scale = 1.0 / math.sqrt(D)
    cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=kb, v2_bias=vb)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    o, lse, grads = _run(ins, cfg, "tcgen05", dtype=torch.float16, halo1=h1, halo2=h2)
    ref = so.forward_backward(q, k1, k2, v1, v2, do, w1, w2, scale, kb, vb, h1, h2)
    assert float((o.float().cpu() - ref[0]).abs().max()) <= TOL_O_BF16
    assert float((lse.cpu() - ref[1]).abs().max()) <= 2e-2
    for nm, g, r in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads, ref[2:]):
        assert _grad_err(g, r) <= TOL_G_BF16, nm


def test_bad_arguments_raise():
    ins = _module_inputs()
    with pytest.raises(ValueError):
        sab.two_simplicial_attention(ins[0], ins[1][:, :50], ins[2], ins[3], ins[4], 8, 8)
    with pytest.raises(TypeError):
        sab.two_simplicial_attention(ins[0], ins[1].float(), ins[2], ins[3], ins[4], 8, 8)
    from simplical_attn_b200._abi import SimplicialAttnError
    with pytest.raises(SimplicialAttnError):
        sab.two_simplicial_attention(ins[0], ins[1], ins[2], ins[3], ins[4], 0, 8)


@pytest.mark.parametrize("w1", [128, 256, 512, 1024])
@pytest.mark.parametrize("w2", [16, 32, 64])
def test_window_sweep_tensor_core_vs_general(w1, w2):
    """The window sweep of the batch x head-parallel configuration (w1 in {128..1024} x w2 in {16,32,64},
    D=128) at a reduced batch and length: both kernel families on the same bf16 inputs."""
    B, N, H, Hkv, D = 1, 1536, 2, 2, 128
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=w1 + w2)
    cfg = dict(w1=w1, w2=w2, scale=1.0 / math.sqrt(D), k2_bias=0.0, v2_bias=0.0)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    o_t, lse_t, g_t = _run(ins, cfg, "tcgen05")
    o_g, lse_g, g_g = _run(ins, cfg, "general")
    assert float((o_t.float() - o_g.float()).abs().max()) <= 3e-2
    assert float((lse_t - lse_g).abs().max()) <= 1e-2
    for nm, a, b in zip(("dq", "dk1", "dk2", "dv1", "dv2"), g_t, g_g):
        assert so.rel_l2(a.float().cpu(), b.float().cpu()) <= TOL_G_BF16, nm


@pytest.mark.parametrize("w2", [16, 32, 64, 128, 200])
def test_partial_gradient_requests_match_full_call(w2):
    """The reference's two backward kernels are separate calls (dQ/dK1/dV1 and dK2/dV2).  Asking the
    tensor-core path for a subset must give the tensors of the full call and None for the rest: exactly
    with 16, 32 and 64 K2 positions (the row kernel with operand / epilogue warpgroups), and to the last
    bit or two of the 16-bit results with 128 (the other row kernel sums dQ in another order when it
    keeps no dK2 / dV2 ring) and 200 (two passes over chunks of the K2 window)."""
    B, N, H, Hkv, D, w1 = 1, 700, 4, 2, 128, 200
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=11 + w2)
    cfg = dict(w1=w1, w2=w2, scale=1.0 / math.sqrt(D), k2_bias=0.0, v2_bias=0.0)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    _, _, full = _run(ins, cfg, "tcgen05")
    for need in ((True, True, False, True, False), (False, False, True, False, True), (True, False, False, False, False),
                 (False, False, False, False, True)):
        _, _, part = _run(ins, cfg, "tcgen05", need=need)
        for nm, n, a, b in zip(("dq", "dk1", "dk2", "dv1", "dv2"), need, part, full):
            if n and w2 <= 64:
                assert torch.equal(a, b), (nm, need)
            elif n:
                assert so.rel_l2(a.float().cpu(), b.float().cpu()) <= 2e-3, (nm, need)
            else:
                assert a is None, (nm, need)


def test_grouped_heads_full_size():
    """The grouped-head configuration (B1, 32 query heads on 2 KV heads, N=16384, D=128, w 512/32): forward
    row slices against the C loop oracle, all five gradients against the general kernels (which sum
    the 16 query heads of a group inside one warp, in a fixed order)."""
    B, N, H, Hkv, D, w1, w2 = 1, 16384, 32, 2, 128, 512, 32
    scale = 1.0 / math.sqrt(D)
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D)
    cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=0.0, v2_bias=0.0)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    o_t, lse_t, g_t = _run(ins, cfg, "tcgen05")
    assert all(bool(torch.isfinite(t.float()).all()) for t in (o_t, *g_t))
    for lo, hi in ((0, 24), (8190, 8200), (16376, 16384)):
        ro, rl = c_oracle.forward(q, k1, k2, v1, v2, w1, w2, scale, row_begin=lo, row_end=hi)
        assert float((o_t[:, lo:hi].float().cpu() - ro[:, lo:hi]).abs().max()) <= TOL_O_BF16
        assert float((lse_t[:, :, lo:hi].cpu() - rl[:, :, lo:hi]).abs().max()) <= 2e-2
    t = {k: v.to(DEV).to(torch.bfloat16) for k, v in ins.items()}
    g_g = sab.two_simplicial_attn_bwd(t["q"], t["k1"], t["k2"], t["v1"], t["v2"], o_t, lse_t, t["do"], w1, w2, scale,
                                      algo="general")
    torch.cuda.synchronize()
    for nm, a, b in zip(("dq", "dk1", "dk2", "dv1", "dv2"), g_t, g_g):
        assert so.rel_l2(a.float().cpu(), b.float().cpu()) <= TOL_G_BF16, nm


# B, N, H, Hkv, D, w1, w2 -- the sizes the headline figures are quoted on
FULL_SIZE_GRAD_CASES = [
    pytest.param((2, 8192, 8, 8, 128, 512, 32), id="B2_H8_N8192_w512x32"),          # single-GPU forward / headline windows
    pytest.param((1, 16384, 32, 2, 128, 512, 32), id="B1_H32_Hkv2_N16384_w512x32"), # grouped heads: 16 query heads per KV head
    pytest.param((1, 8192, 2, 2, 128, 1024, 64), id="B1_H2_N8192_w1024x64"),        # the long-sequence configuration's windows
]


@pytest.mark.parametrize("case", FULL_SIZE_GRAD_CASES)
def test_full_size_gradients_vs_oracle(case):
    """All five gradients of the tensor-core path at full sequence length against the C loop oracle
    (`simplicial/reference.py:39-74` through the pinned C port), on ranges the oracle finishes in
    seconds.  For a range of 64 K rows [k0, k0+64) the oracle is run on every query row that reaches
    it, [k0, k0+64+w1-1): that gives dK1, dV1, dK2 and dV2 of the K rows complete (the sum of the
    shares of those queries) and dQ of all those query rows.  Ranges: the sequence start, an
    unaligned range in the interior; plus dQ of the last rows."""
    B, N, H, Hkv, D, w1, w2 = case
    scale = 1.0 / math.sqrt(D)
    q, k1, k2, v1, v2, do = so.make_inputs(B, N, H, Hkv, D, seed=17, seed_do=18)
    cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=0.0, v2_bias=0.0)
    ins = dict(q=q, k1=k1, k2=k2, v1=v1, v2=v2, do=do)
    _, _, grads = _run(ins, cfg, "tcgen05")
    dq, dk1, dk2, dv1, dv2 = (g.float().cpu() for g in grads)
    assert all(bool(torch.isfinite(g).all()) for g in (dq, dk1, dk2, dv1, dv2))
    for k0 in (0, N // 2 + 37):
        r0, r1 = k0, min(N, k0 + 64 + w1 - 1)
        ref = c_oracle.backward(q, k1, k2, v1, v2, do, w1, w2, scale, row_begin=r0, row_end=r1)
        assert so.rel_l2(dq[:, r0:r1], ref[0][:, r0:r1]) <= TOL_G_BF16, ("dq", k0)
        for nm, g, r in zip(("dk1", "dk2", "dv1", "dv2"), (dk1, dk2, dv1, dv2), ref[1:]):
            assert so.rel_l2(g[:, k0:k0 + 64], r[:, k0:k0 + 64]) <= TOL_G_BF16, (nm, k0)
    r0 = N - 24
    ref = c_oracle.backward(q, k1, k2, v1, v2, do, w1, w2, scale, row_begin=r0, row_end=N)
    assert so.rel_l2(dq[:, r0:], ref[0][:, r0:]) <= TOL_G_BF16, "dq (end)"
    # the last K rows receive gradient only from the last queries: complete in this call as well
    for nm, g, r in zip(("dk1", "dk2", "dv1", "dv2"), (dk1, dk2, dv1, dv2), ref[1:]):
        assert so.rel_l2(g[:, N - 1:], r[:, N - 1:]) <= TOL_G_BF16, (nm, "last row")


@pytest.mark.parametrize("shape", [(5, 512, 4, 2, 128, 128, 32), (1, 384, 8, 8, 128, 96, 16), (2, 256, 8, 2, 64, 64, 32)])
def test_host_pipeline_matches_device_call(shape):
    """Pinned host tensors in, pinned host results out (uploads / kernels / downloads of (sequence,
    head-group) chunks on three streams, strided copies for the head groups).  O, dQ, dK1, dV1 are
    bit-identical to one device call on the whole batch; dK2 and dV2 are sums of per-run partials whose
    run length depends on how many (batch, head) pairs a call holds, so they agree to fp32 rounding of
    the partial sums (well inside bf16 resolution)."""
    from simplical_attn_b200.host_pipeline import HostPipeline, plan_chunks
    B, N, H, Hkv, D, w1, w2 = shape
    ts = [t.to(torch.bfloat16).pin_memory() for t in so.make_inputs(B, N, H, Hkv, D, seed=9, seed_do=10)]
    scale = 1.0 / math.sqrt(D)
    chunks = plan_chunks(B, Hkv)
    assert sorted(chunks) == chunks and sum(h1 - h0 for _, h0, h1 in chunks) == B * Hkv      # every (sequence, KV head) once
    pipe = HostPipeline("cuda")
    for _ in range(2):                                   # second call reuses buffers
        res = pipe.forward_backward(*ts, w1, w2, scale)
    dev = [t.cuda() for t in ts]
    o, lse = sab.two_simplicial_attn_fwd_kernel(*dev[:5], w1, w2, scale)
    grads = sab.two_simplicial_attn_bwd(*dev[:5], o, lse, dev[5], w1, w2, scale)
    for name, a, b in zip(("o", "dq", "dk1", "dk2", "dv1", "dv2"), res, (o,) + tuple(grads)):
        assert a.is_pinned()
        if name in ("dk2", "dv2"):
            assert so.rel_l2(a.float(), b.float().cpu()) <= 2e-3, name
        else:
            assert torch.equal(a, b.cpu()), name


def test_projection_module_matches_oracle_and_trains():
    """Hidden states -> fused input projection -> attention -> output projection: the attention inside reads the
    five strided views of the projection GEMM's output directly; its result equals the CPU oracle on the same
    projected tensors, and gradients reach the projection weights."""
    torch.manual_seed(3)
    B, N, hidden, H, Hkv, D, w1, w2 = 2, 192, 256, 4, 2, 64, 48, 16
    mod = sab.TwoSimplicialSelfAttention(hidden, H, D, w1, w2, kv_heads=Hkv, device=DEV)
    x = (0.5 * torch.randn(B, N, hidden, device=DEV)).to(torch.bfloat16).requires_grad_(True)
    y = mod(x)
    assert y.shape == (B, N, hidden) and bool(torch.isfinite(y.float()).all())
    with torch.no_grad():
        fused = mod.in_proj(x)
        parts = [t.float().cpu() for t in torch.split(fused, mod.widths, dim=-1)]
        q = parts[0].view(B, N, H, D)
        k1, k2, v1, v2 = (t.view(B, N, Hkv, D) for t in parts[1:])
        o_ref, _ = so.forward(q, k1, k2, v1, v2, w1, w2, mod.scale)
        y_ref = torch.nn.functional.linear(o_ref.reshape(B, N, H * D).to(torch.bfloat16).to(DEV), mod.out_proj.weight)
    assert float((y.float() - y_ref.float()).abs().max()) <= 3e-2
    y.float().pow(2).mean().backward()
    for prm in (mod.in_proj.weight, mod.out_proj.weight):
        assert prm.grad is not None and bool(torch.isfinite(prm.grad.float()).all()) and float(prm.grad.float().abs().sum()) > 0
    assert x.grad is not None and x.grad.shape == x.shape


# B, N, H, Hkv, D, w1, w2, k2_bias, v2_bias, halo1, halo2: head dims at the edges of the padded ones, K2 windows around
# the 64 virtual rows of a tile, one and many queries to a tile, K1 windows around a tile's columns
GENERAL_CASES = [
    (1, 1, 1, 1, 8, 1, 1, 0.0, 0.0, 0, 0),
    (1, 37, 2, 1, 33, 17, 3, 0.1, -0.1, 0, 0),
    (2, 70, 3, 3, 32, 64, 64, 0.0, 0.0, 0, 0),
    (1, 150, 2, 2, 40, 65, 65, 0.0, 0.0, 0, 0),
    (1, 140, 4, 2, 96, 16, 24, 0.0, 0.2, 15, 23),
    (1, 90, 1, 1, 130, 33, 16, 0.0, 0.0, 0, 0),
    (1, 200, 2, 1, 200, 80, 130, 0.0, 0.0, 0, 0),
    (1, 75, 1, 1, 256, 100, 7, 0.1, 0.0, 0, 0),
    (3, 600, 4, 4, 64, 128, 2, 0.0, 0.0, 0, 0),
    (1, 160, 2, 1, 33, 90, 3, 0.1, -0.1, 0, 0),
    (1, 140, 4, 2, 96, 100, 24, 0.0, 0.2, 99, 23),
    (1, 190, 1, 1, 130, 120, 16, 0.0, 0.0, 0, 0),
    (1, 150, 2, 1, 256, 150, 7, 0.1, 0.0, 0, 0),
    (1, 130, 2, 2, 8, 100, 5, 0.0, 0.0, 3, 2),
    (2, 70, 2, 1, 100, 6, 5, 0.0, 0.1, 0, 0),
    (4, 40, 2, 2, 64, 3, 3, 0.1, 0.0, 2, 2),
    (2, 60, 1, 1, 200, 10, 3, 0.0, 0.0, 0, 0),
    (2, 50, 2, 2, 20, 3, 2, 0.0, 0.0, 0, 0),
]


def test_general_cases_reach_both_kinds_of_general_kernels():
    """Every kernel, by rows and by tiles, at every padded head dim."""
    seen = set()
    for B, N, H, Hkv, D, w1, w2, _, _, h1, h2 in GENERAL_CASES:
        p = _abi.Params()
        p.B, p.N, p.H, p.Hkv, p.D, p.w1, p.w2, p.halo1, p.halo2, p.dtype, p.scale = B, N, H, Hkv, D, w1, w2, h1, h2, _abi.SA_F32, 1.0
        plan = _abi.load().sa_general_plan(ctypes.byref(p))
        seen |= {(max(32, 1 << (D - 1).bit_length()), kernel, plan >> kernel & 1) for kernel in range(4)}
    assert len(seen) == 4 * 4 * 2, sorted({(d, k, r) for d in (32, 64, 128, 256) for k in range(4) for r in (0, 1)} - seen)


@pytest.mark.parametrize("case", GENERAL_CASES)
def test_general_kernels_vs_cpu_oracle_fp32(case):
    """The oracle in fp64; fp32 sums of at most w1 * w2 terms of order 1 in another order: 1e-5 relative."""
    B, N, H, Hkv, D, w1, w2, kb, vb, h1, h2 = case
    ts = so.make_inputs(B, N, H, Hkv, D, seed=13, seed_do=14, halo1=h1, halo2=h2)
    scale = 1.0 / math.sqrt(D)
    cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=kb, v2_bias=vb)
    o, lse, grads = _run(dict(zip(("q", "k1", "k2", "v1", "v2", "do"), ts)), cfg, "general", dtype=torch.float32, halo1=h1, halo2=h2)
    ref = so.forward_backward(*ts, w1, w2, scale, kb, vb, h1, h2, dtype=torch.float64)
    assert so.rel_l2(o.cpu().double(), ref[0]) <= 1e-5
    assert float((lse.cpu() - ref[1]).abs().max()) <= 1e-5
    for nm, g, r in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads, ref[2:]):
        if float(r.abs().max()) < 1e-12:      # one (j, k) pair to a query: no gradient of the scores
            assert float(g.abs().max()) <= 1e-4, nm
        else:
            assert so.rel_l2(g.cpu().double(), r) <= 1e-5, nm


@pytest.mark.parametrize("w1,w2", [(3, 2), (128, 24)])                  # by rows, by tiles
def test_general_kernels_apply_the_scale_before_large_inputs_meet(w1, w2):
    """Q * 2^75 and K2 * 2^55 overflow fp32 together; with a scale of 2^-130 less they do not, and as powers of two are
    exact, the results are those of the inputs as they were (dQ and dK2 but for their factors)."""
    D = 32
    ts = dict(zip(("q", "k1", "k2", "v1", "v2", "do"), so.make_inputs(1, 200, 1, 1, D, seed=53, seed_do=54)))
    cfg = dict(w1=w1, w2=w2, scale=2.0 ** 6, k2_bias=0.0, v2_bias=0.0)
    ts["q"] = ts["q"] * 2.0 ** -8
    o, lse, g = _run(ts, cfg, "general", dtype=torch.float32)
    big = dict(ts, q=ts["q"] * 2.0 ** 75, k2=ts["k2"] * 2.0 ** 55)
    o2, lse2, g2 = _run(big, dict(cfg, scale=2.0 ** (6 - 130)), "general", dtype=torch.float32)
    assert bool(torch.isfinite(o).all()) and torch.equal(o, o2) and torch.equal(lse, lse2)
    for i in (1, 3, 4):
        assert torch.equal(g[i], g2[i]), i


def test_general_kernels_fp32_error_at_wide_heads():
    """The scores' dot products are summed in blocks.  In one chain over 256 products the error of dQ and dK2 against 64 bits
    is 8e-7 here, by a warp with the head dim across its lanes (32 chains of 8, then a tree) 5.4e-7, in blocks of 16
    4.2e-7: the bound is the second."""
    N, D, w1, w2 = 300, 256, 120, 20
    ts = so.make_inputs(1, N, 1, 1, D, seed=51, seed_do=52, bf16_round=False)
    cfg = dict(w1=w1, w2=w2, scale=1.0 / math.sqrt(D), k2_bias=0.0, v2_bias=0.0)
    _, _, grads = _run(dict(zip(("q", "k1", "k2", "v1", "v2", "do"), ts)), cfg, "general", dtype=torch.float32)
    ref = so.forward_backward(*ts, w1, w2, cfg["scale"], dtype=torch.float64)
    for nm, i in (("dq", 0), ("dk2", 2)):
        assert so.rel_l2(grads[i].cpu().double(), ref[2 + i]) <= 5.4e-7, nm


@pytest.mark.parametrize("N,w1,w2", [(160, 40, 8), (300, 128, 8)])      # the second by tiles
def test_general_kernels_keep_values_that_are_not_finite_to_their_windows(N, w1, w2):
    """An infinity in one row of an input reaches the results of the queries that see it, and of the rows that those
    see, and no others, although tiles hold rows of several windows: everything else equals the run on finite inputs."""
    B, H, D = 1, 1, 32
    ts = dict(zip(("q", "k1", "k2", "v1", "v2", "do"), so.make_inputs(B, N, H, H, D, seed=21, seed_do=22)))
    cfg = dict(w1=w1, w2=w2, scale=1.0 / math.sqrt(D), k2_bias=0.0, v2_bias=0.0)
    clean = _run(ts, cfg, "general", dtype=torch.float32)
    x = 70
    for name, last in (("k1", x + w1 - 1), ("v1", x + w1 - 1), ("k2", x + w2 - 1), ("v2", x + w2 - 1), ("q", x), ("do", x)):
        bad = dict(ts)
        bad[name] = ts[name].clone()
        bad[name][0, x, 0, 3] = float("inf")
        o, _, grads = _run(bad, cfg, "general", dtype=torch.float32)
        for got, want, behind in [(o, clean[0], 0), (grads[0], clean[2][0], 0), (grads[1], clean[2][1], w1 - 1), (grads[2], clean[2][2], w2 - 1),
                                  (grads[3], clean[2][3], w1 - 1), (grads[4], clean[2][4], w2 - 1)]:
            far = torch.ones(N, dtype=torch.bool)
            far[max(0, x - behind):last + 1] = False
            assert torch.equal(got[:, far], want[:, far]), name


@pytest.mark.parametrize("N", [3, 5, 9, 17])
def test_backward_of_many_short_sequences(N):
    """More K1/V1 row tiles than multiprocessors, one to a few tiles of 128 virtual rows to each: the hand-overs of
    the stationary rows and accumulators from one row tile to the next, with next to no tiles between them; and,
    with four sequences, a column kernel that fills less than half of the GPU beside the row kernel."""
    H, D, w1, w2 = 4, 64, 12, 16
    for B in (4, 100):
        ts = so.make_inputs(B, N, H, H, D, seed=31, seed_do=32)
        scale = 1.0 / math.sqrt(D)
        cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=0.0, v2_bias=0.0)
        o, _, grads = _run(dict(zip(("q", "k1", "k2", "v1", "v2", "do"), ts)), cfg, "tcgen05")
        ref = so.forward_backward(*ts, w1, w2, scale)
        # (relative: next to no averaging, so |O| reaches 10 and one bf16 rounding of it 10 * 2^-9)
        assert so.rel_l2(o.float().cpu(), ref[0]) <= TOL_G_BF16
        for nm, g, r in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads, ref[2:]):
            assert _grad_err(g, r) <= TOL_G_BF16, nm


@pytest.mark.parametrize("dtype,score", [(torch.float16, 15.0), (torch.bfloat16, 95.0)])
@pytest.mark.parametrize("D,w2", [(64, 24), (128, 32), (64, 5), (128, 60)])
def test_padding_rows_beside_a_query_of_low_scores(dtype, score, D, w2):
    """Query 0 has one (j, k) pair, whose score is -`score`: e^-LSE does not fit 16 bits.  The virtual rows that only fill a
    tile up (delta >= w2, K2 rows before the first) must not bring it into dK1 and dV1.

    Rounding the D products Q * K2 of a score of that size to 16 bits changes it by up to eps * score, eps * score / sqrt(D)
    where the roundings are independent, and P by as much (relative): that is added to the bf16 tolerance."""
    N, w1, scale = 150, 40, 1.0 / math.sqrt(D)
    ts = dict(zip(("q", "k1", "k2", "v1", "v2", "do"), so.make_inputs(1, N, 1, 1, D, seed=41, seed_do=42)))
    z = (score / (D * scale)) ** (1 / 3)
    ts["q"][0, 0], ts["k1"][0, 0], ts["k2"][0, 0] = z, -z, z
    cfg = dict(w1=w1, w2=w2, scale=scale, k2_bias=0.0, v2_bias=0.0)
    o, lse, grads = _run(ts, cfg, "tcgen05", dtype=dtype)
    assert float(lse.flatten()[0]) < -score + 0.5
    tol = TOL_G_BF16 + score / math.sqrt(D) * (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)
    for nm, g, r in zip(("dq", "dk1", "dk2", "dv1", "dv2"), grads, _run(ts, cfg, "general", dtype=dtype)[2]):
        assert bool(torch.isfinite(g).all()) and so.rel_l2(g.float().cpu(), r.float().cpu()) <= tol, nm


@pytest.mark.parametrize("D,w2", [(64, 24), (128, 32), (64, 5), (128, 60), (64, 1), (128, 100)])
def test_forward_with_values_that_are_not_finite(D, w2):
    """A K1 row of -inf in a column where Q * K2 is positive (a mask: its P is 0) leaves the output finite and equal to
    that of the general kernels; a NaN or an infinity in Q, K2 or V2, or a NaN in K1, reaches the queries that see it
    and no others."""
    N, w1, x = 200, 40, 70
    ts = dict(zip(("q", "k1", "k2", "v1", "v2"), so.make_inputs(1, N, 1, 1, D, seed=43, seed_do=44)))
    for nm in ("q", "k2"):
        ts[nm][..., 3] = ts[nm][..., 3].abs() + 0.125
    for name, value in (("k1", -math.inf), ("q", math.nan), ("q", math.inf), ("k2", math.nan), ("v2", math.nan), ("v2", math.inf), ("k1", math.nan)):
        bad = {nm: t.clone() for nm, t in ts.items()}
        bad[name][0, x, 0, 3] = value
        t = [bad[nm].to(DEV).to(torch.bfloat16) for nm in ("q", "k1", "k2", "v1", "v2")]
        (o, lse), (want, want_lse) = (sab.two_simplicial_attn_fwd_kernel(*t, w1, w2, 1.0 / math.sqrt(D), algo=a) for a in ("tcgen05", "general"))
        assert torch.equal(torch.isfinite(o).all(-1), torch.isfinite(want).all(-1)), (name, value)
        fin = torch.isfinite(o) & torch.isfinite(want)
        assert float((o.float() - want.float())[fin].abs().max()) <= 3e-2, (name, value)      # two bf16-rounded results
        if value == -math.inf:
            assert bool(fin.all()) and float((lse - want_lse).abs().max()) <= 2e-2


@pytest.mark.parametrize("N,H,Hkv,D,w1,w2", [(1100, 8, 8, 64, 64, 4), (1100, 8, 8, 64, 64, 16), (1000, 8, 8, 128, 40, 100), (1300, 16, 4, 128, 20, 100),
                                             (1300, 12, 12, 64, 30, 32)])
def test_row_kernel_beside_or_after_the_column_kernel(N, H, Hkv, D, w1, w2):
    """Where the row kernel runs (beside the column kernel, on the multiprocessors that leaves, or after it) does not touch the
    results: a call for all gradients equals two calls for those of either kernel, bit for bit."""
    ts = so.make_inputs(1, N, H, Hkv, D, seed=61, seed_do=62)
    cfg = dict(w1=w1, w2=w2, scale=1.0 / math.sqrt(D), k2_bias=0.0, v2_bias=0.0)
    ins = dict(zip(("q", "k1", "k2", "v1", "v2", "do"), ts))
    whole = _run(ins, cfg, "tcgen05")[2]
    col, row = _run(ins, cfg, "tcgen05", need=(False, True, False, True, False))[2], _run(ins, cfg, "tcgen05", need=(True, False, True, False, True))[2]
    for i, other in ((0, row), (1, col), (2, row), (3, col), (4, row)):
        assert bool(torch.isfinite(whole[i]).all()) and torch.equal(whole[i], other[i]), i


@pytest.mark.parametrize("name", ["q", "k1", "k2", "v1", "v2", "do"])
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_expanded_inputs(name, dim):
    """An input that is expanded (stride 0) over the batch, the rows or the heads gives what its copy gives."""
    B, N, H, D, w1, w2 = 2, 150, 2, 64, 50, 24
    ts = {nm: t.to(DEV).to(torch.bfloat16) for nm, t in zip(("q", "k1", "k2", "v1", "v2", "do"), so.make_inputs(B, N, H, H, D, seed=71, seed_do=72))}
    ts[name] = ts[name].narrow(dim, 0, 1).expand_as(ts[name])

    def both(t):
        o, lse = sab.two_simplicial_attn_fwd_kernel(*(t[nm] for nm in ("q", "k1", "k2", "v1", "v2")), w1, w2, 0.125, algo="tcgen05")
        return (o, lse) + sab.two_simplicial_attn_bwd(*(t[nm] for nm in ("q", "k1", "k2", "v1", "v2")), o, lse, t["do"], w1, w2, 0.125)

    for a, b in zip(both(ts), both(dict(ts, **{name: ts[name].contiguous()}))):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", ["q", "k2", "v2", "k1"])
def test_forward_with_rows_in_reverse_order(name):
    """A negative row stride, which a tensor map does not hold, takes the general kernels."""
    B, N, H, D, w1, w2 = 1, 150, 2, 64, 50, 24
    names = ("q", "k1", "k2", "v1", "v2")
    ts = {nm: t.to(DEV).to(torch.bfloat16) for nm, t in zip(names, so.make_inputs(B, N, H, H, D, seed=73, seed_do=74))}
    want, want_lse = sab.two_simplicial_attn_fwd_kernel(*(ts[nm] for nm in names), w1, w2, 0.125)
    back = ts[name].flip(1).contiguous()
    o, lse = torch.empty_like(want), torch.empty_like(want_lse)
    p = host._make_params(*(ts[nm] for nm in names), o, w1, w2, 0.125, 0.0, 0.0, 0, 0, "auto")
    setattr(p, name, _abi.Strides(back.stride(0), -back.stride(1), back.stride(2)))
    ptr = {nm: t.data_ptr() for nm, t in ts.items()}
    ptr[name] = back[:, N - 1:].data_ptr()
    ws = torch.zeros(256, dtype=torch.uint8, device=DEV)
    rc = _abi.load().sa_forward(ctypes.byref(p), *(ctypes.c_void_p(ptr[nm]) for nm in names), host._ptr(o), host._ptr(lse), host._ptr(ws), ws.numel(),
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _abi.SA_OK
    assert float((o.float() - want.float()).abs().max()) <= 3e-2 and float((lse - want_lse).abs().max()) <= 1e-2      # (two bf16-rounded results)
