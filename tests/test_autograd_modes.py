"""The operator under torch's modes: which calls the native binding makes itself, and that tracing, forward-mode
differentiation, functorch transforms, tensor subclasses, saved-tensor hooks and CUDA graphs get what an autograd
function gives them."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

import simplical_attn_b200 as sab
from simplical_attn_b200 import _abi


class Sub(torch.Tensor):
    pass


def _inputs(device, seed=0, grad=False):
    g = torch.Generator(device=device).manual_seed(seed)
    return [torch.randn(1, 100, 2, 64, generator=g, device=device).to(torch.bfloat16).requires_grad_(grad) for _ in range(5)]


def _with(ts, i, t):
    return ts[:i] + [t] + ts[i + 1:]


def test_binding_takes_plain_calls_only():
    """(CPU tensors: the choice is made before anything looks at the device.)"""
    plain, ts = _abi.binding().plain, _inputs("cpu")
    assert plain(*ts) and plain(*_inputs("cpu", grad=True))
    for i in range(5):
        assert plain(*_with(ts, i, torch.nn.Parameter(ts[i])))
        assert not plain(*_with(ts, i, ts[i].as_subclass(Sub)))
        assert not plain(*_with(ts, i, None))
        with fwAD.dual_level():
            assert plain(*ts)                                     # a level alone changes nothing
            assert not plain(*_with(ts, i, fwAD.make_dual(ts[i], torch.ones_like(ts[i]))))
        seen = []
        torch.func.vmap(lambda t: seen.append(plain(*_with(ts, i, t))) or t)(ts[i])
        torch.jit.trace(lambda t: seen.append(plain(*_with(ts, i, t))) or t + 0, ts[i], check_trace=False)
        assert seen == [False, False]
    assert plain(*ts)                                             # (the modes were left)


@pytest.mark.gpu
def test_traced_module_replays_the_operator():
    m = sab.TwoSimplicialAttention(64, 50, 24)
    for grad in (False, True):
        traced = torch.jit.trace(m, _inputs("cuda", grad=grad), check_trace=False)
        new = _inputs("cuda", seed=5, grad=grad)
        o, want = traced(*new), m(*new)
        assert torch.equal(o, want)
        if grad:
            for a, b in zip(torch.autograd.grad(o, new, torch.ones_like(o)), torch.autograd.grad(want, new, torch.ones_like(o))):
                assert torch.equal(a, b)


@pytest.mark.gpu
def test_tangents_and_transforms_are_refused():
    m, ts = sab.TwoSimplicialAttention(64, 50, 24), _inputs("cuda")
    with fwAD.dual_level():
        assert torch.equal(m(*ts), m(*_inputs("cuda")))
        for i in range(5):
            with pytest.raises(NotImplementedError):
                m(*_with(ts, i, fwAD.make_dual(ts[i], torch.ones_like(ts[i]))))
    for f in (lambda: torch.func.vmap(lambda q: m(q, *ts[1:]))(ts[0][None]), lambda: torch.func.jvp(lambda q: m(q, *ts[1:]), (ts[0],), (ts[0],)),
              lambda: torch.func.grad(lambda q: m(q, *ts[1:]).float().sum())(ts[0])):
        with pytest.raises(RuntimeError, match="setup_context"):
            f()


@pytest.mark.gpu
def test_tensor_subclasses_are_kept():
    m, ts = sab.TwoSimplicialAttention(64, 50, 24), _inputs("cuda", grad=True)
    want = m(*ts)
    want_g = torch.autograd.grad(want, ts, torch.ones_like(want))
    for i in range(5):
        sub = _inputs("cuda")
        sub[i] = sub[i].as_subclass(Sub)
        sub = [t.requires_grad_() for t in sub]
        o = m(*sub)
        assert type(o) is (Sub if i == 0 else torch.Tensor) and torch.equal(o.as_subclass(torch.Tensor), want)
        o_k, lse = sab.two_simplicial_attn_fwd_kernel(*sub, 50, 24, m.scale)
        assert type(o_k) is type(o) and type(lse) is torch.Tensor
        for a, b in zip(torch.autograd.grad(o, sub, torch.ones_like(o)), want_g):
            assert torch.equal(a.as_subclass(torch.Tensor), b)
    sab.check_device_status()


@pytest.mark.gpu
def test_calls_without_the_binding(monkeypatch):
    m, ts = sab.TwoSimplicialAttention(64, 50, 24), _inputs("cuda", grad=True)
    want = m(*ts)
    want_g = torch.autograd.grad(want, ts, torch.ones_like(want))
    monkeypatch.setattr(_abi, "_binding", False)
    o = m(*ts)
    assert torch.equal(o, want) and all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(o, ts, torch.ones_like(o)), want_g))
    sab.check_device_status()


@pytest.mark.gpu
def test_saved_tensor_hooks_and_checkpointing():
    from torch.utils.checkpoint import checkpoint
    m, ts = sab.TwoSimplicialAttention(64, 50, 24), _inputs("cuda", grad=True)
    one = torch.ones_like(ts[0])
    want = torch.autograd.grad(m(*ts), ts, one)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda()):
        o = m(*ts)
    assert len(packed) == 7                                       # the inputs, O and LSE
    for got in (torch.autograd.grad(o, ts, one), torch.autograd.grad(checkpoint(m, *ts, use_reentrant=False), ts, one)):
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
def test_captured_step_replays_on_new_inputs():
    m, ts = sab.TwoSimplicialAttention(64, 50, 24), _inputs("cuda", grad=True)
    one = torch.ones_like(ts[0])

    def step(x):
        o = m(*x)
        return (o,) + torch.autograd.grad(o, x, one)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(ts)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step(ts)
    new = _inputs("cuda", seed=9, grad=True)
    with torch.no_grad():
        for t, n in zip(ts, new):
            t.copy_(n)
    graph.replay()
    for a, b in zip(out, step(new)):
        assert torch.equal(a, b)
