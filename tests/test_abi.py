"""CPU-side checks of the C-ABI library: it loads, exports every symbol the header declares, and
its argument validation and kernel selection work without a GPU (no compute is launched)."""
import ctypes
import multiprocessing
import os
import re

import pytest

from simplical_attn_b200 import _abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "simplicial_attn_b200.h")


def declared_symbols():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(sa_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_exported():
    lib = _abi.load()
    syms = declared_symbols()
    assert set(_abi.EXPORTS) <= set(syms)
    for s in syms:
        assert hasattr(lib, s), s


def test_struct_layout_matches_header():
    # 11 int32 + 3 float + 12 x (3 x int64)
    assert ctypes.sizeof(_abi.Params) == 11 * 4 + 3 * 4 + 12 * 24
    assert _abi.Params.q.offset == 56


def _params(**kw):
    p = _abi.Params()
    p.B, p.N, p.H, p.Hkv, p.D, p.w1, p.w2 = 1, 64, 4, 2, 128, 16, 8
    p.dtype, p.algo, p.scale = _abi.SA_BF16, _abi.SA_ALGO_AUTO, 0.1
    for name in ("q", "k1", "k2", "v1", "v2", "o", "d_o", "dq", "dk1", "dk2", "dv1", "dv2"):
        setattr(p, name, _abi.Strides(64 * 4 * 128, 4 * 128, 128))
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def test_validation_codes():
    lib = _abi.load()
    nul = ctypes.c_void_p(0)
    args = [nul] * 8 + [0, nul]
    assert lib.sa_forward(ctypes.byref(_params(H=3)), *args) == 2            # H % Hkv
    assert lib.sa_forward(ctypes.byref(_params(w1=0)), *args) == 2
    assert lib.sa_forward(ctypes.byref(_params(halo1=-1)), *args) == 2
    assert lib.sa_forward(ctypes.byref(_params(D=512)), *args) == 4
    assert lib.sa_forward(ctypes.byref(_params(dtype=7)), *args) == 4
    assert lib.sa_forward(ctypes.byref(_params()), *args) == 1               # NULL pointers
    assert "NULL" in _abi.strerror(1)
    with pytest.raises(_abi.SimplicialAttnError):
        _abi.check("sa_forward", 2)


def test_kernel_selection():
    lib = _abi.load()
    r = lambda **kw: lib.sa_resolve_algo(ctypes.byref(_params(**kw)))
    assert r() == _abi.SA_ALGO_TCGEN05
    assert r(D=64) == _abi.SA_ALGO_TCGEN05
    assert r(D=32) == _abi.SA_ALGO_GENERAL
    assert r(dtype=_abi.SA_F32) == _abi.SA_ALGO_GENERAL
    assert r(dtype=_abi.SA_F16) == _abi.SA_ALGO_TCGEN05
    assert r(w2=200, N=4096) == _abi.SA_ALGO_TCGEN05                         # two passes over chunks of the K2 window
    assert r(w2=1025, N=4096) == _abi.SA_ALGO_GENERAL
    assert r(w2=200, N=64) == _abi.SA_ALGO_TCGEN05                           # window clipped to 64 rows
    assert r(algo=_abi.SA_ALGO_GENERAL) == _abi.SA_ALGO_GENERAL
    assert r(D=32, algo=_abi.SA_ALGO_TCGEN05) == -4
    assert r(q=_abi.Strides(1000, 100, 4)) == _abi.SA_ALGO_GENERAL           # rows not 16-byte aligned
    assert r(H=5) == -2
    assert lib.sa_forward_workspace_size(ctypes.byref(_params())) == 256
    assert lib.sa_backward_workspace_size(ctypes.byref(_params())) >= 256
    # a K2 window of more than 128 positions: room for one more O (bf16) and LSE (fp32) in the forward, for one
    # more set of gradients in the backward
    wide, narrow = _params(w2=200, N=4096), _params(w2=100, N=4096)
    assert lib.sa_forward_workspace_size(ctypes.byref(wide)) == 256 + 4096 * 4 * 128 * 2 + 4 * 4096 * 4
    extra = lib.sa_backward_workspace_size(ctypes.byref(wide)) - lib.sa_backward_workspace_size(ctypes.byref(narrow))
    assert extra >= (4096 * 4 * 128 + 4 * 4096 * 2 * 128) * 2


def test_general_kernels_take_short_windows_by_rows():
    """Problems far from the line between the two kinds of general kernels, as measured: fp32, by rows and by tiles, us, forward
    (479 / 1100 at w 16/33, 4314 / 1698 at w 64/64, 12 / 486 for 4096 sequences of one row)."""
    lib = _abi.load()
    plan = lambda **kw: lib.sa_general_plan(ctypes.byref(_params(dtype=_abi.SA_F32, Hkv=4, **kw)))
    assert plan(B=4, N=512, D=128, w1=16, w2=33) == 15
    assert plan(B=4, N=512, D=128, w1=64, w2=64) == 0
    assert plan(B=4096, N=1, D=64, w1=64, w2=64) == 15
    assert plan(B=4, N=512, D=256, w1=4, w2=100) == 15
    assert plan(B=1, N=512, D=64, w1=512, w2=512) == 0
    assert plan(B=4, N=512, D=32, w1=32, w2=33) == 0
    assert plan(N=64, D=64, w1=4, w2=4, halo1=2**20, halo2=2**20) >= 0            # (no overflow)
    assert plan(w1=0) == -2


def test_python_layer_rejects_cpu_tensors():
    import torch
    import simplical_attn_b200 as sab
    x = torch.zeros(1, 8, 1, 16)
    with pytest.raises(RuntimeError):
        sab.two_simplicial_attention(x, x, x, x, x, 4, 4)
    m = sab.TwoSimplicialAttention(16, 4, 4)
    assert len(m.state_dict()) == 0 and abs(m.scale - 0.25) < 1e-12


def test_host_pipeline_chunk_plan():
    from simplical_attn_b200.host_pipeline import plan_chunks
    # whole sequences in the middle, a small head group first and last
    assert plan_chunks(3, 16) == [(0, 0, 4), (0, 4, 16), (1, 0, 16), (2, 0, 12), (2, 12, 16)]
    assert plan_chunks(1, 16) == [(0, 0, 4), (0, 4, 12), (0, 12, 16)]
    assert plan_chunks(2, 1) == [(0, 0, 1), (1, 0, 1)]
    assert plan_chunks(1, 2) == [(0, 0, 1), (0, 1, 2)]
    for B, Hkv in ((1, 1), (2, 2), (5, 3), (16, 16), (2, 8)):
        ch = plan_chunks(B, Hkv)
        assert sorted(ch) == ch and all(h1 > h0 for _, h0, h1 in ch)
        assert sum(h1 - h0 for _, h0, h1 in ch) == B * Hkv


def test_cpu_list_parsing_and_numa_helper_without_a_gpu():
    from simplical_attn_b200 import host_pipeline as hp
    assert hp._cpu_list("0-3,8,10-11\n") == {0, 1, 2, 3, 8, 10, 11}
    assert hp._cpu_list("") == set()
    assert hp.local_cpus("cuda:0") is None or isinstance(hp.local_cpus("cuda:0"), set)      # no GPU here: None
    with hp.near("cuda:0") as took_effect:                                                   # must be harmless
        assert took_effect in (False, True)


def test_binding_without_a_compiler(monkeypatch):
    """A binding that was built for another torch (or not at all) is not loaded where it cannot be built again: calls go
    through ctypes, after a warning."""
    import torch
    import simplical_attn_b200 as sab
    from simplical_attn_b200 import build as b
    assert _abi.binding() is not None and not b.binding_stale()
    x = torch.zeros(1, 8, 1, 16)
    for change in (lambda m: m.setattr(torch, "__version__", "0.0"), lambda m: m.setattr(b, "BINDING", b.BINDING + ".missing")):
        with monkeypatch.context() as m:
            m.setattr(_abi, "_binding", None)
            m.setattr(b, "have_host_compiler", lambda: False)
            change(m)
            assert b.binding_stale()
            with pytest.warns(RuntimeWarning, match="no C\\+\\+ compiler"):
                assert _abi.binding() is None
            with pytest.raises(RuntimeError, match="CUDA tensors only"):      # (this layer's check of the call)
                sab.two_simplicial_attention(x, x, x, x, x, 4, 4)
    assert _abi.binding() is not None


def _rebuild(path):
    from simplical_attn_b200 import build as b
    _abi.load()                        # (what the binding is linked against)
    b.LIB_DIR, b.BINDING, b.BINDING_STAMP = path, os.path.join(path, "sa_torch.so"), os.path.join(path, "sa_torch.so.sources")
    b.build_binding()
    return _abi._import(b.BINDING).devices()


def test_binding_is_built_once_by_processes_that_start_together(tmp_path, monkeypatch):
    """Several processes find the binding missing (the ranks of a job on a machine with another torch): one builds it, and
    every one of them loads a whole file.  The compiler here copies the built one in two halves, with a pause, and counts."""
    from simplical_attn_b200 import build as b
    cxx = tmp_path / "g++"
    cxx.write_text(f"""#!/bin/sh
echo run >> {tmp_path}/runs
while [ "$1" != -o ]; do shift; done
head -c 100000 {b.BINDING} > "$2"; sleep 0.5; tail -c +100001 {b.BINDING} >> "$2"
""")
    cxx.chmod(0o755)
    monkeypatch.setenv("PATH", f"{tmp_path}:{os.environ['PATH']}")
    with multiprocessing.get_context("spawn").Pool(3) as pool:
        assert pool.map(_rebuild, [str(tmp_path / "lib")] * 3, chunksize=1) == [[]] * 3
    assert (tmp_path / "runs").read_text() == "run\n"
    assert sorted(os.listdir(tmp_path / "lib")) == [".lock", "sa_torch.so", "sa_torch.so.sources"]


def test_library_staleness_follows_source_contents(tmp_path, monkeypatch):
    """The library counts as current exactly while the digest recorded at build time matches the sources,
    whatever the file times say."""
    from simplical_attn_b200 import build as b
    assert not b._stale()                                   # built by the session fixture / build step
    digest = b.source_digest()
    assert open(b.STAMP).read().strip() == digest
    monkeypatch.setattr(b, "NVCC_FLAGS", b.NVCC_FLAGS + ["-DSOMETHING_ELSE"])
    assert b.source_digest() != digest and b._stale()       # other flags (or sources): stale
