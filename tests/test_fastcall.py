"""The native GEMM and attention calls take what they can launch as it lies, and leave everything else to the Python statements."""
import math
import re
import sys
import types

import pytest
import torch

import kareus_b200.kernels as K


class _Sub(torch.Tensor):
    pass


def test_calls_without_a_launch_are_left_alone():
    from kareus_b200.kernels import build, cuda as KC
    if not (build.LIB.exists() and build.FASTCALL.exists()):
        pytest.skip("native library not built")
    KC.lib()
    a = torch.randn(8, 16, dtype=torch.bfloat16)
    for x in (a, a.float(), a.as_subclass(_Sub), a.to_sparse(), torch.empty(8, 16, device="meta"), None, 3):
        assert K._FAST.gemm(x, a, False, True, None) is None
        assert K._FAST.attention_fwd(x, a, a, 1.0, True, 0) is None
    assert torch.equal(K.gemm(a, a), K.ref.gemm(a, a))


@pytest.mark.parametrize("module", [None, types.SimpleNamespace(torch_version="1.0"), types.SimpleNamespace()])
def test_library_loads_without_the_module(monkeypatch, module):
    """Missing, built for another PyTorch, built from older sources: every call takes the Python statements."""
    from kareus_b200.kernels import build, cuda as KC
    if not build.LIB.exists():
        pytest.skip("native library not built")
    monkeypatch.setattr(KC, "_LIB", None)
    monkeypatch.setattr(K, "_FAST", None)
    monkeypatch.delattr(K, "_fastcall", raising=False)
    monkeypatch.setitem(sys.modules, "kareus_b200.kernels._fastcall", module)
    with pytest.warns(RuntimeWarning, match="cannot be loaded"):
        KC.lib()
    assert KC.is_loaded() and K._FAST is None
    a = torch.randn(8, 16, dtype=torch.bfloat16)
    assert torch.equal(K.gemm(a, a), K.ref.gemm(a, a))


def test_build_goes_on_without_the_module(monkeypatch, tmp_path):
    from kareus_b200.kernels import build

    def fails(force=False):
        raise RuntimeError("no Python.h")
    monkeypatch.setattr(build, "build_fastcall", fails)
    monkeypatch.setattr(build, "is_current", lambda: True)
    monkeypatch.setattr(build, "FASTCALL", tmp_path / "_fastcall.so")
    build.FASTCALL.write_bytes(b"of other sources")
    with pytest.warns(RuntimeWarning, match="no Python.h"):
        assert build.build() == build.LIB
    assert not build.FASTCALL.exists()


def test_both_sides_of_a_native_call_include_its_signature():
    from kareus_b200.kernels import build
    header = (build.CSRC / "native_calls.h").read_text()
    called = set(re.findall(r"\bkb_\w+(?=\()", build.FASTCALL_SRC.read_text()))
    assert called == set(re.findall(r"\bkb_\w+(?=\()", header)) and len(called) == 7
    for name in called:
        sources = [p for p in build.CSRC.glob("*.cu") if re.search(rf'extern "C" \w+ {name}\(', p.read_text())]
        assert len(sources) == 1 and '#include "native_calls.h"' in sources[0].read_text(), name
    assert build.CSRC / "native_calls.h" in build.FASTCALL_DEPS


def _outcome(fn):
    """Result of a call, or the type of its error."""
    try:
        r = fn()
    except Exception as e:
        return type(e)
    torch.cuda.synchronize()
    return r if isinstance(r, tuple) else (r,)


def _same_as_python(monkeypatch, fn, direct, native):
    """``fn`` with and without the native calls; ``direct`` is the native call itself, which takes the arguments or (``native``
    false) leaves them alone."""
    from kareus_b200.kernels import cuda as KC, launch_count
    KC.lib()
    KC.status_word(torch.device("cuda", torch.cuda.current_device()))
    assert K._FAST is not None and (direct() is not None) == native
    n0 = launch_count()
    fast = _outcome(fn)
    n1 = launch_count()
    with monkeypatch.context() as m:
        m.setattr(K, "_FAST", None)
        slow = _outcome(fn)
    assert launch_count() - n1 == n1 - n0
    assert isinstance(fast, type) == isinstance(slow, type), (fast, slow)
    if isinstance(fast, type):
        assert fast is slow
        return
    for a, b in zip(fast, slow, strict=True):
        assert type(a) is type(b) and a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype
        assert a.requires_grad == b.requires_grad and torch.equal(a, b)


def _bf16(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "rows", "param", "odd_rows", "offset", "cols", "subclass", "fp32", "three", "one_row",
                                  "no_rows", "mismatch"])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
def test_gemm_forms(monkeypatch, form, ta, tb):
    torch.manual_seed(0)
    M, N, Kd = 72, 136, 200
    a, b = _bf16(*((Kd, M) if ta else (M, Kd))), _bf16(*((N, Kd) if tb else (Kd, N)))
    wide = lambda t, pad, off: torch.cat([torch.zeros(t.shape[0], off, device="cuda").bfloat16(), t,
                                          torch.zeros(t.shape[0], pad, device="cuda").bfloat16()], 1)[:, off:off + t.shape[1]]
    a, b = {
        "plain": lambda: (a, b), "rows": lambda: (wide(a, 24, 8), wide(b, 8, 16)),
        "param": lambda: (a, torch.nn.Parameter(b)), "odd_rows": lambda: (wide(a, 3, 0), b), "offset": lambda: (wide(a, 7, 1), b),
        "cols": lambda: (a.t().contiguous().t(), b), "subclass": lambda: (a.as_subclass(_Sub), b), "fp32": lambda: (a.float(), b.float()),
        "three": lambda: (a[None], b), "one_row": lambda: (a[:, :1] if ta else a[:1], b),
        "no_rows": lambda: (a[:, :0] if ta else a[:0], b), "mismatch": lambda: (a[8:] if ta else a[:, 8:], b),
    }[form]()
    _same_as_python(monkeypatch, lambda: K.gemm(a, b, trans_a=ta, trans_b=tb), lambda: K._FAST.gemm(a, b, ta, tb, None),
                    form in ("plain", "rows", "param", "one_row"))


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [64, 4096])
@pytest.mark.parametrize("form", ["plain", "view", "transposed", "bf16", "shape"])
def test_accumulating_gemm_forms(monkeypatch, tokens, form):
    torch.manual_seed(0)
    from kareus_b200.kernels import cuda as KC
    dy, x = _bf16(tokens, 5120), _bf16(tokens, 3072)
    # over 4096 rows the parts of a K split add in order, through a workspace
    assert (KC.lib().kb_gemm_accum_scratch_floats(5120, 3072, tokens, 0) > 0) == (tokens == 4096)
    base = torch.randn(5120, 3072, device="cuda")

    def out():
        return {"plain": lambda: base.clone(), "view": lambda: torch.cat([base, base])[5120:], "transposed": lambda: base.t().contiguous().t(),
                "bf16": lambda: base.bfloat16(), "shape": lambda: base[:8].clone()}[form]()

    def call():
        c = out()
        r = K.gemm(dy, x, trans_a=True, trans_b=False, accumulate=c)
        assert r is c
        return r
    _same_as_python(monkeypatch, call, lambda: K._FAST.gemm(dy, x, True, False, out()), form in ("plain", "view"))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["packed", "four_dims", "off_keys", "batch_major", "int_scale", "float_offset", "kv_len", "wide_head",
                                  "groups", "no_queries"])
def test_attention_forms(monkeypatch, form):
    torch.manual_seed(0)
    s, b, g, rep, d = 70, 2, 2, 2, 128
    packed = _bf16(s, b, g, (rep + 2) * d)
    q, k, v = packed[..., :rep * d].unflatten(-1, (rep, d)), packed[..., rep * d:-d], packed[..., -d:]
    scale, off, kw = 1 / math.sqrt(d), 0, {}
    if form == "four_dims":
        q = q.reshape(s, b, g * rep, d)
    elif form == "off_keys":
        k, v, off = _bf16(s + 128, b, g, d), _bf16(s + 128, b, g, d), 128
    elif form == "batch_major":
        k, v = (t.transpose(0, 1).contiguous().transpose(0, 1) for t in (k, v))
    elif form == "int_scale":
        scale = 1
    elif form == "float_offset":
        off = 0.0
    elif form == "kv_len":
        kw = {"kv_len": 33}
    elif form == "wide_head":
        q, k, v = _bf16(s, b, g, rep, 64), _bf16(s, b, g, 64), _bf16(s, b, g, 64)
    elif form == "groups":
        k, v = k[:, :, :1], v[:, :, :1]
    elif form == "no_queries":
        q = q[:0]
    native = form in ("packed", "four_dims", "off_keys", "batch_major")
    fwd = lambda: K.attention_fwd(q, k, v, scale, causal=True, q_offset=off, **kw)
    _same_as_python(monkeypatch, fwd, lambda: None if kw else K._FAST.attention_fwd(q, k, v, scale, True, off), native)
    r = _outcome(fwd)
    if isinstance(r, type):
        return
    out, lse = r
    do = _bf16(*out.shape)
    # every dK and dV has one sum of its own, and dQ the contributions of at most two key tiles: bitwise the same each time
    _same_as_python(monkeypatch, lambda: K.attention_bwd(do, q, k, v, out, lse, scale, causal=True, q_offset=off, **kw),
                    lambda: None if kw else K._FAST.attention_bwd(q, k, v, scale, True, off, do, out, lse), native)


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("accumulate", [False, True])
def test_errors_name_the_shape(monkeypatch, native, accumulate):
    """An error of the runtime that nobody has fetched (a device number out of range, refused on the host) is reported by the next call."""
    import ctypes
    from kareus_b200.kernels import cuda as KC
    KC.lib()
    a, b = _bf16(72, 200), _bf16(136, 200)
    c = torch.zeros(72, 136, device="cuda") if accumulate else None
    K.gemm(a, b, accumulate=c)
    assert (K._FAST.gemm(a, b, False, True, c) is not None)
    if not native:
        monkeypatch.setattr(K, "_FAST", None)
    assert ctypes.CDLL("libcudart.so.12").cudaSetDevice(1 << 20) != 0
    with pytest.raises(KC.KernelError, match="gemm M=72 N=136 K=200 failed"):
        K.gemm(a, b, accumulate=c)
    torch.cuda.synchronize()
    K.gemm(a, b, accumulate=c)


@pytest.mark.gpu
def test_transforms_and_switches(monkeypatch):
    a, b = _bf16(4, 64, 64), _bf16(64, 64)
    K.gemm(a[0], b)
    with pytest.raises(RuntimeError, match="storage"):              # no data pointer under vmap: refused, as by the Python statements
        torch.vmap(lambda x: K.gemm(x, b))(a)
    monkeypatch.setenv("KAREUS_B200_LIBRARY_BASELINE", "1")
    n = K.launch_count()
    K.gemm(a[0], b)
    assert K.launch_count() == n
