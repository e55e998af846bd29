"""The native call path (``csrc/host.cpp``) against the Python path it stands in for -- the one a replaced
``flash_cuda.fwd`` or a tracing compiler gets: same bits forward and backward, through casts, strided inputs and
autocast; the same refusals; and the autograd contract (one differentiation, inputs changed in between)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,autocast,strided", [
    (torch.float32, None, False), (torch.float32, torch.bfloat16, False), (torch.bfloat16, None, True),
    (torch.float16, None, False)])
def test_native_and_python_paths_agree(dtype, autocast, strided, monkeypatch):
    from machinelearning_b200 import flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    torch.manual_seed(0)
    B, T, H, Hkv, D = 2, 70, 4, 2, 64
    mk = lambda h: torch.randn(B, h, T, D, device="cuda", dtype=dtype).transpose(1, 2)
    if not strided:
        mk = lambda h: torch.randn(B, T, h, D, device="cuda", dtype=dtype)
    q, k, v = (mk(h).requires_grad_() for h in (H, Hkv, Hkv))
    do = torch.randn(B, T, H, D, device="cuda", dtype=autocast or dtype)

    def both(**kw):
        with torch.autocast("cuda", dtype=autocast or torch.bfloat16, enabled=autocast is not None):
            y = fc.flash_attn(q, k, v, **kw)
        return (y, *torch.autograd.grad(y, (q, k, v), do))

    for kw in ({}, dict(window=20, sinks=3), dict(block=16), dict(use_mma=False, scale=0.3)):
        native = both(**kw)
        with monkeypatch.context() as m:
            m.setattr(fc, "fwd", lambda *a: fc._own_fwd(*a))
            general = both(**kw)
        assert all(torch.equal(a, b) and a.dtype == b.dtype for a, b in zip(native, general))


def test_refusals_and_the_autograd_contract():
    from machinelearning_b200 import flash_cuda as fc
    q = torch.randn(1, 16, 2, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    for bad in (dict(window=4, sinks=4), dict(block=-1), dict(block=4, window=8)):
        with pytest.raises(ValueError):
            fc.flash_attn(q, q, q, **bad)
    with pytest.raises(ValueError):
        fc.flash_attn(q, q[..., :48], q)
    with pytest.raises(ValueError):
        fc.flash_attn(q.float(), q.float(), q.float(), use_mma=True)
    do = torch.randn_like(q, requires_grad=True)
    g, = torch.autograd.grad(fc.flash_attn(q, q, q), q, do, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        g.sum().backward()
    y = fc.flash_attn(q, q, q)
    with torch.no_grad():
        q.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward(do)
    y = fc.flash_attn(q, q, q)
    y.backward(do)
    with pytest.raises(RuntimeError, match="second time"):
        y.backward(do)


def test_arguments_as_the_python_path_takes_them():
    """Numbers of any kind, as int() and float() read them; what is no tensor raises instead of being read as one."""
    import numpy as np
    from machinelearning_b200 import flash_cuda as fc
    q = torch.randn(1, 40, 2, 64, device="cuda", dtype=torch.bfloat16)
    want = fc.flash_attn(q, q, q, 0.25, window=8, sinks=2)
    for window, sinks, scale in ((8.0, 2.0, np.float32(0.25)), (np.int64(8), True + 1, torch.tensor(0.25)),
                                 (torch.tensor(8), torch.tensor(2, device="cuda"), "0.25")):
        assert torch.equal(fc.flash_attn(q, q, q, scale, window=window, sinks=sinks), want)
        assert torch.equal(fc.fwd(q, q, q, scale, 1, window, sinks)[0], want)
    k = q.transpose(1, 2).contiguous()
    want = fc.flash_attn_cached(q, k, k, 0.25, causal=True, window=8, sinks=2)
    assert torch.equal(fc.flash_attn_cached(q, k, k, np.float64(0.25), causal=np.bool_(True), window=8.0, sinks=2.0), want)
    for bad in ({"window": None}, {"window": "x"}, {"use_mma": np.ones(2)}):
        with pytest.raises((TypeError, ValueError)):
            fc.flash_attn(q, q, q, **bad)
    with pytest.raises(TypeError):
        fc.fwd(q, None, q, 0.25, True)
    o, lse = fc.fwd(q, q, q, 0.25, True)
    with pytest.raises(TypeError):
        fc.bwd(None, q, q, q, o, lse, 0.25, True)
