"""What the mask hides does not reach a row, whatever stands there: infinities and NaN in hidden rows of K, V, Q and dO
leave the visible pairs' results as they are, bit for bit, in the fp32 kernels and the small cached blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BAD = [float("nan"), float("inf"), float("-inf")]


def _spoil(t, rows, dim):
    """A copy of `t` with every element of these rows of dimension `dim` NaN or infinite."""
    t = t.clone()
    bad = torch.tensor(BAD, device=t.device, dtype=t.dtype).repeat(t.shape[-1])[:t.shape[-1]]
    t.transpose(0, dim)[rows] = bad
    return t


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["fp32", "bf16"])
@pytest.mark.parametrize("B,T,H,Hkv,D,window,sinks,block", [
    (1, 100, 2, 1, 64, 0, 0, 0), (2, 130, 4, 2, 128, 0, 0, 0), (1, 200, 2, 2, 32, 40, 4, 0), (1, 150, 2, 2, 64, 0, 0, 48),
    (13, 150, 16, 16, 64, 0, 0, 0)])
def test_hidden_rows_of_the_fp32_kernels(B, T, H, Hkv, D, window, sinks, block, dtype):
    from machinelearning_b200 import flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = (torch.randn(B, T, h, D, device="cuda", generator=g).to(dtype) for h in (H, Hkv, Hkv, H))

    def passes(q, k, v, do):
        o, lse = fc.fwd(q, k, v, D ** -0.5, False, window, sinks, block)
        return (o, *fc.bwd(do, q, k, v, o, lse, D ** -0.5, False, window, sinks, block=block))

    clean = passes(q, k, v, do)
    # the last tokens: no earlier query sees them (a block-causal query sees its own block's)
    n = T - 1 - (T - 1) % block if block else T - 3
    late = slice(n, T)
    spoilt = passes(q, _spoil(k, late, 1), _spoil(v, late, 1), do)
    for a, b in zip(clean[:2], spoilt[:2]):                                          # o, dq
        assert torch.equal(a[:, :n], b[:, :n]) and not torch.isfinite(b[:, n:].float()).all()
    # the first queries: later keys are not seen by them, so their dK and dV do not hear of them
    m = block if block else 5
    early = slice(0, m)
    spoilt = passes(_spoil(q, early, 1), k, v, _spoil(do, early, 1))
    for a, b in zip(clean[2:], spoilt[2:]):                                          # dk, dv
        assert torch.equal(a[:, m:], b[:, m:]) and not torch.isfinite(b[:, :m].float()).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16], ids=["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("B,T,H,Hkv,L,D", [(1, 1, 4, 2, 300, 64), (2, 5, 2, 2, 90, 128), (1, 12, 4, 4, 2100, 64),
                                           (1, 60, 4, 2, 200, 32), (1, 9, 2, 2, 1500, 128), (1, 100, 2, 2, 250, 128)])
def test_hidden_rows_of_a_cache(B, T, H, Hkv, L, D, dtype):
    """Slots of the cache that no query may see (positions beyond every query's) and, of the block itself, later tokens."""
    from machinelearning_b200 import flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    g = torch.Generator(device="cuda").manual_seed(L)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)
    q, k, v = mk(B, T, H, D), mk(B, Hkv, L, D), mk(B, Hkv, L, D)
    qpos = torch.arange(5000, 5000 + T, device="cuda")
    kpos = torch.cat([torch.arange(5000 - L + T, 5000, device="cuda"), qpos])
    unused = torch.randperm(L - T, generator=torch.Generator().manual_seed(L))[:(L - T) // 3].cuda()
    kpos[unused] = 1 << 40
    go = lambda k, v, **kw: fc.flash_attn_cached(q, k, v, causal=True, return_lse=True, **kw)
    clean = go(k, v, qpos=qpos, kpos=kpos)
    spoilt = go(_spoil(k, unused, 2), _spoil(v, unused, 2), qpos=qpos, kpos=kpos)
    assert all(torch.equal(a, b) for a, b in zip(clean, spoilt))
    if T > 1:
        y, lse = go(k, v)
        y1, lse1 = go(_spoil(k, slice(L - 1, L), 2), _spoil(v, slice(L - 1, L), 2))
        assert torch.equal(y[:, :-1], y1[:, :-1]) and torch.equal(lse[..., :-1], lse1[..., :-1])
        assert torch.isnan(y1[:, -1].float()).all()
    # what a row does see counts: an infinity in V alone
    v1 = v.clone()
    v1[:, :, L - T, 1], v1[:, :, 3, 2] = float("inf"), float("-inf")
    y, y1 = go(k, v)[0].float(), go(k, v1)[0].float()
    assert (y1[..., 1] == float("inf")).all() and (y1[..., 2] == float("-inf")).all()
    assert torch.equal(y[..., 3:], y1[..., 3:]) and torch.equal(y[..., 0], y1[..., 0])
