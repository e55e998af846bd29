"""The register-tiled fp32-arithmetic kernels (``use_mma=False``) against the float64 oracle at lengths around their
16-, 32- and 64-row tiles, each of those heights (chosen by the number of row tiles per SM), every head dim and mask."""
import math

import numpy as np
import pytest
import torch

from oracle import attention_f64 as orc

pytestmark = pytest.mark.gpu

#        B, T, H, Hkv, D, window, sinks, block, dtype
CASES = [(1, 1, 1, 1, 64, 0, 0, 0, torch.float32), (1, 31, 2, 1, 128, 0, 0, 0, torch.float32),
         (2, 33, 2, 2, 32, 0, 0, 0, torch.float32), (1, 65, 4, 2, 64, 0, 0, 0, torch.float32),
         (1, 129, 2, 1, 128, 40, 0, 0, torch.float32), (1, 200, 2, 2, 64, 70, 65, 0, torch.float32),
         (1, 190, 4, 1, 32, 0, 0, 100, torch.float32), (1, 130, 2, 2, 64, 0, 0, 130, torch.bfloat16),
         (3, 200, 16, 16, 64, 0, 0, 0, torch.float32), (6, 200, 16, 8, 128, 0, 0, 90, torch.float32),
         (13, 130, 12, 4, 64, 50, 3, 0, torch.float32), (13, 97, 16, 16, 32, 0, 0, 0, torch.float16)]


@pytest.mark.parametrize("B,T,H,Hkv,D,window,sinks,block,dtype", CASES)
def test_fp32_tiles_match_the_oracle(B, T, H, Hkv, D, window, sinks, block, dtype):
    from machinelearning_b200 import flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    g = torch.Generator().manual_seed(T + D)
    q, k, v, do = (torch.randn(B, T, h, D, generator=g).to(dtype).cuda() for h in (H, Hkv, Hkv, H))
    scale = 1.0 / math.sqrt(D)
    o, lse = fc.fwd(q, k, v, scale, False, window, sinks, block)
    got = (o, lse, *fc.bwd(do, q, k, v, o, lse, scale, False, window, sinks, block=block))
    want = (*orc.attention_fwd(q, k, v, scale, window, sinks, block),
            *orc.attention_bwd(do, q, k, v, scale, window, sinks, block))
    for name, a, w in zip(("o", "lse", "dq", "dk", "dv"), got, want):
        tol = 2e-5 if dtype == torch.float32 else 1e-5 if name == "lse" else 2e-2
        assert np.abs(a.double().cpu().numpy() - w).max() <= tol * max(1.0, np.abs(w).max()), name


def _relative(a, want):
    return ((a.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("B,T,H,Hkv,D", [(2, 700, 6, 2, 128), (40, 100, 16, 16, 64), (16, 600, 8, 8, 128)])
def test_fp32_sums_are_short(B, T, H, Hkv, D):
    """Rounding errors of a sum of n terms in one chain have a spread of sqrt(n / 2) half units in the last place, of runs of
    8 whose totals are added sqrt(4 + n / 16).  Runs leave 1.4e-7 relative (2-norm) of O here, chains of D and of T 2.0e-7 to
    3.6e-7."""
    from machinelearning_b200 import flash_cuda as fc
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = (torch.randn(B, T, h, D, device="cuda", generator=g) for h in (H, Hkv, Hkv))
    o, _ = fc.fwd(q, k, v, D ** -0.5, False)
    s = torch.einsum("bthd,bshd->bhts", q.double(), k.double().repeat_interleave(H // Hkv, 2)) * D ** -0.5
    s = s.masked_fill(~torch.ones(T, T, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.einsum("bhts,bshd->bthd", s.softmax(-1), v.double().repeat_interleave(H // Hkv, 2))
    assert _relative(o, want) <= 1.7e-7


@pytest.mark.parametrize("T,H,Hkv,L,D", [(1, 12, 12, 1057, 64), (64, 4, 4, 16448, 128), (15, 4, 4, 700, 64), (4, 4, 4, 4097, 128)])
def test_fp32_cached_sums_are_short(T, H, Hkv, L, D):
    """The same over a cache: 1.6e-7 to 2.2e-7, with one chain of D and one of a CTA's keys 3.1e-7 to 9.3e-7."""
    from machinelearning_b200 import flash_cuda as fc
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = (torch.randn(1, *s, D, device="cuda", generator=g) for s in ((T, H), (Hkv, L), (Hkv, L)))
    o = fc.flash_attn_cached(q, k, v, causal=True)
    s = torch.einsum("bthd,bhsd->bhts", q.double(), k.double()) * D ** -0.5
    i = torch.arange(L - T, L, device="cuda")[:, None]
    s = s.masked_fill(torch.arange(L, device="cuda")[None] > i, float("-inf"))
    assert _relative(o, torch.einsum("bhts,bhsd->bthd", s.softmax(-1), v.double())) <= 2.6e-7
