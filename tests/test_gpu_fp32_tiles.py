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
