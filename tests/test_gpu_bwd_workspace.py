"""Backward at head dim 128 with room for dS behind the tape: the dK/dV pass leaves dS in the
scratch and dQ is one product over it.  Held to the float64 oracle and, bit for bit, to the layout that
recomputes dS (tape-only scratch), at lengths around the 64- and 128-row tile edges, under every mask, with the
scratch poisoned and with room for one (batch, KV head) pair at a time."""
import math

import numpy as np
import pytest
import torch

from oracle import attention_f64 as orc

pytestmark = pytest.mark.gpu

#        B, T, H, Hkv, window, sinks, block, dtype
CASES = [(1, 1, 1, 1, 0, 0, 0, torch.bfloat16), (2, 65, 2, 1, 0, 0, 0, torch.float16),
         (1, 128, 2, 2, 0, 0, 0, torch.bfloat16), (1, 257, 4, 2, 0, 0, 0, torch.bfloat16),
         (1, 513, 2, 2, 64, 0, 0, torch.bfloat16), (1, 700, 2, 1, 200, 4, 0, torch.float16),
         (1, 640, 2, 2, 300, 130, 0, torch.bfloat16), (3, 333, 3, 1, 0, 0, 100, torch.bfloat16),
         (1, 385, 2, 2, 0, 0, 385, torch.float16)]


def _backward(lib, L, do, q, k, v, o, lse, scale, window, sinks, block, nbytes):
    B, T, H, D = q.shape
    code = L.DTYPE_BF16 if q.dtype == torch.bfloat16 else L.DTYPE_F16
    scratch = torch.full((nbytes,), 0xff, dtype=torch.uint8, device="cuda")           # NaN in every type
    dq, dk, dv = (torch.full_like(t, float("nan")) for t in (q, k, v))
    L.check("nlfa_bwd_masked", lib.nlfa_bwd_masked(
        *(t.data_ptr() for t in (do, q, k, v, o, lse, dq, dk, dv, scratch)), nbytes, B, T, H, k.shape[2], D, scale,
        window, sinks, block, code, L.PATH_TENSOR, L.PASS_ALL, torch.cuda.current_stream().cuda_stream))
    return dq, dk, dv


@pytest.mark.parametrize("B,T,H,Hkv,window,sinks,block,dtype", CASES)
def test_backward_with_room_for_ds(B, T, H, Hkv, window, sinks, block, dtype):
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    lib, D = fc._load(), 128
    g = torch.Generator().manual_seed(T + H)
    q, k, v, do = (torch.randn(B, T, h, D, generator=g).to(dtype).cuda() for h in (H, Hkv, Hkv, H))
    scale = 1.0 / math.sqrt(D)
    o, lse = fc.fwd(q, k, v, scale, True, window, sinks, block)
    code = L.DTYPE_BF16 if dtype == torch.bfloat16 else L.DTYPE_F16
    dims = (B, T, H, Hkv, D, window, sinks, block, code, L.PATH_TENSOR)
    tape = lib.nlfa_bwd_scratch_bytes(B, T, H)
    base, tiles, pairs = (tape + 255) // 256 * 256, (T + 127) // 128, B * Hkv
    whole = base + B * H * tiles * tiles * 32768                     # every tile pair: enough for any mask
    assert lib.nlfa_bwd_workspace_kernel_count(*dims, whole) == 3
    # the least that holds one pair: its launches go pair by pair
    count = lambda n: lib.nlfa_bwd_workspace_kernel_count(*dims, base + n * (H // Hkv) * 32768)
    one_pair = whole
    if pairs > 1:
        n = next(n for n in range(1, tiles * tiles + 1) if count(n) > 3)
        assert count(n) == 1 + 2 * pairs
        one_pair = base + n * (H // Hkv) * 32768
    args = (lib, L, do, q, k, v, o, lse, scale, window, sinks, block)
    recomputed, left, by_pair = (_backward(*args, n) for n in (tape, whole, one_pair))
    want = orc.attention_bwd(do, q, k, v, scale, window, sinks, block)
    for a, b, c, w in zip(recomputed, left, by_pair, want):
        assert torch.equal(a, b) and torch.equal(b, c)
        assert np.abs(b.double().cpu().numpy() - w).max() <= 2e-2 * max(np.abs(w).max(), 1e-2)


@pytest.mark.parametrize("B,T,H,Hkv,window", [(7, 1200, 16, 16, 0), (40, 1500, 6, 2, 0), (12, 1700, 16, 16, 700)])
def test_heads_in_groups_change_nothing(B, T, H, Hkv, window):
    """Streamed tiles beyond L2: the dK/dV pass takes its heads in (uneven) groups."""
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    lib, D = fc._load(), 128
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = (torch.randn(B, T, h, D, device="cuda", generator=g).bfloat16() for h in (H, Hkv, Hkv, H))
    scale = 1.0 / math.sqrt(D)
    o, lse = fc.fwd(q, k, v, scale, True, window, 0, 0)
    whole = lib.nlfa_bwd_workspace_bytes(B, T, H, Hkv, D, window, 0, 0, L.DTYPE_BF16, L.PATH_TENSOR)
    assert lib.nlfa_bwd_workspace_kernel_count(B, T, H, Hkv, D, window, 0, 0, L.DTYPE_BF16, L.PATH_TENSOR, whole) == 3
    args = (lib, L, do, q, k, v, o, lse, scale, window, 0, 0)
    for a, b in zip(_backward(*args, lib.nlfa_bwd_scratch_bytes(B, T, H)), _backward(*args, whole)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("extreme,same", [(dict(block=(1 << 31) - 1), dict(block=333)),
                                          (dict(window=(1 << 31) - 1, sinks=(1 << 31) - 2), dict())])
def test_extents_next_to_two_to_the_31(extreme, same):
    from machinelearning_b200 import flash_cuda as fc
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k, v, do = (torch.randn(40, 333, h, 128, device="cuda", generator=g).bfloat16() for h in (4, 2, 2, 4))
    runs = []
    for kw in (extreme, same):
        o, lse = fc.fwd(q, k, v, 0.1, True, **kw)
        runs.append((o, lse, *fc.bwd(do, q, k, v, o, lse, 0.1, True, **kw)))
    assert all(torch.equal(a, b) for a, b in zip(*runs))


def test_backward_without_memory_for_the_workspace():
    """When the allocator has no room for dS the backward goes on with the tape, to the same bits."""
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    B, T, H, D = 4, 4096, 16, 128
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k, v = (torch.randn(B, T, H, D, device="cuda", generator=g).bfloat16().requires_grad_() for _ in range(3))
    do = torch.randn(B, T, H, D, device="cuda", generator=g).bfloat16()
    y = fc.flash_attn(q, k, v)
    want = torch.autograd.grad(y, (q, k, v), do, retain_graph=True)
    size = fc._load().nlfa_bwd_workspace_bytes(B, T, H, H, D, 0, 0, 0, L.DTYPE_BF16, L.PATH_TENSOR)
    assert size > 1 << 30
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:                                             # what is in use, the three gradients, and half of the workspace
        room = torch.cuda.memory_reserved() + 3 * do.nbytes + size // 2
        torch.cuda.set_per_process_memory_fraction(room / total)
        got = torch.autograd.grad(y, (q, k, v), do)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
