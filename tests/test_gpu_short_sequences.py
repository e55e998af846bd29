"""Units with one query tile (T up to 128, or an odd number of tiles) when every CTA works through several of them:
the warpgroup without a tile must not release the other one's buffers.  Forward and backward against plain
float32 attention on the GPU, and bit-equal on repetition."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,Hkv,D,dtype", [
    (60, 33, 12, 12, 64, torch.bfloat16), (40, 128, 12, 4, 64, torch.float16), (60, 300, 12, 12, 64, torch.bfloat16),
    (22, 60, 12, 12, 128, torch.float16), (40, 128, 12, 6, 128, torch.bfloat16), (60, 90, 12, 3, 32, torch.bfloat16)])
def test_many_units_with_one_tile(B, T, H, Hkv, D, dtype):
    from machinelearning_b200 import flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = (torch.randn(B, T, h, D, device="cuda", generator=g).to(dtype) for h in (H, Hkv, Hkv, H))
    qf, kf, vf = (t.float().requires_grad_() for t in (q, k, v))
    s = torch.einsum("bthd,bshd->bhts", qf, kf.repeat_interleave(H // Hkv, 2)) * D ** -0.5
    s = s.masked_fill(~torch.ones(T, T, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.einsum("bhts,bshd->bthd", s.softmax(-1), vf.repeat_interleave(H // Hkv, 2))
    want = (want.detach(), *torch.autograd.grad(want, (qf, kf, vf), do.float()))
    runs = []
    for _ in range(3):
        o, lse = fc.fwd(q, k, v, D ** -0.5, True)
        runs.append((o, *fc.bwd(do, q, k, v, o, lse, D ** -0.5, True)))
    for a, b, c, w in zip(*runs, want):
        assert torch.equal(a, b) and torch.equal(a, c)
        assert (a.float() - w).abs().max().item() <= 2e-2 * w.abs().max().item()
