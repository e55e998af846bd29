"""The dK/dV pass hands its units out in groups of (batch, KV head) pairs, one pair per SM, or in groups of equal size where the
last would have less than half as many: gradients against plain float32 autograd at both edges of that rule, and which
of its layouts a window with sinks gets."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (32, torch.float16), (128, torch.bfloat16)])
@pytest.mark.parametrize("extra,groups", [(0, 1), (1, 1), (0.5, 1), (0.49, 1), (1, 2), (-1, 1)])
def test_gradients_for_any_number_of_pairs(D, dtype, extra, groups):
    from machinelearning_b200 import flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B, T, H, window, sinks = groups * sms + (int(extra * sms) if isinstance(extra, float) else extra), 300, 2, 140, 3
    g = torch.Generator(device="cuda").manual_seed(B + D)
    q, k, v, do = (torch.randn(B, T, h, D, device="cuda", generator=g).to(dtype) for h in (H, 1, 1, H))
    scale = D ** -0.5
    o, lse = fc.fwd(q, k, v, scale, True, window, sinks)
    got = fc.bwd(do, q, k, v, o, lse, scale, True, window, sinks)
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
    keep = (j <= i) & ((j > i - (window - sinks)) | (j < sinks))
    qf, kf, vf = (t.float().requires_grad_() for t in (q, k, v))
    s = torch.einsum("bthd,bsd->bhts", qf, kf[:, :, 0]) * scale
    p = s.masked_fill(~keep, float("-inf")).softmax(-1)
    torch.einsum("bhts,bsd->bthd", p, vf[:, :, 0]).backward(do.float())
    # o, P, dS and the results are rounded to 16 bits: four errors of at most 2^-8 of the largest terms
    for a, want in zip(got, (qf.grad, kf.grad, vf.grad)):
        assert (a.float() - want).abs().max().item() <= 4 * 2.0 ** -8 * want.abs().max().item()


def test_long_sink_blocks_keep_the_delta_kernel():
    """One sink block's unit is group * T / 128 iterations; dQ runs beside it unless it is at most 0.8 of a CTA's share."""
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    count = lambda B, T: fc._load().nlfa_bwd_workspace_kernel_count(B, T, 12, 4, 64, 500, 16, 0, L.DTYPE_BF16, L.PATH_TENSOR, 0)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    enough = -(-5 * 256 * sms // (4 * 4 * (2 * 500 + 640)))           # pairs * (2 w + 640) * 4 >= 5 * 256 * SMs, four pairs each
    assert count(enough, 16384) == 2
    assert count(enough - 1, 16384) == 3


def test_long_sink_blocks_leave_no_ds():
    """At head dim 128 dS is left behind for the dQ pass unless one sink block is more than 1.5 of a CTA's share of the dK/dV
    pass; with either amount of scratch the gradients have the same bits."""
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    lib = fc._load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    T, window, sinks = 9000, 260, 5
    enough = -(-2 * 256 * sms // (3 * (2 * window + 896)))                   # 3 * pairs * (2 w + 896) >= 2 * 256 * SMs
    tape = lambda B: (lib.nlfa_bwd_scratch_bytes(B, T, 2) + 255) // 256 * 256
    size = lambda B: lib.nlfa_bwd_workspace_bytes(B, T, 2, 1, 128, window, sinks, 0, L.DTYPE_BF16, L.PATH_TENSOR)
    assert size(enough) > tape(enough) and size(enough - 1) <= tape(enough - 1)
    B = 3
    g = torch.Generator(device="cuda").manual_seed(2)
    q, k, v, do = (torch.randn(B, T, h, 128, device="cuda", generator=g).bfloat16() for h in (2, 1, 1, 2))
    scale = 128 ** -0.5
    o, lse = fc.fwd(q, k, v, scale, True, window, sinks)
    got = fc.bwd(do, q, k, v, o, lse, scale, True, window, sinks)
    want = [torch.empty_like(t) for t in (q, k, v)]
    scratch = torch.empty(tape(B) + (256 << 20), dtype=torch.uint8, device="cuda")      # 3 pairs x 2 heads x ~280 tiles of 32 KB
    ptr = lambda t: t.data_ptr()
    assert lib.nlfa_bwd_workspace_kernel_count(B, T, 2, 1, 128, window, sinks, 0, L.DTYPE_BF16, L.PATH_TENSOR, scratch.numel()) == 3
    assert lib.nlfa_bwd_masked(*map(ptr, (do, q, k, v, o, lse, *want, scratch)), scratch.numel(), B, T, 2, 1, 128, scale, window, sinks, 0,
                               L.DTYPE_BF16, L.PATH_TENSOR, L.PASS_ALL, torch.cuda.current_stream().cuda_stream) == 0
    assert all(torch.equal(a, b) for a, b in zip(got, want))
