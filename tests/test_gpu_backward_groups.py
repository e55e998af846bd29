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


def _shares(T, window, sinks, pairs):
    """The dK/dV pass's longest unit (a key block's query tiles, for each head of the group) over what falls to one SM, counted
    from the visible pairs themselves."""
    n = -(-T // 128)
    units = []
    for j in range(n):
        k0, k1 = 128 * j, min(T, 128 * j + 128) - 1
        last = lambda k: T - 1 if k < sinks else min(T - 1, k + window - sinks - 1)          # last query that sees key k
        reach = max(last(k0), last(k1), last(min(k1, sinks - 1)) if k0 < sinks else 0)
        units.append(reach // 128 - j + 1)
    return max(units) * torch.cuda.get_device_properties(0).multi_processor_count / (pairs * sum(units))


# several sink blocks, windows as long as the row, pairs for either side of the lines
SINKS = [(16384, 500, 16), (6000, 150, 16), (4096, 2000, 1000), (4096, 4000, 600), (2048, 2000, 130), (3000, 1000, 300), (8192, 300, 100)]


@pytest.mark.parametrize("T,window,sinks", SINKS)
def test_long_sink_blocks_keep_the_delta_kernel(T, window, sinks):
    """dQ runs beside the dK/dV pass, and so behind a Delta kernel, where a key block with sinks is longer than an SM's share."""
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    kernels = {}
    for B in range(1, 40):
        if B * 64 * -(-T // 128) < 16 * torch.cuda.get_device_properties(0).multi_processor_count:
            continue
        shares = _shares(T, window, sinks, 4 * B)
        kernels[shares <= 1] = fc._load().nlfa_bwd_workspace_kernel_count(B, T, 64, 4, 64, window, sinks, 0, L.DTYPE_BF16, L.PATH_TENSOR, 0)
        assert kernels[shares <= 1] == (2 if shares <= 1 else 3), (B, shares)
    assert kernels[True] == 2


@pytest.mark.parametrize("T,window,sinks", SINKS)
def test_long_sink_blocks_get_no_ds_scratch(T, window, sinks):
    """At head dim 128 there is room for dS unless a key block with sinks is more than 1.4 of an SM's share of one launch."""
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    lib, sms = fc._load(), torch.cuda.get_device_properties(0).multi_processor_count
    seen = set()
    for H, Hkv in ((4, 4), (64, 4)):
        for B in range(1, 30):
            tape = (lib.nlfa_bwd_scratch_bytes(B, T, H) + 255) // 256 * 256
            size = lib.nlfa_bwd_workspace_bytes(B, T, H, Hkv, 128, window, sinks, 0, L.DTYPE_BF16, L.PATH_TENSOR)
            tiles = -(-T // 128)
            widest = max(min(t, -(-sinks // 128)) + t - max(min(t, -(-sinks // 128)), max(0, 128 * t - (window - sinks) + 1) // 128) + 1
                         for t in range(tiles))                                    # key blocks of a query tile
            most = (4 << 30) // (widest * tiles * 32768 * (H // Hkv))             # pairs of one launch
            if most == 0:
                assert size <= tape
                continue
            parts = -(-B * Hkv // most)
            per = -(-B * Hkv // parts)
            full = 2 * per * tiles >= 3 * sms and (parts == 1 or per * tiles >= 3 * sms)
            wanted = full and _shares(T, window, sinks, per) <= 1.4
            assert (size > tape) == wanted, (B, H, parts, _shares(T, window, sinks, per))
            seen.add((full, wanted))
    assert (True, True) in seen


def test_either_amount_of_scratch_gives_the_same_bits_under_sinks():
    from machinelearning_b200 import _lib as L, flash_cuda as fc
    lib = fc._load()
    T, window, sinks = 9000, 260, 5
    tape = lambda B: (lib.nlfa_bwd_scratch_bytes(B, T, 2) + 255) // 256 * 256
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
