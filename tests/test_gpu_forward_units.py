"""Both unit heights of the tensor-core forward -- one query tile, and two (long rows and more tiles than SMs, or K and V beyond
L2, at head dims up to 64; more than two tiles per SM at 128) -- and both widths of its key blocks, against plain float32
attention on the GPU, at odd and even numbers of tiles, under every mask, and the logsumexp with them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#        B, T, H, Hkv, D, window, sinks, block, dtype
CASES = [(1, 4200, 5, 1, 64, 0, 0, 0, torch.bfloat16), (1, 4353, 6, 2, 32, 0, 0, 0, torch.float16),   # two tiles
         (1, 4300, 5, 5, 64, 4150, 70, 0, torch.bfloat16), (1, 4480, 5, 5, 64, 0, 0, 700, torch.bfloat16),
         (16, 2100, 8, 8, 64, 0, 0, 0, torch.float16),                             # .. for K and V beyond L2
         (25, 300, 4, 2, 128, 0, 0, 0, torch.bfloat16), (25, 385, 4, 4, 128, 150, 9, 0, torch.float16),
         (25, 290, 4, 1, 128, 0, 0, 100, torch.bfloat16),
         (1, 4096, 3, 1, 64, 0, 0, 0, torch.bfloat16), (1, 4200, 4, 2, 64, 0, 0, 0, torch.bfloat16),  # one tile
         (1, 1100, 4, 2, 32, 200, 5, 0, torch.bfloat16), (3, 700, 6, 2, 128, 0, 0, 96, torch.float16)]


# one tile of each kind of mask next to the line between the widths of key blocks, and masks with many tiles
CASES += [(8, 1500, 9, 3, 64, 300, 4, 0, torch.bfloat16), (8, 1473, 9, 9, 32, 333, 70, 0, torch.float16),
          (12, 1100, 12, 4, 64, 200, 0, 0, torch.bfloat16), (12, 1025, 12, 12, 64, 256, 0, 0, torch.float16),
          (12, 1000, 12, 4, 32, 0, 0, 0, torch.bfloat16), (12, 1088, 12, 12, 32, 0, 0, 100, torch.float16),
          (30, 450, 12, 6, 32, 0, 0, 0, torch.bfloat16), (60, 63, 20, 4, 32, 0, 0, 16, torch.bfloat16),
          (1, 191, 2, 2, 32, 65, 1, 0, torch.bfloat16), (2, 256, 3, 3, 64, 30, 0, 0, torch.float16),
          (2, 1000, 3, 3, 64, 66, 0, 0, torch.bfloat16), (2, 1000, 3, 1, 32, 120, 65, 0, torch.bfloat16)]

# key blocks of 64: the edges of a window at, before and behind a block's, sinks of part of a block and of a whole one, ragged rows;
# the shortest row that gets them, its last tile one row high; T = 63 .. 65 into a block, few tiles and many
NARROW = [(1, 3000, 2, 1, 64, 64, 4, 0, torch.bfloat16), (1, 1089, 4, 2, 32, 50, 0, 0, torch.float16),
          (1, 2111, 3, 3, 64, 128, 64, 0, torch.float16), (2, 257, 2, 2, 32, 66, 1, 0, torch.bfloat16),
          (8, 1500, 9, 3, 64, 69, 4, 0, torch.bfloat16), (8, 1473, 9, 9, 32, 2, 0, 0, torch.float16),
          (12, 1024, 12, 4, 64, 65, 0, 0, torch.bfloat16), (12, 1025, 12, 12, 64, 33, 20, 0, torch.float16),
          (1, 4096, 3, 1, 64, 64, 0, 0, torch.float16), (30, 448, 12, 6, 32, 129, 64, 0, torch.bfloat16)]


@pytest.mark.parametrize("B,T,H,Hkv,D,window,sinks,block,dtype,width", [(*c, 128) for c in CASES] + [(*c, 64) for c in NARROW])
def test_forward_in_both_unit_heights(B, T, H, Hkv, D, window, sinks, block, dtype, width):
    from machinelearning_b200 import flash_cuda as fc
    assert fc.is_available(), fc.unavailable_reason()
    from machinelearning_b200 import _lib
    assert fc._load().nlfa_fwd_key_block(T, D, window, sinks, block, _lib.DTYPE_BF16, _lib.PATH_TENSOR) == width
    g = torch.Generator(device="cuda").manual_seed(T + D)
    q, k, v = (torch.randn(B, T, h, D, device="cuda", generator=g).to(dtype) for h in (H, Hkv, Hkv))
    scale = D ** -0.5
    o, lse = fc.fwd(q, k, v, scale, True, window, sinks, block)
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
    keep = (j // block <= i // block) if block else (j <= i)
    if window:
        keep = keep & ((j > i - (window - sinks)) | (j < sinks))
    for b in range(0, B, 6):
        s = torch.einsum("thd,shd->hts", q[b].float(), k[b].float().repeat_interleave(H // Hkv, 1)) * scale
        s = s.masked_fill(~keep, float("-inf"))
        want = torch.einsum("hts,shd->thd", s.softmax(-1), v[b].float().repeat_interleave(H // Hkv, 1))
        assert (o[b].float() - want).abs().max().item() <= 2e-2 * want.abs().max().item()
        assert (lse[b] - s.logsumexp(-1)).abs().max().item() <= 1e-3


@pytest.mark.parametrize("D,window,sinks", [(64, 64, 0), (32, 64, 4), (64, 128, 0), (64, 256, 0), (32, 400, 4), (64, 66, 0)])
def test_the_end_of_a_row_changes_nothing_before_it(D, window, sinks):
    """Causal rows see nothing behind them: the first rows of a longer call have the bits of the shorter one, also where the last
    tile is cut."""
    from machinelearning_b200 import flash_cuda as fc
    q, k, v = (torch.randn(1, 1152, 6, D, device="cuda", generator=torch.Generator(device="cuda").manual_seed(D)).half() for _ in range(3))
    o, lse = fc.fwd(q, k, v, D ** -0.5, True, window, sinks)
    for T in (1024, 1025, 1060, 1088, 1090):
        o1, lse1 = fc.fwd(*(t[:, :T].contiguous() for t in (q, k, v)), D ** -0.5, True, window, sinks)
        assert torch.equal(o1, o[:, :T]) and torch.equal(lse1, lse[:, :, :T])


@pytest.mark.parametrize("D,window,sinks", [(64, 2, 0), (64, 16, 0), (32, 65, 0), (64, 69, 4), (32, 129, 64), (64, 96, 0), (64, 200, 0),
                                            (32, 160, 0)])
def test_windows_lose_no_precision_to_the_width_of_key_blocks(D, window, sinks):
    """Error to 64 bits against that of a float64 walk in blocks of 128 that rounds only P and o: the two share their roundings but
    for the last bits of the scores, so a quarter of a percent is far above their difference and far below what a row's
    reference taken from fewer keys costs (0.5 to 0.9%)."""
    from machinelearning_b200 import flash_cuda as fc
    T, H, dtype, scale = 4096, 40, torch.bfloat16, D ** -0.5
    g = torch.Generator(device="cuda").manual_seed(window)
    q, k, v = (torch.randn(1, T, H, D, device="cuda", generator=g).to(dtype) for _ in range(3))
    o, _ = fc.fwd(q, k, v, scale, True, window, sinks)
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
    keep = (j <= i) & ((j > i - (window - sinks)) | (j < sinks))
    got = walk = 0.0
    for h in range(H):
        s = (q[0, :, h].double() @ k[0, :, h].double().T * scale).masked_fill(~keep, float("-inf"))
        exact = s.softmax(-1) @ v[0, :, h].double()
        # the reference of a row is the maximum of the first block its tile visits, the first visible one's if that hides from it
        # (a later block would have to exceed it by a factor of 256)
        by_block = s.view(T, T // 128, 128).amax(-1)
        first = (by_block > float("-inf")).int().argmax(-1)
        p = (s - by_block.gather(1, first[:, None])).exp()
        mean = (p.to(dtype).double() @ v[0, :, h].double()) / p.sum(-1, keepdim=True)
        got += (o[0, :, h].double() - exact).square().sum()
        walk += (mean.to(dtype).double() - exact).square().sum()
    assert got.sqrt().item() <= 1.0025 * walk.sqrt().item(), (got.sqrt() / walk.sqrt()).item()
