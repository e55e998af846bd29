"""The cached forward where its row combination can go wrong, against the float64 oracle: rows that do not divide
by the CTAs a tile's keys are split over (or are fewer than those), one to four warps of rows, a second softmax
warpgroup without a key block, CTAs that see no key; and the same split in fp32."""
import numpy as np
import pytest
import torch

from oracle import cached_f64


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32], ids=["fp16", "fp32"])
@pytest.mark.parametrize("T,H,Hkv,L,D,causal,window", [
    (1, 1, 1, 130, 64, True, 0),            # one row; the first CTA's second warpgroup has no block
    (1, 8, 2, 5000, 128, True, 0),          # four rows, more CTAs than rows
    (20, 3, 3, 250, 128, False, 0),         # two blocks, one CTA: finished without a split
    (40, 2, 2, 200, 128, True, 0),          # the same with two warps of rows
    (100, 2, 2, 129, 64, True, 0),          # .. with four
    (33, 2, 2, 700, 32, False, 0),          # two warps of rows
    (37, 4, 2, 2300, 64, True, 0),          # three
    (128, 1, 1, 4100, 128, True, 0),        # four
    (50, 6, 2, 1000, 128, True, 0),         # tiles of a ragged number of rows
    (30, 12, 12, 1050, 64, True, 0),        # fp32: two rows a thread, fewer CTAs than two per SM
    (9, 4, 4, 3000, 64, True, 100),         # a window: most of the keys are not visited
])
def test_rows_of_a_split_cache_match_the_oracle(T, H, Hkv, L, D, causal, window, dtype):
    from machinelearning_b200 import flash_cuda
    assert flash_cuda.is_available(), flash_cuda.unavailable_reason()
    g = torch.Generator().manual_seed(T + L)
    q = torch.randn(1, T, H, D, generator=g).to("cuda", dtype)
    k = torch.randn(1, Hkv, L, D, generator=g).to("cuda", dtype)
    v = torch.randn(1, Hkv, L, D, generator=g).to("cuda", dtype)
    y, lse = flash_cuda.flash_attn_cached(q, k, v, causal=causal, window=window, return_lse=True)
    n = lambda x: x.double().cpu().numpy()
    ref, lse_ref = cached_f64.forward(n(q), n(k), n(v), 1.0 / np.sqrt(D), np.arange(L - T, L), np.arange(L), causal,
                                      window, 0)
    tol = 1e-5 if dtype == torch.float32 else 5e-3 * np.abs(ref).max()
    assert np.abs(n(y) - ref).max() <= tol
    assert np.abs(n(lse) - lse_ref).max() <= (1e-5 if dtype == torch.float32 else 1e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("T,H,Hkv,L,D", [
    # the rows a CTA finishes, eight columns a thread: at most two CTAs share four key blocks, so more than 256 pieces of four
    (64, 16, 16, 500, 128),                 # .. two copies of the rows
    (30, 16, 16, 500, 128),                 # .. four
    (101, 3, 3, 300, 128),                  # .. one, rows that do not divide by the CTAs
    (77, 4, 4, 500, 64),
    (64, 16, 16, 2048, 128),                # split over eight CTAs: just 256 pieces of four
    (128, 3, 3, 1500, 64),                  # one copy, up to six CTAs, which the rows do not divide by
    (32, 12, 12, 1056, 64),                 # four columns a thread: at most 256 pieces of four however it is split
    (70, 2, 2, 1300, 32),                   # head dim 32: the second warpgroup's half of the columns is none
    (9, 160, 160, 400, 32),                 # .. whole tiles, finished where their sums are
    (100, 150, 150, 300, 128),              # whole tiles, one copy: 64 columns a thread
    (5, 150, 150, 90, 128),                 # whole tiles of one key block
])
def test_pieces_of_finished_rows_match_the_oracle(T, H, Hkv, L, D):
    from machinelearning_b200 import flash_cuda
    g = torch.Generator().manual_seed(T * L)
    q, k, v = (torch.randn(1, *s, D, generator=g).to("cuda", torch.bfloat16) for s in ((T, H), (Hkv, L), (Hkv, L)))
    y, lse = flash_cuda.flash_attn_cached(q, k, v, causal=True, return_lse=True)
    n = lambda x: x.double().cpu().numpy()
    ref, lse_ref = cached_f64.forward(n(q), n(k), n(v), 1.0 / np.sqrt(D), np.arange(L - T, L), np.arange(L), True, 0, 0)
    # P and the result rounded to 8 bits of mantissa, errors of a row's keys independent: 2^-9 of the largest value each
    assert np.abs(n(y) - ref).max() <= 8e-3 * np.abs(ref).max()
    assert np.abs(n(lse) - lse_ref).max() <= 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32], ids=["fp16", "fp32"])
def test_sinks_next_to_two_to_the_31(dtype):
    from machinelearning_b200 import flash_cuda
    g = torch.Generator().manual_seed(0)
    q, k, v = (torch.randn(1, *s, 64, generator=g).to("cuda", dtype) for s in ((40, 4), (2, 900), (2, 900)))
    want = flash_cuda.flash_attn_cached(q, k, v, causal=True)
    for window, sinks in (((1 << 31) - 1, (1 << 31) - 2), ((1 << 31) - 1, 0), (901, 900)):
        assert torch.equal(flash_cuda.flash_attn_cached(q, k, v, causal=True, window=window, sinks=sinks), want)


def _sparse(T, L, dtype=torch.float32):
    """A window of 256 with 4 sinks over a cache that was not compacted, its keys in an order of their own."""
    g = torch.Generator().manual_seed(L)
    q, k, v = (torch.randn(1, *s, 64, generator=g).to("cuda", dtype) for s in ((T, 4), (2, L), (2, L)))
    kpos = torch.arange(L).reshape(-1, 8).flip(1).reshape(-1) if L % 8 == 0 else torch.arange(L)
    return q, k, v, torch.arange(L - T, L), kpos


@pytest.mark.gpu
@pytest.mark.parametrize("T,L", [(1, 16384), (5, 9000), (40, 20001), (17, 130), (3, 70000)])
def test_hidden_stretches_of_a_cache_with_positions(T, L):
    from machinelearning_b200 import flash_cuda
    q, k, v, qpos, kpos = _sparse(T, L)
    y, lse = flash_cuda.flash_attn_cached(q, k, v, qpos=qpos, kpos=kpos, causal=True, window=256, sinks=4, return_lse=True)
    n = lambda x: x.double().cpu().numpy()
    ref, lse_ref = cached_f64.forward(n(q), n(k), n(v), 0.125, qpos.numpy(), kpos.numpy(), True, 256, 4)
    assert np.abs(n(y) - ref).max() <= 1e-5 and np.abs(n(lse) - lse_ref).max() <= 1e-5


@pytest.mark.gpu
def test_hidden_stretches_of_a_cache_are_not_read():
    """Of 262,144 keys a window shows 256: a fraction of the time of a causal call, which reads them all."""
    from machinelearning_b200 import flash_cuda
    q, k, v, qpos, kpos = _sparse(1, 262144)
    qpos, kpos = qpos.cuda(), kpos.cuda()

    def microseconds(**kw):
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                flash_cuda.flash_attn_cached(q, k, v, qpos=qpos, kpos=kpos, causal=True, **kw)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return sorted(times)[6]

    assert microseconds(window=256, sinks=4) < 0.5 * microseconds()


@pytest.mark.gpu
@pytest.mark.parametrize("T", [4, 40])
def test_positions_of_an_unmasked_block_may_be_anything(T):
    from machinelearning_b200 import flash_cuda
    g = torch.Generator().manual_seed(T)
    q, k, v = (torch.randn(1, *s, 64, generator=g).to("cuda", torch.bfloat16) for s in ((T, 4), (2, 300), (2, 300)))
    kpos = torch.full((300,), 2147483647, dtype=torch.int32, device="cuda")
    kpos[::3] = -5
    y = flash_cuda.flash_attn_cached(q, k, v, qpos=torch.zeros(T, dtype=torch.int32, device="cuda"), kpos=kpos)
    assert torch.equal(y, flash_cuda.flash_attn_cached(q, k, v))
