"""Scheduler counters under concurrency: a captured graph replaying on one stream while eager
launches run on another (needs a B200).

The persistent kernels take their work units from a pair of device counters.  A launch made under
stream capture keeps the counters it was given for as long as its graph is replayed, so those come
from a range that is never handed to another launch; eager launches take turns on a ring of their
own.  Two kernels that shared a pair would skip units and leave rows unwritten, silently -- the
check is bit-equality with results computed alone.
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_graph_replay_and_eager_launches_do_not_share_work_counters():
    from machinelearning_b200 import flash_cuda as fc
    assert fc.mma_available(), fc.mma_unavailable_reason()
    torch.manual_seed(11)
    D = 64
    scale = 1.0 / math.sqrt(D)
    mk = lambda b, t, h: torch.randn(b, t, h, D, device="cuda").bfloat16()
    qa, ka, va, da = mk(2, 512, 4), mk(2, 512, 2), mk(2, 512, 2), mk(2, 512, 4)     # the graph's problem
    qb, kb, vb, db = mk(3, 384, 2), mk(3, 384, 2), mk(3, 384, 2), mk(3, 384, 2)     # the eager one

    def run(q, k, v, d):
        o, lse = fc.fwd(q, k, v, scale, True)
        return (o, lse, *fc.bwd(d, q, k, v, o, lse, scale, True))

    want_a = [t.clone() for t in run(qa, ka, va, da)]
    want_b = [t.clone() for t in run(qb, kb, vb, db)]
    torch.cuda.synchronize()

    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        run(qa, ka, va, da)                      # warm-up on the capture stream
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            got_a = run(qa, ka, va, da)
    torch.cuda.synchronize()

    bad = 0
    for i in range(1000):
        with torch.cuda.stream(side):
            graph.replay()
        got_b = run(qb, kb, vb, db)              # eager, on the default stream, overlapping the replay
        if i % 50 == 49:
            torch.cuda.synchronize()
            bad += sum(not torch.equal(g, w) for g, w in zip(got_a, want_a))
            bad += sum(not torch.equal(g, w) for g, w in zip(got_b, want_b))
    torch.cuda.synchronize()
    assert bad == 0


def test_overlapped_launches_give_the_bits_of_serialised_ones():
    """The tensor-core kernels are launched with programmatic stream serialization (a kernel's set-up
    runs beside its predecessor's last CTAs, the dQ pass fills the SMs the dK/dV pass leaves);
    ``NLFA_PDL=0`` launches them the plain way.  The two must agree bit for bit, back to back, with a
    window and without."""
    import os
    import subprocess
    import sys
    import pathlib
    root = pathlib.Path(__file__).resolve().parent.parent
    script = f"""
import sys, math, hashlib
sys.path.insert(0, {str(root)!r})
import torch
from machinelearning_b200 import flash_cuda as fc
assert fc.mma_available(), fc.mma_unavailable_reason()
h = hashlib.sha256()
for (B, T, H, Hkv, D, w, s) in ((3, 700, 4, 2, 64, 0, 0), (2, 1024, 4, 4, 128, 0, 0), (2, 900, 4, 2, 64, 128, 4)):
    g = torch.Generator(device="cuda").manual_seed(5)
    mk = lambda heads: torch.randn(B, T, heads, D, device="cuda", generator=g).bfloat16()
    q, k, v, d = mk(H), mk(Hkv), mk(Hkv), mk(H)
    for _ in range(20):                        # back to back: every launch has a predecessor still running
        o, lse = fc.fwd(q, k, v, 1 / math.sqrt(D), True, w, s)
        grads = fc.bwd(d, q, k, v, o, lse, 1 / math.sqrt(D), True, w, s)
    torch.cuda.synchronize()
    for t in (o, lse, *grads):
        h.update(t.cpu().contiguous().view(torch.uint8).numpy().tobytes())
print("digest", h.hexdigest())
"""
    digests = []
    for flag in ("1", "0"):
        env = dict(os.environ, NLFA_PDL=flag)
        r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300, env=env)
        assert r.returncode == 0, r.stderr[-2000:]
        digests.append(r.stdout.strip().splitlines()[-1])
    assert digests[0] == digests[1]


def test_delta_formed_in_the_dq_pass_gives_the_bits_of_the_delta_kernel():
    """Large problems at head dim 64 skip the Delta kernel: the dQ pass forms the row sums of dO * O
    itself (same additions in the same order) and runs before the dK/dV pass.  ``NLFA_DELTA_IN_DQ``
    forces either layout; every gradient must agree bit for bit, causal, windowed and block-causal,
    with query rows past the end of the last tile."""
    import os
    import subprocess
    import sys
    import pathlib
    root = pathlib.Path(__file__).resolve().parent.parent
    script = f"""
import sys, math, hashlib
sys.path.insert(0, {str(root)!r})
import torch
from machinelearning_b200 import flash_cuda as fc
assert fc.mma_available(), fc.mma_unavailable_reason()
h = hashlib.sha256()
for (B, T, H, Hkv, w, s, blk) in ((3, 700, 4, 2, 0, 0, 0), (2, 1000, 6, 6, 128, 4, 0), (2, 517, 4, 1, 0, 0, 96), (40, 1024, 12, 12, 0, 0, 0)):
    g = torch.Generator(device="cuda").manual_seed(6)
    mk = lambda heads: torch.randn(B, T, heads, 64, device="cuda", generator=g).bfloat16()
    q, k, v, d = mk(H), mk(Hkv), mk(Hkv), mk(H)
    for _ in range(3):
        o, lse = fc.fwd(q, k, v, 0.125, True, w, s, blk)
        grads = fc.bwd(d, q, k, v, o, lse, 0.125, True, w, s, block=blk)
    torch.cuda.synchronize()
    for t in grads:
        h.update(t.cpu().contiguous().view(torch.uint8).numpy().tobytes())
print("digest", h.hexdigest())
"""
    digests = []
    for flag in ("1", "0"):
        env = dict(os.environ, NLFA_DELTA_IN_DQ=flag)
        r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300, env=env)
        assert r.returncode == 0, r.stderr[-2000:]
        digests.append(r.stdout.strip().splitlines()[-1])
    assert digests[0] == digests[1]


def test_captures_of_the_elementwise_steps_and_of_parts_are_not_limited():
    """Scheduler counters are handed out once to captured launches, 15,360 per process.  The elementwise backward kernels
    take none, however often they are captured, and a D = 128 backward in parts takes two, as one without parts does."""
    from machinelearning_b200 import _lib as L, flash_cuda as fc, qk_prologue, value_gate
    assert fc.is_available(), fc.unavailable_reason()
    lib = fc._load()
    g = torch.Generator(device="cuda").manual_seed(0)
    x, gy, v0 = (torch.randn(2, 40, 2, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
    w, lam = torch.randn(64, device="cuda", generator=g), torch.tensor([0.3], device="cuda")
    _, rstd = qk_prologue.fwd(x, w, None, None, 1e-6, torch.bfloat16)
    want = (*qk_prologue.bwd(gy, x, w, None, None, rstd), *value_gate.blend_bwd(gy, x, v0, lam))
    out = [torch.empty_like(t) for t in want]
    s1 = torch.full((lib.nlfa_qk_prologue_scratch_bytes(64),), 0xff, dtype=torch.uint8, device="cuda")
    s2 = torch.full((lib.nlfa_value_blend_scratch_bytes(),), 0xff, dtype=torch.uint8, device="cuda")
    # one (batch, KV head) pair's dS at a time: 1,024 parts
    B, T, H, D = 256, 8, 4, 128
    q, k, v, do = (torch.randn(B, T, H, D, device="cuda", generator=g).bfloat16() for _ in range(4))
    o, lse = fc.fwd(q, k, v, 0.1, True)
    grads = fc.bwd(do, q, k, v, o, lse, 0.1, True)
    parts = [torch.empty_like(t) for t in grads]
    tape = (lib.nlfa_bwd_scratch_bytes(B, T, H) + 255) // 256 * 256
    s3 = torch.empty(tape + 32768, dtype=torch.uint8, device="cuda")
    assert lib.nlfa_bwd_workspace_kernel_count(B, T, H, H, D, 0, 0, 0, L.DTYPE_BF16, L.PATH_TENSOR, s3.numel()) == 2049
    bf16 = L.DTYPE_BF16

    def steps(stream, n):
        for _ in range(n):
            L.check("prologue", lib.nlfa_qk_prologue_bwd(
                gy.data_ptr(), bf16, x.data_ptr(), bf16, w.data_ptr(), None, None, rstd.data_ptr(), out[0].data_ptr(),
                out[1].data_ptr(), s1.data_ptr(), s1.numel(), 2, 40, 2, 64, stream))
            L.check("blend", lib.nlfa_value_blend_bwd(
                gy.data_ptr(), bf16, x.data_ptr(), v0.data_ptr(), bf16, lam.data_ptr(), out[2].data_ptr(), out[3].data_ptr(),
                out[4].data_ptr(), s2.data_ptr(), s2.numel(), x.numel(), stream))

    def in_parts(stream):
        L.check("parts", lib.nlfa_bwd_masked(
            *(t.data_ptr() for t in (do, q, k, v, o, lse, *parts, s3)), s3.numel(), B, T, H, H, D, 0.1, 0, 0, 0, bf16,
            L.PATH_TENSOR, L.PASS_ALL, stream))

    steps(torch.cuda.current_stream().cuda_stream, 1)
    in_parts(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for run, count in ((lambda s: steps(s, 500), 17), (in_parts, 8)):            # 17,000 launches, 16,384 in parts
        for _ in range(count):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                run(torch.cuda.current_stream().cuda_stream)
        for t in (*out, *parts):
            t.fill_(float("nan"))
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        got, ref = (out, want) if count == 17 else (parts, grads)
        assert all(torch.equal(a, b) for a, b in zip(got, ref))
