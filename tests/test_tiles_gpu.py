"""The FP32 tile-task kernel at the edges of its tiles, task groups and loads."""

from __future__ import annotations

import pytest
import torch

import oracle
from gpumode_cholesky_b200 import cholesky, inputs
from gpumode_cholesky_b200.ragged import RaggedPlan, pack

pytestmark = pytest.mark.gpu

# Orders one tile over the small kernels, around multiples of 64, odd ones
# (4-byte loads) and multiples of 4; batches below and above one task group.
SHAPES = [(1, 129), (3, 191), (2, 192), (2, 193), (5, 255), (4, 256), (2, 257), (500, 130), (300, 196), (2, 700), (1, 1001)]


@pytest.mark.parametrize("batch,n", SHAPES)
def test_tiles_against_oracle(batch, n):
    a = inputs.well_conditioned(batch, n, 100 + n, device="cpu")
    info = torch.full((batch,), 9, dtype=torch.int32, device="cuda")
    out = torch.full((batch, n, n), float("nan"), device="cuda")
    first = cholesky(a.cuda(), mode="fp32", info=info, out=out).clone()
    again = cholesky(a.cuda(), mode="fp32")
    assert torch.equal(first, again)
    assert not info.any()
    assert not torch.triu(first, 1).any()
    some = sorted({0, batch // 2, batch - 1})
    l64, _ = oracle.potrf_f64(a[some].numpy())
    want = torch.from_numpy(l64)
    got = first[some].cpu().double()
    # Eigenvalues of M M^T / n + I lie in [1, 5]: n + 1 roundings, amplified 5 times.
    assert float(torch.linalg.norm(got - want) / torch.linalg.norm(want)) <= 5 * (n + 1) * 2.0**-24


def test_streams_do_not_meet():
    """Two streams, each with its own workspace, against one after the other."""
    a = [inputs.well_conditioned(6, 321, s, device="cuda") for s in (1, 2)]
    want = [cholesky(x, mode="fp32") for x in a]
    streams = [torch.cuda.Stream() for _ in a]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(5):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[k].append(cholesky(a[k], mode="fp32"))
    torch.cuda.synchronize()
    for k in range(2):
        assert all(torch.equal(g, want[k]) for g in got[k])


def test_captured_and_replayed():
    a = inputs.well_conditioned(3, 200, 5, device="cuda")
    want = cholesky(a, mode="fp32")
    out = torch.empty_like(a)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        cholesky(a, mode="fp32", out=out)
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


def test_same_values_as_the_ragged_schedule():
    orders = [129, 192, 200, 333, 515]
    mats = [inputs.well_conditioned(1, n, n, device="cuda")[0] for n in orders]
    buf, ns, offs = pack(mats)
    out = RaggedPlan(ns, offs, mode="fp32").factor(buf)
    for m, n, o in zip(mats, ns, offs):
        assert torch.equal(cholesky(m[None], mode="fp32")[0], out[o : o + n * n].view(n, n))
