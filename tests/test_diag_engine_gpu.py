"""The 64x64 diagonal engine's edges, through the n > 128 factorizations.

The engine works in panels of 16 columns and groups of 4 pivots, with a fast
form for normal pivots and a general one: a pivot that fails, or is subnormal,
at each kind of place in that structure.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from gpumode_cholesky_b200 import cholesky, inputs

pytestmark = pytest.mark.gpu

PLACES = (0, 3, 4, 15, 16, 30, 32, 47, 48, 63, 64, 81, 127, 128, 190)


@pytest.mark.parametrize("mode", ["fp32", "bf16x3"])
def test_failing_pivot_at_every_kind_of_place(mode):
    n = 192
    a = inputs.well_conditioned(len(PLACES), n, 11, device="cpu")
    for b, k in enumerate(PLACES):
        a[b, k, k] = -1.0
    info = torch.zeros(len(PLACES), dtype=torch.int32, device="cuda")
    l = cholesky(a.cuda(), mode=mode, info=info).cpu()
    assert info.cpu().tolist() == [k + 1 for k in PLACES]
    # The columns before the failing one are those of the matrix without it.
    fixed = a.clone()
    for b, k in enumerate(PLACES):
        fixed[b, k, k] = a.abs().sum()
    want = cholesky(fixed.cuda(), mode=mode).cpu()
    for b, k in enumerate(PLACES):
        assert torch.equal(l[b, :, :k], want[b, :, :k])
        assert torch.isnan(l[b, k:, k]).all()


@pytest.mark.parametrize("first", [0, 5, 16, 40, 63, 64, 130])
def test_subnormal_pivots(first):
    """Rows and columns from `first` on scaled by 2^-64: their pivots are near 2^-127, subnormal."""
    n = 192
    a = inputs.well_conditioned(2, n, 12, device="cpu").double() / 4.0
    s = torch.ones(n, dtype=torch.float64)
    s[first:] = 2.0**-64
    scaled = (a * s[:, None] * s[None, :]).float()
    assert (scaled.diagonal(dim1=-2, dim2=-1)[:, first:] < 1.17549435e-38).all()
    info = torch.ones(2, dtype=torch.int32, device="cuda")
    l = cholesky(scaled.cuda(), mode="fp32", info=info).cpu().double() / s[:, None]
    assert info.cpu().tolist() == [0, 0]
    # The input as rounded to FP32 is what is factored; what is left is that the
    # products and sums near 2^-128 are rounded to multiples of 2^-149: at
    # most n + 2 of those per element, against pivots of at least 2^-129.
    exact = torch.from_numpy(np.linalg.cholesky((scaled.double() / s[:, None] / s[None, :]).numpy()))
    rel = torch.linalg.norm(l - exact) / torch.linalg.norm(exact)
    assert float(rel) <= (n + 2) * 2.0**-20, float(rel)


def test_oracle_agrees_on_the_failing_place():
    a = inputs.well_conditioned(1, 192, 13, device="cpu")
    a[0, 81, 81] = -1.0
    _, info = oracle.potrf_f64(a.numpy())
    assert int(info[0]) == 82


@pytest.mark.parametrize("n", [33, 47, 48, 49, 63, 64, 65, 66, 79, 80, 81, 96, 97, 111, 112, 113, 127, 128])
def test_small_orders(n):
    """One CTA per matrix: the edges of its panels, blocks and vector loads."""
    batch = 5
    a = inputs.well_conditioned(batch, n, 200 + n, device="cpu")
    bad = [None, 0, n - 1, 17, 31]
    for b, k in enumerate(bad):
        if k is not None:
            a[b, k, k] = -1.0
    info = torch.full((batch,), 9, dtype=torch.int32, device="cuda")
    out = torch.full((batch, n, n), float("nan"), device="cuda")
    l = cholesky(a.cuda(), info=info, out=out).cpu()
    assert info.cpu().tolist() == [0 if k is None else k + 1 for k in bad]
    assert not torch.triu(l, 1).any()
    l64, _ = oracle.potrf_f64(a[:1].numpy())
    want = torch.from_numpy(l64)[0]
    # Eigenvalues of M M^T / n + I lie in [1, 5]: n + 1 roundings, amplified 5 times.
    assert float(torch.linalg.norm(l[0].double() - want) / torch.linalg.norm(want)) <= 5 * (n + 1) * 2.0**-24
    for b, k in enumerate(bad):
        if k is not None:
            assert torch.isfinite(l[b, :, :k]).all() and torch.isnan(l[b, k:, k]).all()
