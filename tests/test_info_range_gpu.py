"""info names a pivot of the matrix, never one of the padding beyond its order.

An infinite last pivot is positive, so info is 0, but L's last entry is NaN, and
identity padding behind it must not count as the failing pivot it then is.
"""

from __future__ import annotations

import pytest
import torch

from gpumode_cholesky_b200 import cholesky, inputs
from gpumode_cholesky_b200.ragged import RaggedPlan, pack

pytestmark = pytest.mark.gpu

ORDERS = [1, 5, 31, 32, 33, 50, 63, 64, 65, 100, 127, 128, 129, 150, 192, 200, 333]


def _with_infinite_last_pivot(n: int) -> torch.Tensor:
    a = inputs.well_conditioned(2, n, 60 + n, device="cpu")
    a[1, n - 1, n - 1] = float("inf")
    return a.cuda()


@pytest.mark.parametrize("mode", ["fp32", "fp32+fp64diag", "tf32", "bf16x3"])
@pytest.mark.parametrize("n", ORDERS)
def test_dense(n, mode):
    a = _with_infinite_last_pivot(n)
    info = torch.full((2,), 9, dtype=torch.int32, device="cuda")
    l = cholesky(a, mode=mode, info=info)
    assert info.tolist() == [0, 0]
    assert torch.isfinite(l[0]).all() and torch.isfinite(l[1, : n - 1]).all()
    assert not torch.triu(l, 1).any()


@pytest.mark.parametrize("mode", ["fp32", "tf32", "bf16x3"])
def test_packed_list(mode):
    buf, ns, offs = pack([_with_infinite_last_pivot(n)[1] for n in ORDERS])
    info = torch.full((len(ns),), 9, dtype=torch.int32, device="cuda")
    RaggedPlan(ns, offs, mode=mode).factor(buf, info=info)
    assert info.tolist() == [0] * len(ns)
