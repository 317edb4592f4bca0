"""The split path's outer blocks below order 12288: batches, partial last blocks, and just outside the rule.

Bars as for the split path's other orders: relative residual 1e-5 (BF16x3),
2e-3 (TF32), 1e-4 (FP8) on Gram matrices with eigenvalues in [1, 5].
"""

from __future__ import annotations

import pytest
import torch

from gpumode_cholesky_b200 import cholesky, inputs

pytestmark = pytest.mark.gpu

BAR = {"bf16x3": 1e-5, "tf32": 2e-3, "fp8": 1e-4}

# Every remainder of the block columns modulo the outer block's four, more
# matrices than a step has CTAs for, and (first and last) just no outer blocks.
SHAPES = [(6, 1088), (7, 1088), (6, 1152), (6, 1216), (140, 1280), (4, 2048), (1, 6720), (1, 7232), (2, 5056), (1, 6592)]


@pytest.mark.parametrize("batch,n", SHAPES)
@pytest.mark.parametrize("mode", ["bf16x3", "tf32", "fp8"])
def test_outer_blocks(mode, batch, n):
    a = inputs.well_conditioned(batch, n, seed=n + batch, device="cuda")
    info = torch.full((batch,), -9, dtype=torch.int32, device="cuda")
    l = cholesky(a, mode=mode, info=info)
    assert (info == 0).all()
    assert (torch.triu(l, 1) == 0).all()
    assert (torch.diagonal(l, dim1=-2, dim2=-1) > 0).all()
    for b in range(0, batch, 8):  # slices of FP64
        ld, ad = l[b : b + 8].double(), a[b : b + 8].double()
        res = torch.linalg.matrix_norm(ld @ ld.transpose(-1, -2) - ad) / torch.linalg.matrix_norm(ad)
        assert res.max().item() <= BAR[mode]
    assert torch.equal(l, cholesky(a, mode=mode))
    # A bad pivot in the last block column, and one in the last whole outer block.
    late, last = n - 300, n - 2
    a[0, late, late] = -1.0
    a[batch - 1, last, last] = -1.0
    cholesky(a, mode=mode, info=info)
    assert info[batch - 1].item() == (last + 1 if batch > 1 else late + 1)
    assert info[0].item() == late + 1
    assert (info[1 : batch - 1] == 0).all()
