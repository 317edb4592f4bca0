"""The solves, the Gaussian-process loss and the adjoint at orders up to 128, against FP64."""

from __future__ import annotations

import pytest
import torch

from gpumode_cholesky_b200 import cholesky, inputs, potrf_backward
from gpumode_cholesky_b200.gp import gp_nll_from_factor, gp_nll_lbar, trsv

pytestmark = pytest.mark.gpu


def _rel(x: torch.Tensor, ref: torch.Tensor) -> float:
    return (torch.linalg.norm((x.double() - ref).flatten()) / torch.linalg.norm(ref.flatten())).item()


@pytest.mark.parametrize("n", [1, 5, 31, 32, 33, 63, 64, 65, 97, 127, 128])
def test_small_orders_of_the_solves_and_the_adjoint(n):
    """Edges of the small kernels' warps and paddings: solves, loss, Lbar and the adjoint against FP64."""
    batch = 3
    a = inputs.well_conditioned(batch, n, 40 + n, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    y = torch.randn((batch, n), device="cuda", generator=gen)
    l = cholesky(a, mode="fp32")
    ld = l.double()
    loss, alpha = gp_nll_from_factor(l, y)
    a64 = torch.linalg.solve_triangular(ld, y.double().unsqueeze(-1), upper=False).squeeze(-1)
    x64 = torch.linalg.solve_triangular(ld.transpose(-1, -2), y.double().unsqueeze(-1), upper=True).squeeze(-1)
    # Eigenvalues of A in [1, 5]: at most sqrt(5) amplification of n + 2 roundings.
    tol = 3 * (n + 2) * 2.0**-24
    assert torch.equal(trsv(l, y), alpha)
    assert _rel(alpha, a64) <= tol
    assert _rel(trsv(l, y, trans=True), x64) <= tol
    want = 0.5 * (a64 * a64).sum(-1) + torch.log(torch.diagonal(ld, dim1=-2, dim2=-1)).sum(-1)
    assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5 * n)
    gl = torch.randn(batch, device="cuda", generator=gen)
    beta, lbar = gp_nll_lbar(l, alpha, gl)
    assert torch.equal(beta, trsv(l, alpha, trans=True))
    bd, ad, gd = beta.double(), alpha.double(), gl.double().view(-1, 1, 1)
    lb64 = gd * (torch.tril(-bd.unsqueeze(-1) * ad.unsqueeze(-2)) + torch.diag_embed(1 / torch.diagonal(ld, dim1=-2, dim2=-1)))
    assert _rel(lbar, lb64) <= 1e-6
    # The adjoint: S = L^{-T} Phi(L^T Lbar) L^{-1}, five products of length n,
    # amplified by at most the condition number 5.
    inv = torch.linalg.inv(ld)
    p = torch.tril(ld.transpose(-1, -2) @ lbar.double())
    p = p - 0.5 * torch.diag_embed(torch.diagonal(p, dim1=-2, dim2=-1))
    s = inv.transpose(-1, -2) @ p @ inv
    assert _rel(potrf_backward(l, lbar), 0.5 * (s + s.transpose(-1, -2))) <= 5 * 5 * (n + 2) * 2.0**-24
