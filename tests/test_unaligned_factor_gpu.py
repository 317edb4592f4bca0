"""Solves with a factor or a result that does not start on a 16-byte boundary."""

from __future__ import annotations

import pytest
import torch

from gpumode_cholesky_b200 import _lib, cholesky, inputs, potrf_backward
from gpumode_cholesky_b200.gp import gp_nll_from_factor, gp_nll_lbar, trsv

pytestmark = pytest.mark.gpu


def _shifted(t: torch.Tensor) -> torch.Tensor:
    """The same values four bytes past an allocation's start, contiguous."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    view = buf[1:].view(t.shape)
    view.copy_(t)
    assert view.is_contiguous() and view.data_ptr() % 16 == 4
    return view


def _rel(x: torch.Tensor, ref: torch.Tensor) -> float:
    return float(torch.linalg.norm(x.double() - ref) / torch.linalg.norm(ref))


@pytest.mark.parametrize("n", [32, 64, 100, 128, 129, 132, 192, 516, 1024])
def test_a_factor_off_the_boundary(n):
    a = inputs.well_conditioned(3, n, 80 + n, device="cuda")
    l = _shifted(cholesky(a, mode="fp32"))
    y = _shifted(torch.randn((3, n), device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)))
    ld, yd = l.double(), y.double().unsqueeze(-1)
    al = torch.linalg.solve_triangular(ld, yd, upper=False).squeeze(-1)
    be = torch.linalg.solve_triangular(ld.transpose(-1, -2), yd, upper=True).squeeze(-1)
    # Eigenvalues of A in [1, 5]: at most sqrt(5) amplification of n + 2 roundings.
    tol = 3 * (n + 2) * 2.0**-24
    assert _rel(trsv(l, y), al) <= tol
    assert _rel(trsv(l, y, trans=True), be) <= tol
    loss, alpha = gp_nll_from_factor(l, y)
    assert _rel(alpha, al) <= tol
    g = torch.ones(3, device="cuda")
    beta, lbar = gp_nll_lbar(l, y, g)
    assert torch.equal(beta, trsv(l, y, trans=True))
    # Into a result off the boundary, and the adjoint of operands off it.
    out = _shifted(torch.zeros_like(lbar))
    st = _lib.load().b2p_gp_nll_backward(
        l.data_ptr(), y.data_ptr(), g.data_ptr(), beta.data_ptr(), out.data_ptr(), 3, n,
        torch.cuda.current_stream().cuda_stream,
    )
    assert st == _lib.B2P_OK
    torch.cuda.synchronize()
    assert torch.equal(out, lbar)
    assert torch.equal(potrf_backward(l, out), potrf_backward(l.clone(), lbar))
