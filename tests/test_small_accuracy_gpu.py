"""Rounding errors of the small orders' kernels against FP32 forms of known order.

The reference forms run here, on the CPU, in FP32 with fused multiply-adds (a
product of two FP32 numbers is exact in FP64, so rounding the FP64 sum to FP32
is one fused multiply-add but for double roundings, one in 2^29).  A kernel that
groups its sums worse loses 10 to 50 % on squared-exponential covariances, whose
elements nearly cancel; two runs of the same order of operations differ by less
than 5 % in a root mean square over these many elements.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from gpumode_cholesky_b200 import cholesky
from gpumode_cholesky_b200.gp import trsv

pytestmark = pytest.mark.gpu

SLACK = 1.05
BATCH = 64


def _fma(a, b, c):
    return (a.astype(np.float64) * b + c).astype(np.float32)


def _covariances(n: int, noise: float, seed: int) -> np.ndarray:
    """Squared-exponential covariances over points in the unit cube, with noise."""
    rng = np.random.default_rng(seed)
    x = rng.random((BATCH, n, 3)).astype(np.float32)
    scale = (0.2 + 0.3 * rng.random((BATCH, 1, 1))).astype(np.float32)
    k = np.exp(-0.5 * ((x[:, :, None] - x[:, None]) ** 2).sum(-1) / (scale * scale)).astype(np.float32)
    k = 0.5 * (k + k.transpose(0, 2, 1))
    k[:, range(n), range(n)] += np.float32(noise)
    return k


def _gram(n: int, seed: int) -> np.ndarray:
    m = np.random.default_rng(seed).standard_normal((BATCH, n, n)).astype(np.float32)
    a = m @ m.transpose(0, 2, 1) / np.float32(n)
    a = 0.5 * (a + a.transpose(0, 2, 1))
    a[:, range(n), range(n)] += np.float32(1.0)
    return a


def _factor_blocks_of_32(a: np.ndarray) -> np.ndarray:
    """Product by product within 32 columns; the rest less the sum of the 32 products."""
    s, n = a.copy(), a.shape[1]
    for kb in range(0, n, 32):
        e = min(n, kb + 32)
        for k in range(kb, e):
            d = s[:, k, k].copy()
            y = (1.0 / np.sqrt(d.astype(np.float64))).astype(np.float32)
            s[:, k, k] = d * y
            s[:, k + 1 :, k] *= y[:, None]
            low = s[:, k + 1 :, k]
            s[:, k + 1 :, k + 1 : e] = _fma(-low[:, :, None], s[:, k + 1 : e, k][:, None, :], s[:, k + 1 :, k + 1 : e])
        if e < n:
            acc = np.zeros_like(s[:, e:, e:])
            for m in range(kb, e):
                acc = _fma(s[:, e:, m][:, :, None], s[:, e:, m][:, None, :], acc)
            s[:, e:, e:] -= acc
    return np.tril(s)


def _rms(x: np.ndarray, ref: np.ndarray) -> float:
    return float(np.sqrt(((x - ref) ** 2).sum() / (ref**2).sum()))


@pytest.mark.parametrize("n", [33, 40, 64, 65, 96, 128])
@pytest.mark.parametrize("kind", ["gram", "noise 0.1", "noise 0.001"])
def test_factor_no_further_off_than_blocks_of_32(n, kind):
    a = _gram(n, n) if kind == "gram" else _covariances(n, float(kind.split()[1]), n)
    exact = np.linalg.cholesky(a.astype(np.float64))
    got = cholesky(torch.from_numpy(a).cuda(), mode="fp32").cpu().numpy()
    assert _rms(got, exact) <= SLACK * _rms(_factor_blocks_of_32(a), exact)


def _solve_transposed(l: np.ndarray, b: np.ndarray) -> np.ndarray:
    """L^T x = b in blocks of 32 rows: a block's products in eight sums of four, added in pairs."""
    x, n = b.copy(), b.shape[1]
    inv = np.float32(1.0) / l[:, range(n), range(n)]
    for r0 in range((n - 1) // 32 * 32, -1, -32):
        e = min(n, r0 + 32)
        for j in range(e - 1, r0 - 1, -1):
            x[:, j] *= inv[:, j]
            x[:, r0:j] = _fma(-l[:, j, r0:j], x[:, j : j + 1], x[:, r0:j])
        p = np.zeros((8, x.shape[0], r0), dtype=np.float32)
        for j in range(r0, e):
            p[(j - r0) // 4] = _fma(l[:, j, :r0], x[:, j : j + 1], p[(j - r0) // 4])
        x[:, :r0] -= ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]))
    return x


@pytest.mark.parametrize("n", [40, 64, 67, 96, 128])
@pytest.mark.parametrize("noise", [0.1, 0.001])
def test_transposed_solve_no_further_off_than_sums_of_four(n, noise):
    l = np.linalg.cholesky(_covariances(n, noise, n + 1).astype(np.float64)).astype(np.float32)
    b = np.random.default_rng(n).standard_normal((BATCH, n)).astype(np.float32)
    exact = np.linalg.solve(l.astype(np.float64).transpose(0, 2, 1), b.astype(np.float64)[..., None])[..., 0]
    got = trsv(torch.from_numpy(l).cuda(), torch.from_numpy(b).cuda(), trans=True).cpu().numpy()
    assert _rms(got, exact) <= SLACK * _rms(_solve_transposed(l, b), exact)
