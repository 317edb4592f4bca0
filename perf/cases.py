"""The work whose speed is tracked: a user's calls through the public entry points.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges.
A case is a dict: ``kind`` picks the entry point, the rest are its sizes.

kinds
  forward   ``custom_kernel(A)``: the drop-in, "auto" precision
  mode      ``cholesky(A, mode=..., info=...)``: the caller names the precision
  gp        ``gp_nll(A, y)`` and its gradients in A and y (one training step's work)
  grad      ``cholesky_differentiable(A)`` and the gradient of A for a given dLoss/dL
  ragged    ``RaggedPlan.factor`` on a packed list of different orders, plan built once

Inputs are seeded synthetic SPD matrices: batches M M^T / n + I, single large
ones G G^T / n + 0.1 I, and for ``gp`` an RBF covariance over points in the
unit cube with observation noise of variance 0.1.
"""

from __future__ import annotations

import math
import random

import torch

DEV = "cuda"


def listed() -> list[dict]:
    return [
        # The smallest call: a handful of small matrices of an odd order, as in
        # a filter update or a Newton step.  Latency is all there is.
        {"name": "forward_16x100", "kind": "forward", "batch": 16, "n": 100},
        # Very many very small matrices (per-sample covariances): the
        # benchmark's small workload, bound by memory.
        {"name": "forward_4096x32", "kind": "forward", "batch": 4096, "n": 32},
        # Second-order optimiser blocks: the two shapes of the benchmark's default step.
        {"name": "forward_640x512", "kind": "forward", "batch": 640, "n": 512},
        {"name": "forward_60x1024", "kind": "forward", "batch": 60, "n": 1024},
        # An order that is no multiple of the block size.
        {"name": "forward_50x500", "kind": "forward", "batch": 50, "n": 500},
        # Plain FP32, asked for by name, with the info vector.
        {"name": "fp32_8x2048", "kind": "mode", "mode": "fp32", "batch": 8, "n": 2048},
        # One large matrix, by the drop-in; and the largest, in the FP8 mode.
        {"name": "forward_1x8192", "kind": "forward", "batch": 1, "n": 8192},
        {"name": "fp8_1x16384", "kind": "mode", "mode": "fp8", "batch": 1, "n": 16384},
        # Gaussian-process likelihood, forward and backward: many small
        # problems, and a few of 2048 points.
        {"name": "gp_256x128", "kind": "gp", "batch": 256, "n": 128},
        {"name": "gp_8x2048", "kind": "gp", "batch": 8, "n": 2048},
        # A factorization inside a differentiable program.
        {"name": "grad_64x256", "kind": "grad", "batch": 64, "n": 256},
        # A list of matrices of all orders, packed.
        {"name": "ragged_400", "kind": "ragged", "mode": "bf16x3", "count": 400, "lo": 16, "hi": 2048, "orders_seed": 7},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _batch(rng: random.Random, n: int, most: int) -> int:
    """A batch of order n, with at most 4e7 elements and 6e10 multiply-adds' worth of n^3."""
    return _log_int(rng, 1, max(1, min(most, int(4e7 / n**2), int(6e10 / n**3))))


def draw(rng: random.Random) -> dict:
    kind = rng.choices(("forward", "mode", "gp", "grad", "ragged", "large"), (5, 4, 3, 3, 2, 2))[0]
    if kind == "large":
        # One large matrix; orders that are multiples of 64 (the tensor modes' own).
        n = 64 * _log_int(rng, 40, 224)
        if n >= 12288 or rng.random() < 0.5:
            return {"kind": "mode", "mode": rng.choice(("fp8", "bf16x3")), "batch": 1, "n": n}
        return {"kind": "forward", "batch": 1, "n": n}
    if kind == "ragged":
        hi = _log_int(rng, 100, 2048)
        count = _log_int(rng, 20, max(40, min(1500, int(1.5e9 / hi**2))))
        mode = rng.choice(("bf16x3", "bf16x3", "fp32"))
        return {"kind": "ragged", "mode": mode, "count": count, "lo": 16, "hi": hi, "orders_seed": rng.randrange(1 << 20)}
    n = _log_int(rng, 16, 2048)
    if n > 128 and rng.random() < 0.5:
        n = 64 * round(n / 64)
    if kind in ("gp", "grad"):
        return {"kind": kind, "batch": _batch(rng, n, 512), "n": n}
    case = {"kind": kind, "batch": _batch(rng, n, 8192), "n": n}
    if kind == "mode":
        case["mode"] = rng.choice(("fp32", "fp32", "tf32", "bf16x3"))
    return case


def _sym(a: torch.Tensor) -> torch.Tensor:
    return (0.5 * (a + a.transpose(-1, -2))).contiguous()


def _gram(gen: torch.Generator, batch: int, n: int, shift: float) -> torch.Tensor:
    m = torch.randn((batch, n, n), device=DEV, dtype=torch.float32, generator=gen)
    g = (m @ m.transpose(-1, -2)) / float(n)
    del m
    g.diagonal(dim1=-2, dim2=-1).add_(shift)
    return _sym(g)


def _rbf(gen: torch.Generator, batch: int, n: int) -> torch.Tensor:
    x = torch.rand((batch, n, 3), device=DEV, dtype=torch.float32, generator=gen)
    scale = 0.2 + 0.3 * torch.rand((batch, 1, 1), device=DEV, dtype=torch.float32, generator=gen)
    d2 = torch.zeros((batch, n, n), device=DEV, dtype=torch.float32)
    for i in range(3):
        d2 += (x[:, :, None, i] - x[:, None, :, i]).square()
    k = torch.exp(-0.5 * d2 / (scale * scale))
    k.diagonal(dim1=-2, dim2=-1).add_(0.1)
    return _sym(k)


def _orders(case: dict) -> list[int]:
    """Log-uniform orders in [lo, hi]."""
    rng = random.Random(case["orders_seed"])
    return [_log_int(rng, case["lo"], case["hi"]) for _ in range(case["count"])]


def _offsets(orders: list[int]) -> list[int]:
    """Element offsets of a packed list, each matrix on a 16-byte boundary, and the total."""
    offs, at = [], 0
    for n in orders:
        offs.append(at)
        at += (n * n + 3) // 4 * 4
    return offs + [at]


def _inputs(case: dict, seed: int) -> dict:
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "ragged":
        orders = _orders(case)
        offs = _offsets(orders)
        buf = torch.zeros(offs[-1], device=DEV, dtype=torch.float32)
        for n, o in zip(orders, offs):
            buf[o : o + n * n] = _gram(gen, 1, n, 1.0).reshape(-1)
        return {"a": buf, "orders": orders, "offsets": offs[:-1]}
    batch, n = case["batch"], case["n"]
    if kind == "gp":
        return {"a": _rbf(gen, batch, n), "y": torch.randn((batch, n), device=DEV, dtype=torch.float32, generator=gen)}
    a = _gram(gen, batch, n, 0.1 if batch == 1 and n > 2048 else 1.0)
    if kind == "grad":
        return {"a": a, "lbar": torch.randn((batch, n, n), device=DEV, dtype=torch.float32, generator=gen).tril_()}
    return {"a": a}


def prepare(case: dict, seed: int) -> dict:
    import gpumode_cholesky_b200 as lib

    state = {"lib": lib, "kind": case["kind"], "mode": case.get("mode"), **_inputs(case, seed)}
    if case["kind"] == "mode":
        state["info"] = torch.zeros(case["batch"], dtype=torch.int32, device=DEV)
    if case["kind"] in ("gp", "grad"):
        state["a"].requires_grad_(True)
    if case["kind"] == "gp":
        state["y"].requires_grad_(True)
    if case["kind"] == "ragged":
        from gpumode_cholesky_b200.ragged import RaggedPlan

        state["plan"] = RaggedPlan(state["orders"], state["offsets"], mode=case["mode"], device=torch.device(DEV, torch.cuda.current_device()))
        state["out"] = torch.zeros_like(state["a"])
        state["info"] = torch.zeros(case["count"], dtype=torch.int32, device=DEV)
    return state


def run(state: dict):
    lib, kind, a = state["lib"], state["kind"], state["a"]
    if kind == "forward":
        return lib.custom_kernel(a)
    if kind == "mode":
        return {"l": lib.cholesky(a, mode=state["mode"], info=state["info"]), "info": state["info"]}
    if kind == "gp":
        loss = lib.gp_nll(a, state["y"])
        ga, gy = torch.autograd.grad(loss.sum(), (a, state["y"]))
        return {"loss": loss, "ga": ga, "gy": gy}
    if kind == "grad":
        l = lib.cholesky_differentiable(a)
        (ga,) = torch.autograd.grad(l, a, state["lbar"])
        return {"l": l, "ga": ga}
    return {"l": state["plan"].factor(a, out=state["out"], info=state["info"]), "info": state["info"]}


def work(case: dict) -> dict:
    if case["kind"] == "ragged":
        orders = _orders(case)
        return {"bytes": 8.0 * sum(n * n for n in orders), "flops": sum(n**3 for n in orders) / 3.0}
    batch, n = case["batch"], case["n"]
    if case["kind"] == "gp":  # A in, its gradient out; the factor, and the inverse from it
        return {"bytes": batch * (8.0 * n * n + 8.0 * n + 4.0), "flops": batch * float(n**3)}
    if case["kind"] == "grad":  # A and dLoss/dL in, L and dLoss/dA out; the factor, L^T Lbar, two solves of which half is kept
        return {"bytes": batch * 16.0 * n * n, "flops": batch * 2.0 * n**3}
    return {"bytes": batch * 8.0 * n * n, "flops": batch * n**3 / 3.0}


def exact(case: dict, seed: int):
    given = _inputs(case, seed)
    kind = case["kind"]
    if kind == "ragged":
        out = torch.zeros(given["a"].shape, device=DEV, dtype=torch.float64)
        for n, o in zip(given["orders"], given["offsets"]):
            out[o : o + n * n] = torch.linalg.cholesky(given["a"][o : o + n * n].view(n, n).double()).reshape(-1)
        return {"l": out, "info": torch.zeros(case["count"], dtype=torch.int32, device=DEV)}
    a = given["a"].double()
    if kind == "gp":
        y = given["y"].double()
        l = torch.linalg.cholesky(a)
        inv = torch.cholesky_inverse(l)
        beta = (inv @ y.unsqueeze(-1)).squeeze(-1)
        loss = 0.5 * (y * beta).sum(-1) + l.diagonal(dim1=-2, dim2=-1).log().sum(-1)
        return {"loss": loss, "ga": 0.5 * (inv - beta.unsqueeze(-1) * beta.unsqueeze(-2)), "gy": beta}
    if kind == "grad":
        a.requires_grad_(True)
        l = torch.linalg.cholesky(a)
        (ga,) = torch.autograd.grad(l, a, given["lbar"].double())
        return {"l": l.detach(), "ga": ga}
    l = torch.linalg.cholesky(a)
    if kind == "mode":
        return {"l": l, "info": torch.zeros(case["batch"], dtype=torch.int32, device=DEV)}
    return l
