"""Host threads that factor on streams of their own at the same time.

The split path, the blocked path's look-ahead and the packed lists fork work to
library streams through events that all calls on a device share.  A call that
enqueues while another thread's call does must not wait on the other's events:
its look-ahead would start before the panels it reads are final.
"""

from __future__ import annotations

import threading

import pytest
import torch

from gpumode_cholesky_b200 import cholesky, inputs
from gpumode_cholesky_b200.ragged import RaggedPlan, pack

pytestmark = pytest.mark.gpu

CALLS = 12


def _in_threads(work) -> list[list[torch.Tensor]]:
    """work(k) CALLS times in thread k on stream k, both threads at once; the results."""
    got: list[list[torch.Tensor]] = [[], []]
    errors: list[BaseException] = []
    start = threading.Barrier(2)
    streams = [torch.cuda.Stream() for _ in got]
    torch.cuda.synchronize()

    def run(k: int) -> None:
        try:
            with torch.cuda.stream(streams[k]):
                start.wait(timeout=60)
                for _ in range(CALLS):
                    got[k].append(work(k))
        except BaseException as e:  # reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors and not any(t.is_alive() for t in threads), errors
    torch.cuda.synchronize()
    return got


# Split path without and with outer blocks; the blocked path's look-ahead.
@pytest.mark.parametrize("batch,n,mode", [(2, 1280, "bf16x3"), (1, 8192, "bf16x3"), (3, 448, "fp32+fp64diag")])
def test_two_threads_factor_at_once(batch, n, mode):
    a = [inputs.well_conditioned(batch, n, 30 + k, device="cuda") for k in range(2)]
    want = [cholesky(x, mode=mode) for x in a]
    got = _in_threads(lambda k: cholesky(a[k], mode=mode))
    for k in range(2):
        assert all(torch.equal(l, want[k]) for l in got[k])


def test_two_threads_factor_packed_lists_at_once():
    lists = [[200, 333, 640, 1100, 1300], [192, 450, 700, 1024, 1400]]
    packed = [pack([inputs.well_conditioned(1, n, n + k, device="cuda")[0] for n in ns]) for k, ns in enumerate(lists)]
    plans = [RaggedPlan(ns, offs, mode="bf16x3") for _, ns, offs in packed]
    # The gaps between packed matrices are not written.
    want = [plans[k].factor(packed[k][0], out=torch.zeros_like(packed[k][0])) for k in range(2)]
    got = _in_threads(lambda k: plans[k].factor(packed[k][0], out=torch.zeros_like(packed[k][0])))
    for k in range(2):
        assert all(torch.equal(l, want[k]) for l in got[k])
