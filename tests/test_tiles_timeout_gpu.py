"""The FP32 tile-task kernel when one of its waits gives up.

b2p_debug_potrf_tiles_stall starts one matrix's count of finished tiles far
below zero, so that the wait of its third diagonal tile runs out after the
caller's number of polls.  Every CTA must then leave, and nothing may look like
a result: info is -1 and the diagonal of L NaN for the whole batch, whichever
CTA stored last.  The next call on the same workspace is correct.
"""

from __future__ import annotations

import pytest
import torch

from gpumode_cholesky_b200 import _lib, cholesky, inputs

pytestmark = pytest.mark.gpu


# One tile column more than the wait needs, an odd order, and batches of more
# than one task group (whose first diagonal tiles wait for nothing).
@pytest.mark.parametrize("batch,n,matrix", [(1, 192, 0), (5, 193, 3), (3, 700, 1), (2000, 192, 700)])
@pytest.mark.parametrize("with_info", [True, False])
def test_a_wait_that_gives_up_marks_the_whole_batch(batch, n, matrix, with_info):
    lib = _lib.load()
    a = inputs.well_conditioned(batch, n, 7, device="cuda")
    want = cholesky(a, mode="fp32")
    out = torch.zeros_like(a)
    info = torch.full((batch,), 9, dtype=torch.int32, device="cuda")
    nbytes = lib.b2p_potrf_workspace_size(batch, n, _lib.MODE_FP32)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    info_ptr = info.data_ptr() if with_info else None
    st = lib.b2p_debug_potrf_tiles_stall(
        a.data_ptr(), out.data_ptr(), batch, n, matrix, 20000, ws.data_ptr(), nbytes, info_ptr, stream
    )
    assert st == _lib.B2P_OK, lib.b2p_last_error()
    torch.cuda.synchronize()
    if with_info:
        assert (info == -1).all()
    assert torch.isnan(out.diagonal(dim1=-2, dim2=-1)).all()
    st = lib.b2p_potrf_batched(
        a.data_ptr(), out.data_ptr(), batch, n, _lib.MODE_FP32, ws.data_ptr(), nbytes, info_ptr, stream
    )
    assert st == _lib.B2P_OK, lib.b2p_last_error()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    if with_info:
        assert not info.any()


def test_the_diagnostic_refuses_what_it_cannot_run():
    lib = _lib.load()
    a = torch.eye(192, device="cuda").repeat(2, 1, 1)
    out = torch.empty_like(a)
    ws = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    args = lambda n=192, matrix=0, polls=100, nbytes=1 << 20: (
        a.data_ptr(), out.data_ptr(), 2, n, matrix, polls, ws.data_ptr(), nbytes, None, None,
    )
    for bad in (args(n=128), args(matrix=2), args(matrix=-1), args(polls=0), args(polls=(1 << 24) + 1)):
        assert lib.b2p_debug_potrf_tiles_stall(*bad) == _lib.B2P_ERR_INVALID_ARG
    assert lib.b2p_debug_potrf_tiles_stall(*args(nbytes=100)) == _lib.B2P_ERR_WORKSPACE
