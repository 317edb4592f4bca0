"""Which split-path calls take outer blocks, seen by the workspace they ask for (no GPU needed)."""

from __future__ import annotations

import pytest

from gpumode_cholesky_b200 import _lib

# Two outer-block buffers of n x (64 W) FP32 values per matrix.
CASES = [
    # Just below 104 block rows, and from there on.
    (6, 1088, 0), (5, 1280, 0), (3, 2048, 0), (1, 6592, 0),
    (7, 1088, 4), (6, 1152, 4), (300, 1088, 4), (4, 2048, 4), (1, 6656, 4), (1, 8192, 4), (1, 12224, 4),
    # Two buffers of 2048 bytes a row: 2 GiB at most.
    (963, 1088, 4), (1800, 1088, 0), (13500, 1088, 0), (128, 8192, 4), (150, 8192, 0),
    (1, 12288, 8), (100, 12288, 8), (1, 16384, 8),
]  # fmt: skip


@pytest.mark.parametrize("batch,n,width", CASES)
@pytest.mark.parametrize("mode", [_lib.MODE_TF32, _lib.MODE_BF16X3, _lib.MODE_FP8])
def test_outer_block_buffers(batch, n, width, mode):
    lib = _lib.load()
    ws = lib.b2p_potrf_path_workspace_size(batch, n, mode, _lib.PATHS["split"])
    rows = batch * n
    # Panel copies (4 bytes an element below the diagonal blocks) and two FP32
    # panel buffers of 64 columns; alignments and FP8 scales are below 256 bytes a row.
    N = n // 64
    rest = batch * 2 * (N * (N - 1) // 2) * 64 * 64 * 2 + 2 * rows * 64 * 4
    outer = 2 * rows * 64 * width * 4
    assert rest + outer <= ws <= rest + outer + 256 * rows


@pytest.mark.parametrize("n", [1088, 1152, 2048, 8192, 12224])
def test_a_workspace_serves_every_smaller_batch(n):
    lib = _lib.load()
    most = 2**31 // (2048 * n)  # the last batch with outer blocks
    batches = sorted({1, 2, 5, 6, 7, 8, most - 1, most, most + 1, 2 * most, 8 * most})
    sizes = [lib.b2p_potrf_path_workspace_size(b, n, _lib.MODE_BF16X3, _lib.PATHS["split"]) for b in batches]
    assert sizes == sorted(sizes)
