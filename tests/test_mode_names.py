"""What a mode may be does not depend on the calls before."""

from __future__ import annotations

import numpy as np
import pytest

from gpumode_cholesky_b200 import _lib
from gpumode_cholesky_b200.potrf import resolve_mode


@pytest.mark.parametrize("like", [float, np.float32, np.int64])
@pytest.mark.parametrize("first", [False, True])
def test_a_number_that_is_no_int_is_refused_before_and_after_its_equal(like, first):
    n = 160 if first else 192  # an order of its own, so that each case starts uncached
    if first:
        assert resolve_mode(_lib.MODE_BF16X3, n) == _lib.MODE_BF16X3
    with pytest.raises(AttributeError):
        resolve_mode(like(_lib.MODE_BF16X3), n)
    assert resolve_mode("bf16x3", n) == resolve_mode(_lib.MODE_BF16X3, n) == _lib.MODE_BF16X3
