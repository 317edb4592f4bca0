"""More matrices than SMs at orders where one CTA has the SM: full waves and a clustered tail."""

import pytest
import torch

from gpumode_cholesky_b200 import cholesky

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bf16x3", "tf32+guard"])
@pytest.mark.parametrize("n", [576, 1024])
@pytest.mark.parametrize("extra", [1, 80])
def test_more_matrices_than_sms(mode, n, extra):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch = sms + extra  # a tail of one matrix, and one of more than half a wave
    gen = torch.Generator(device="cuda").manual_seed(n + extra)
    m = torch.randn((batch, n, n), device="cuda", generator=gen)
    a = m @ m.transpose(-1, -2) / n
    a.diagonal(dim1=-2, dim2=-1).add_(1.0)
    a[1, 7, 7] = -1.0  # one in the first wave that is not positive definite, one in the last
    a[batch - 1, n - 1, n - 1] = -1.0
    info = torch.zeros(batch, dtype=torch.int32, device="cuda")
    want_info = torch.zeros_like(info)
    got = cholesky(a, mode=mode, info=info)
    # The one-CTA-per-matrix kernel does the same arithmetic: bitwise equal.
    want = cholesky(a, mode=mode, info=want_info, path="fused")
    assert torch.equal(info, want_info)
    assert info[1] == 8 and info[batch - 1] == n and info.count_nonzero() == 2
    good = info == 0
    assert torch.equal(got[good], want[good])
