"""The device of a call is made current by torch's exchange, whatever torch says is current."""

from __future__ import annotations

import pytest
import torch

from gpumode_cholesky_b200 import potrf


@pytest.mark.parametrize("before", [0, 1])
def test_every_call_exchanges_and_goes_back(monkeypatch, before):
    calls = []
    # A device torch has yet to switch to counts as current for getDevice.
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 1, raising=False)

    def exchange(index):
        calls.append(("to", index))
        return before

    monkeypatch.setattr(torch._C, "_cuda_exchangeDevice", exchange, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_maybeExchangeDevice", lambda index: calls.append(("back", index)), raising=False)
    with pytest.raises(KeyError):
        with potrf._on_device(torch.device("cuda", 1)):
            calls.append("work")
            raise KeyError
    assert calls == [("to", 1), "work"] + ([("back", before)] if before != 1 else [])
