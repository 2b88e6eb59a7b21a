"""The stream handle that launches go to: torch's raw accessor where torch has
it, else the public call; a tensor off the GPU raises either way."""
import types

import pytest
import torch

from ginkgo_b200 import matrix


@pytest.mark.parametrize("raw", [True, False])
def test_handle(monkeypatch, raw):
    t = types.SimpleNamespace(device=torch.device("cuda", 1))
    asked = []

    def public(device):
        asked.append(("public", device.index))
        return types.SimpleNamespace(cuda_stream=77)

    def accessor(index):
        asked.append(("raw", index))
        return 77

    monkeypatch.setattr(torch.cuda, "current_stream", public)
    monkeypatch.setattr(matrix, "_raw_stream", accessor if raw else None)
    assert matrix._stream(t) == 77
    assert asked == [("raw" if raw else "public", 1)]


@pytest.mark.parametrize("raw", [True, False])
def test_cpu_tensor_raises(monkeypatch, raw):
    monkeypatch.setattr(matrix, "_raw_stream", (lambda index: 77) if raw else None)
    with pytest.raises((ValueError, RuntimeError, AssertionError)):
        matrix._stream(torch.zeros(3))
