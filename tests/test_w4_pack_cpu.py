"""Which matrices `quant.quantize_w4` / `quantize_w4_gate_up` hand to the GPU packer: those that its kernel can
read, where its library can run. All others take torch's operators, as they did before there was a kernel."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from qengine_b200 import quant


@pytest.mark.parametrize("capability,built,taken", [((10, 0), True, True), ((10, 3), True, False), ((9, 0), True, False),
                                                    ((12, 0), True, False), ((10, 0), False, False)])
def test_only_where_the_library_runs(monkeypatch, tmp_path, capability, built, taken):
    """sm_100a code runs on capability 10.0 only, and packing must not need the library elsewhere."""
    lib = tmp_path / "libqengine_b200.so"
    if built:
        lib.touch()
    monkeypatch.setattr(quant, "_LIBRARY", lib, raising=False)
    monkeypatch.setattr(torch.cuda, "get_device_capability", lambda device=None: capability)
    m = SimpleNamespace(is_cuda=True, device=torch.device("cuda:0"), dtype=torch.bfloat16, shape=(16, 128),
                        numel=lambda: 2048, stride=lambda d: (128, 1)[d])
    assert quant._on_gpu(m) == taken
    assert quant._on_gpu(m, m) == taken
