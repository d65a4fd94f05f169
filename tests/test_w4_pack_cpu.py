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
    monkeypatch.setattr(quant, "_packer_runs_on", quant._packer_runs_on.__wrapped__)  # asked anew
    monkeypatch.setattr(quant, "_plain", lambda m: True, raising=False)  # the stand-in is no tensor
    m = SimpleNamespace(is_cuda=True, device=torch.device("cuda:0"), dtype=torch.bfloat16, shape=(16, 128),
                        numel=lambda: 2048, stride=lambda d: (128, 1)[d])
    assert quant._on_gpu(m) == taken
    assert quant._on_gpu(m, m) == taken


def test_fake_tensors_take_the_torch_packer():
    """Shape propagation has no data to launch a kernel on."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        w = torch.empty(40, 300, dtype=torch.bfloat16, device="cuda")
        p, gu = quant.quantize_w4(w), quant.quantize_w4_gate_up(w, w)
    assert p.qw.shape == (3, 6, 32, 4) and p.scales.shape == (3, 3, 16) and p.qw.device.type == "cuda"
    assert gu.qw.shape == (5, 6, 32, 4) and gu.gate_up


def test_what_is_not_plain_memory():
    w = torch.randn(16, 128)
    assert quant._plain(w) and quant._plain(torch.nn.Parameter(w)) and not quant._traced()
    assert not quant._plain(torch._neg_view(w))
    seen = []
    torch.func.vmap(lambda m: seen.append(quant._plain(m)) or m)(torch.stack([w, w]))
    assert seen == [False]
