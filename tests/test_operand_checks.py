"""What the launch builders refuse, on tensors that have a device but no memory (no GPU is needed and nothing is launched)."""
import types

import pytest
import torch
from torch._subclasses import FakeTensorMode

from helix_b200 import ops

H, F = torch.float16, torch.float32


def _t(*shape, dtype=H):
    return torch.empty(shape, dtype=dtype, device="cuda:0")


EXPANDED = {
    "weights for all batches": lambda: ops.launch_gemm_f16(_t(4, 8, 16), _t(8, 16).expand(4, 8, 16), _t(4, 8, 8)),
    "one row of A": lambda: ops.launch_gemm_f16(_t(1, 16).expand(8, 16), _t(8, 16), _t(8, 8)),
    "rows of C on each other": lambda: ops.launch_gemm_f16(_t(8, 16), _t(8, 16), _t(8).expand(8, 8)),
    "one vector": lambda: ops.launch_gemv_f16(_t(64, 16), _t(16).expand(3, 16), _t(3, 64)),
    "one row of weights": lambda: ops.launch_gemv_f16(_t(16).expand(64, 16), _t(3, 16), _t(3, 64)),
    "one output": lambda: ops.launch_gemv_f16(_t(64, 16), _t(3, 16), _t(3, 1).expand(3, 64)),
    "one fp32 vector": lambda: ops.launch_gemv_f32(_t(64, 16, dtype=F), _t(16, dtype=F).expand(3, 16), _t(3, 64, dtype=F)),
    "one fp32 row": lambda: ops.launch_gemm_f32(_t(16, dtype=F).expand(8, 16), _t(16, 8, dtype=F), _t(8, 8, dtype=F)),
}


@pytest.mark.parametrize("name", list(EXPANDED))
def test_expanded_operands_are_refused(name):
    with FakeTensorMode(), pytest.raises(ValueError, match="expanded"):
        EXPANDED[name]()


def _on(index, *shape):
    """What the checks read of a tensor on device `index`, which this machine may not have."""
    return types.SimpleNamespace(is_cuda=True, device=torch.device("cuda", index), shape=shape, dtype=H, dim=lambda: len(shape),
                                 get_device=lambda: index,
                                 stride=lambda: (shape[-1], 1))


@pytest.mark.parametrize("devices", [(0, 0, 1), (0, 1, 0), (1, 0, 0)])
@pytest.mark.parametrize("launch", [ops.launch_gemm_f16, ops.launch_gemv_f16, ops.launch_gemv_f32, ops.launch_gemm_f32])
def test_operands_of_two_devices_are_refused(launch, devices):
    with pytest.raises(ValueError, match="different devices"):
        launch(*(_on(d, 8, 8) for d in devices))


def test_a_batch_of_another_size_is_refused():
    with FakeTensorMode():
        for b, out in ((_t(1, 8, 16), _t(4, 8, 8)), (_t(4, 8, 16), _t(1, 8, 8))):
            with pytest.raises(AssertionError):
                ops.launch_gemm_f16(_t(4, 8, 16), b, out)


def test_eager_operators_run_on_the_current_device_only(monkeypatch):
    queued = []
    monkeypatch.setattr(ops, "run", queued.append)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    here, there = (types.SimpleNamespace(_refs=(_on(d, 8, 8),)) for d in (0, 1))
    ops._run_eager(here)
    with pytest.raises(ValueError, match="current"):
        ops._run_eager(there)
    assert queued == [here]


def test_expanded_dimensions_of_one_element_pass():
    with FakeTensorMode():
        ops._require_cuda(_t(1, 16).expand(1, 16), _t(8, 16)[:0], _t(3, 8, 16)[:1].expand(1, 8, 16))
