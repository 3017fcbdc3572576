"""Where the native module of the eager operators cannot be used, the same launches go through ctypes (no GPU needed)."""
import os
import subprocess
import sys
import types

import pytest
import torch

from helix_b200 import _lib, ops

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def without_module(monkeypatch):
    monkeypatch.setitem(sys.modules, "helix_b200._eager_call", None)     # importing it raises ImportError
    import helix_b200
    monkeypatch.delattr(helix_b200, "_eager_call", raising=False)
    monkeypatch.setattr(ops, "_eager", None)


def test_launches_go_through_ctypes_without_the_module(without_module, monkeypatch):
    queued, rc = [], [0]

    def launch(l, status, stream):
        queued.append((l, status, stream))
        return rc[0]

    fake = types.SimpleNamespace(helix_launch=launch, helix_status_string=lambda s: b"")
    monkeypatch.setattr(_lib, "load", lambda: fake)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(ops, "_stream", lambda dev: 77 + dev)
    monkeypatch.setitem(ops._status_words, 3, torch.zeros(1, dtype=torch.int32))
    l = ops.Launch()
    with pytest.warns(RuntimeWarning, match="_eager_call is not used"):
        ops.run(l)
    ops.run(l)                                                           # warned once
    assert [q[1:] for q in queued] == [(ops._status_words[3].data_ptr(), 80)] * 2
    h = torch.zeros(8, 8, dtype=torch.float16)
    assert ops._native().gemm_f16(h, h, None) is None
    rc[0] = -1
    with pytest.raises(_lib.HelixError):
        ops.run(l)


@pytest.mark.parametrize("version,native", [(torch.__version__, True), ("1.0", False)])
def test_the_module_serves_the_torch_it_was_built_for(version, native):
    code = ("import warnings, torch; torch.__version__ = %r; from helix_b200 import ops\n"
            "with warnings.catch_warnings(record=True) as w:\n    warnings.simplefilter('always'); n = ops._native()\n"
            "print(type(n).__name__, len(w))") % version
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, check=True, cwd=ROOT).stdout.split()
    assert out == (["module", "0"] if native else ["_PythonCalls", "1"])
