"""Eager operators: the native call against the Python implementation it stands for, over the forms both accept and refuse."""
import threading

import pytest
import torch
from torch.overrides import TorchFunctionMode

from helix_b200 import _lib, ops


class _Covers:
    """Stands in for the native module and covers nothing, so that the Python implementation runs."""

    def __getattr__(self, name):
        if name == "run":
            return ops._eager.run
        return lambda *args: None


def _both(monkeypatch, call):
    """Results (or exceptions) of the native call and of the Python implementation."""
    got = []
    for native in (True, False):
        with monkeypatch.context() as m:
            if not native:
                ops._native()
                m.setattr(ops, "_native", lambda: _Covers())
            try:
                got.append(call())
            except Exception as e:
                got.append((type(e), getattr(e, "status", None)))
    return got


def _rand(*shape, dtype=torch.float16):
    return torch.randn(*shape, device="cuda", dtype=torch.float32).to(dtype)


CALLS = {
    "gemv": lambda: ops.gemv_f16(_w["w"], _w["x"]),
    "gemv rows apart": lambda: ops.gemv_f16(_w["w"][:, :64], _w["x"][:, :64]),
    "gemv own output": lambda: ops.gemv_f16(_w["w"], _w["x"], out=torch.zeros(3, 512, device="cuda", dtype=torch.float16)[:, :300]),
    "gemv transposed output": lambda: ops.gemv_f16(_w["w"], _w["x"], out=torch.zeros(300, 3, device="cuda", dtype=torch.float16).t()),
    "gemv few rows, cut K": lambda: ops.gemv_f16(_w["long"], _w["longx"]),
    "gemv unaligned": lambda: ops.gemv_f16(_w["w"][:, 1:65], _w["x"][:, :64]),
    "gemv columns first": lambda: ops.gemv_f16(_w["w"].t().contiguous().t(), _w["x"]),
    "gemv wrong K": lambda: ops.gemv_f16(_w["w"], _w["x"][:, :64]),
    "gemv wrong type": lambda: ops.gemv_f16(_w["w"].float(), _w["x"]),
    "gemv nine vectors": lambda: ops.gemv_f16(_w["w"], _w["x"].repeat(3, 1)),
    "gemv on the CPU": lambda: ops.gemv_f16(_w["w"].cpu(), _w["x"].cpu()),
    "gemv parameter": lambda: ops.gemv_f16(torch.nn.Parameter(_w["w"]), _w["x"]),
    "gemv one vector for all": lambda: ops.gemv_f16(_w["w"], _w["x"][:1].expand(3, -1)),
    "gemv one row for all": lambda: ops.gemv_f16(_w["w"][:1].expand(300, -1), _w["x"]),
    "gemv expanded output": lambda: ops.gemv_f16(_w["w"], _w["x"], out=torch.zeros(300, device="cuda", dtype=torch.float16).expand(3, 300)),
    "gemv one expanded vector": lambda: ops.gemv_f16(_w["w"], _w["x"][:1].expand(1, -1)),
    "gemv_f32 one vector for all": lambda: ops.gemv_f32(_w["w"].float(), _w["x"][:1].float().expand(3, -1)),
    "gemm weights for all batches": lambda: ops.gemm_f16(_w["a3"], _w["b3"][0].expand(2, -1, -1)),
    "gemm one batch, expanded": lambda: ops.gemm_f16(_w["a3"][:1], _w["b3"][0].expand(1, -1, -1)),
    "gemm one row for all": lambda: ops.gemm_f16(_w["a"][:1].expand(70, -1), _w["w"]),
    "gemm_f32 one row for all": lambda: ops.gemm_f32(_w["a"][:1].float().expand(70, -1), _w["w"].float().t().contiguous()),
    "gemv_f32": lambda: ops.gemv_f32(_w["w"].float(), _w["x"].float()),
    "gemm": lambda: ops.gemm_f16(_w["a"], _w["w"]),
    "gemm batched": lambda: ops.gemm_f16(_w["a3"], _w["b3"]),
    "gemm rows apart": lambda: ops.gemm_f16(_w["a"][:, :64], _w["w"][:, :64], out=torch.zeros(70, 400, device="cuda", dtype=torch.float16)[:, :300]),
    "gemm wrong shape": lambda: ops.gemm_f16(_w["a"], _w["w"][:, :64]),
    "gemm workspace": lambda: ops.gemm_f16(_w["a"][:40, :], _rand(2048, 136)),
    "gemm_f32": lambda: ops.gemm_f32(_w["a"].float(), _w["w"].float().t().contiguous()),
    "gemm_f32 transposed": lambda: ops.gemm_f32(_w["a"].float().t().contiguous(), _w["w"].float().t().contiguous(), trans_a=True),
    "conv": lambda: ops.conv2d_f16_nhwc(_w["img"], _w["flt"], 1, 1),
    "conv strided own output": lambda: ops.conv2d_f16_nhwc(_w["img"], _w["flt"], 2, 1, out=torch.zeros(2, 5, 6, 16, device="cuda", dtype=torch.float16)),
    "conv wrong output": lambda: ops.conv2d_f16_nhwc(_w["img"], _w["flt"], 2, 1, out=torch.zeros(2, 5, 5, 16, device="cuda", dtype=torch.float16)),
    "conv not contiguous": lambda: ops.conv2d_f16_nhwc(_w["img"].transpose(1, 2), _w["flt"], 1, 1),
    "conv filter too large": lambda: ops.conv2d_f16_nhwc(_w["img"][:, :1].contiguous(), _w["flt"], 1, 0),
    "conv_f32": lambda: ops.conv2d_f32_nhwc(_w["img"].float(), _w["flt"].float(), 1, 1),
}
_w = {}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CALLS))
def test_native_call_and_python_agree(monkeypatch, name):
    torch.manual_seed(3)
    _w.update(w=_rand(300, 136), x=_rand(3, 136), long=_rand(64, 16384), longx=_rand(2, 16384), a=_rand(70, 136),
              a3=_rand(2, 70, 136), b3=_rand(2, 72, 136), img=_rand(2, 9, 11, 8), flt=_rand(16, 3, 3, 8))
    new_b = CALLS[name]
    torch.manual_seed(4)
    state = torch.cuda.get_rng_state()

    def call():
        torch.cuda.set_rng_state(state)     # a call that draws an operand draws the same one
        return new_b()

    native, python = _both(monkeypatch, call)
    if isinstance(python, tuple):
        assert native == python
    else:
        assert type(native) is type(python) and native.stride() == python.stride() and not native.requires_grad
        assert torch.equal(native, python)


# what the native module must serve itself (or refuse, where the launch does); everything else it leaves to Python
SERVES = {"gemv", "gemv rows apart", "gemv own output", "gemv transposed output", "gemv few rows, cut K", "gemv parameter",
          "gemv one expanded vector", "gemv_f32", "gemm", "gemm batched", "gemm rows apart", "gemm workspace", "gemm one batch, expanded",
          "gemm_f32", "gemm_f32 transposed", "conv", "conv strided own output", "conv_f32"}
REFUSES = {"gemv unaligned", "gemv nine vectors"}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CALLS))
def test_native_call_serves_what_it_should(monkeypatch, name):
    torch.manual_seed(3)
    _w.update(w=_rand(300, 136), x=_rand(3, 136), long=_rand(64, 16384), longx=_rand(2, 16384), a=_rand(70, 136),
              a3=_rand(2, 70, 136), b3=_rand(2, 72, 136), img=_rand(2, 9, 11, 8), flt=_rand(16, 3, 3, 8))
    native, seen = ops._native(), []

    class Watch:
        def __getattr__(self, op):
            def call(*args):
                seen.append("refused")
                got = getattr(native, op)(*args)
                seen[-1] = "left" if got is None else "served"
                return got
            return native.run if op == "run" else call

    monkeypatch.setattr(ops, "_native", Watch)
    try:
        CALLS[name]()
    except Exception:
        pass
    torch.cuda.synchronize()
    assert seen == ["served" if name in SERVES else "refused" if name in REFUSES else "left"]


@pytest.mark.gpu
def test_native_call_leaves_function_modes_to_python():
    a, b = _rand(70, 136), _rand(300, 136)
    plain, calls = ops.gemm_f16(a, b), []

    class Mode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            calls.append(func)
            return func(*args, **(kwargs or {}))

    with Mode():
        assert ops._native().gemm_f16(a, b, None) is None
        got = ops.gemm_f16(a, b)
    assert torch.equal(got, plain) and calls


@pytest.mark.gpu
def test_native_calls_follow_streams_and_threads():
    a, b, w, x = _rand(70, 136), _rand(300, 136), _rand(300, 136), _rand(3, 136)
    assert not ops.launch_gemm_f16(a, b, torch.empty(70, 300, device="cuda", dtype=torch.float16)).ws    # no scratch is shared
    want = ops.gemm_f16(a, b), ops.gemv_f16(w, x)
    zeros = torch.zeros_like(a)
    torch.cuda.synchronize()
    wrong = []

    def work():
        try:
            torch.cuda.set_device(0)
            side = torch.cuda.Stream()
            with torch.cuda.stream(side):
                mine = torch.empty_like(a)
                for _ in range(50):
                    mine.copy_(zeros)                       # the product must come after these on this thread's stream
                    torch.cuda._sleep(20000)
                    mine.copy_(a)
                    got = ops.gemm_f16(mine, b), ops.gemv_f16(w, x)
                    side.synchronize()
                    if not all(torch.equal(g, r) for g, r in zip(got, want)):
                        wrong.append("differs")
        except Exception as e:
            wrong.append(repr(e))

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.gpu
@pytest.mark.parametrize("name", [n for n in CALLS if "for all" in n or "expanded output" in n])
def test_expanded_operands_are_refused(name):
    _w.update(w=_rand(300, 136), x=_rand(3, 136), a=_rand(70, 136), a3=_rand(2, 70, 136), b3=_rand(2, 72, 136))
    with pytest.raises(ValueError, match="expanded"):
        CALLS[name]()


@pytest.mark.gpu
def test_run_takes_prepared_launches_only():
    w, x = _rand(64, 64), _rand(1, 64)
    out = torch.empty(1, 64, device="cuda", dtype=torch.float16)
    ops.run(ops.launch_gemv_f16(w, x, out))
    assert torch.equal(out, ops.gemv_f16(w, x))
    with pytest.raises(TypeError):
        ops.run(_lib.Cfg())
    bad = ops.launch_gemv_f16(w, x, out)
    bad.lda = 63
    with pytest.raises(_lib.HelixError):
        ops.run(bad)


def test_host_tensors_are_left_to_python():
    native = ops._native()
    h = torch.zeros(8, 8, dtype=torch.float16)
    assert native.gemv_f16(h, h, None) is None and native.gemm_f16(h, h, None) is None
    assert native.gemm_f32(h.float(), h.float(), False, None) is None
    assert native.conv2d_f16(h.view(1, 2, 4, 8), h.view(1, 2, 4, 8), 1, 0, None) is None
    with pytest.raises(ValueError):
        ops.gemm_f16(h, h)
