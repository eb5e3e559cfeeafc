"""The compiled launch binding: plain arguments reach the C function as ctypes would pass them, everything
else goes to the general (ctypes) call.  The library's functions are replaced by recording callbacks."""
import ctypes as C
import types

import pytest
import torch

from tuiskollm_b200 import _lib, build, ops


@pytest.fixture
def recorder():
    native = _lib.native(ops._launch)
    lib = _lib.load()
    calls, kept = [], []

    def stub(name):
        result, arguments = _lib.SIGNATURES[name]

        def body(*values):
            calls.append((name, values))
            return 5 if calls[0] == "fail" else 0

        kept.append(C.CFUNCTYPE(result, *arguments)(body))
        return C.cast(kept[-1], C.c_void_p).value

    general = []
    native.bind(stub, lambda *a: general.append(a))
    yield native, calls, general
    native.bind(lambda name: C.cast(getattr(lib, name), C.c_void_p).value, ops._launch)


def _context(address=0x7000):
    checked = []
    return types.SimpleNamespace(handle=C.c_void_p(address), checked=checked, check=checked.append)


def test_plain_arguments_arrive_as_ctypes_passes_them(recorder):
    native, calls, general = recorder
    c = _context()
    native.tk100_residual_rms_norm_quantize_nvfp4(c, 0x11, 3, 1 << 44, None, 0x30, 4, 5, 6, 7, 0.1, 8, 9)
    native.tk100_rms_norm(c, 0, (1 << 32) + 2, 1, 2, (1 << 64) - 16)  # masked like C.c_int
    native.tk100_fp8_gdn_output(c, 0, -1, 6144, None, 1, 2, 3, 4, 5)
    assert general == [] and c.checked == []
    assert calls[0] == ("tk100_residual_rms_norm_quantize_nvfp4",
                        (0x7000, 0x11, 3, 1 << 44, None, 0x30, 4, 5, 6, 7, C.c_float(0.1).value, 8, 9))
    assert calls[1][1] == (0x7000, None, 2, 1, 2, (1 << 64) - 16)
    assert calls[2][1][2:5] == (-1, 6144, None)


def test_a_failing_launch_is_checked_by_the_context(recorder):
    native, calls, general = recorder
    calls.append("fail")
    c = _context()
    native.tk100_rms_norm(c, 0, 1, 1, 2, 3)
    assert c.checked == [5] and general == []


@pytest.mark.parametrize("change", ["host", "float rows", "bool stream", "int divisor", "closed", "count", "object"])
def test_other_arguments_go_to_the_general_call(recorder, change):
    native, calls, general = recorder
    c = _context()
    arguments = [c, 0x11, 3, 16, 32, 48, 0.5, 80, 96, 0.25, 112]
    if change == "host":
        arguments[3] = torch.zeros(4)
    elif change == "float rows":
        arguments[2] = 3.0
    elif change == "bool stream":
        arguments[1] = True
    elif change == "int divisor":
        arguments[6] = 1
    elif change == "closed":
        c.handle = None
    elif change == "count":
        arguments.pop()
    else:
        arguments[3] = object()
    native.tk100_nvfp4_down(*arguments)
    assert calls == [] and len(general) == 1
    assert general[0][0] == "tk100_nvfp4_down"
    assert all(a is b for a, b in zip(general[0][1:], arguments, strict=True))


def test_the_general_call_reports_as_before():
    c = types.SimpleNamespace(_lib=_lib.load(), handle=None, check=lambda status: status)
    with pytest.raises(ops.GpuError) as info:
        _lib.native(ops._launch).tk100_rms_norm(c, 0, 1, torch.zeros(4), 2, 3)
    assert info.value.code == "gpu.context"
    with pytest.raises(C.ArgumentError):
        _lib.native(ops._launch).tk100_rms_norm(c, 0, 1.5, 1, 2, 3)


def test_a_binding_of_another_torch_or_interpreter_is_not_taken(monkeypatch):
    build.build_binding()
    assert not build.binding_is_stale()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.binding_is_stale()
    monkeypatch.undo()
    monkeypatch.setattr(build.sysconfig, "get_config_var", lambda name: ".other.so")
    assert build.binding_is_stale()


def test_without_a_binding_launches_take_the_general_call(monkeypatch):
    def fails(*_):
        raise RuntimeError("no compiler")

    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.setattr(build, "build_binding", fails)
    calls = []
    with pytest.warns(RuntimeWarning, match="no compiler"):
        native = _lib.native(lambda *a: calls.append(a))
    native.tk100_rms_norm("context", None, 1, 2, 3, 4)
    assert calls == [("tk100_rms_norm", "context", None, 1, 2, 3, 4)]


@pytest.mark.gpu
def test_tensors_and_streams(recorder):
    native, calls, general = recorder
    c = _context()
    x = torch.zeros((4, 64), dtype=torch.bfloat16, device="cuda")
    parameter = torch.nn.Parameter(x[1:])
    side = torch.cuda.Stream()
    native.tk100_rms_norm(c, None, 1, x, parameter, x[2:])
    with torch.cuda.stream(side):
        native.tk100_rms_norm(c, None, 1, x, None, x)
    assert [v for _, v in calls] == [
        (0x7000, torch.cuda.current_stream().cuda_stream or None, 1, x.data_ptr(), x.data_ptr() + 128, x.data_ptr() + 256),
        (0x7000, side.cuda_stream, 1, x.data_ptr(), None, x.data_ptr())]
    native.tk100_rms_norm(c, side, 1, x, x, x)
    native.tk100_rms_norm(c, None, 1, x[:, ::2], x, x)
    assert len(calls) == 2 and [g[0] for g in general] == ["tk100_rms_norm"] * 2
    with pytest.raises(ops.GpuError) as info:
        ops._launch("tk100_rms_norm", types.SimpleNamespace(_lib=_lib.load(), handle=None, check=None), side, 1,
                    x[:, ::2], x, x)
    assert info.value.code == "gpu.launch"
