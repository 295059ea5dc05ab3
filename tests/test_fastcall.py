"""The extension module that makes the launch calls: what it takes, it passes as the Python function does; the
rest it hands to that function. A host callback stands in for the entry point."""
import ctypes as C
import os
import sys
import sysconfig

import pytest
import torch

import sager_b200
from sager_b200 import _fastcall, build, capi, ops

KINDS = "pipfiqzdp"                   # (not a list of the header's: every kind of parameter once, generated below)
STREAM = 0x5EED


@pytest.fixture
def bound():
    """An entry point of the parameter list of sgr_rmsnorm_quant_f16 (pppp i f i p) that records its arguments."""
    kinds = capi.kinds_of(capi.prototypes()["sgr_rmsnorm_quant_f16"])
    assert kinds == "ppppifip"
    seen, slow_calls, rc = [], [], [0]
    proto = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_float, C.c_int, C.c_void_p)

    @proto
    def entry(*a):
        seen.append(a)
        return rc[0]

    def slow(*args):
        slow_calls.append(args)
        return "slow"

    def fail(code):
        raise capi.SagerError("entry", code)

    _fastcall.setup(torch.Tensor, torch.nn.Parameter, lambda: STREAM, lambda dev: STREAM + dev, lambda: 1)
    fn = _fastcall.bind(kinds, C.cast(entry, C.c_void_p).value, slow, fail, "entry")
    yield fn, seen, slow_calls, rc, entry
    _fastcall.setup(torch.Tensor, torch.nn.Parameter, ops._stream, ops._raw_stream, ops._device)


def test_arguments_arrive_as_given(bound):
    fn, seen, slow_calls, rc, _ = bound
    t, p = torch.zeros(4), torch.nn.Parameter(torch.zeros(4))
    assert fn(t, p, None, 2 ** 63 + 8, -5, 0.5, True) is None and not slow_calls
    got = seen[-1]
    assert got[:4] == (t.data_ptr(), p.data_ptr(), None, 2 ** 63 + 8) and got[4:7] == (-5, 0.5, 1)
    assert got[7] in (STREAM, STREAM + 1)                              # the first call asks the Python function
    fn(t, t[1:], t, t, 2 ** 31 - 1, 1e-6, -2 ** 31)
    got = seen[-1]
    assert got[1] == t.data_ptr() + 4 and got[4] == 2 ** 31 - 1 and got[6] == -2 ** 31 and got[7] == STREAM + 1
    assert got[5] == C.c_float(1e-6).value


class Sub(torch.Tensor):
    pass


@pytest.mark.parametrize("args", [
    (0, 0, 0, 0, 2 ** 31, 0.5, 1), (0, 0, 0, 0, 1.0, 0.5, 1), (0, 0, 0, 0, 1, 1, 1), (0, 0, 0, -1, 1, 0.5, 1),
    (0, 0, 0, 2 ** 64, 1, 0.5, 1), (0, 0, 0, 0, 1, 0.5), (0, 0, 0, 0, 1, 0.5, 1, 1), (C.c_void_p(8), 0, 0, 0, 1, 0.5, 1), (b"x", 0, 0, 0, 1, 0.5, 1),
], ids=lambda a: repr(a)[:40])
def test_the_rest_goes_to_the_python_function(bound, args):
    fn, seen, slow_calls, _, _ = bound
    assert fn(*args) == "slow" and slow_calls == [args] and not seen


def test_subclasses_and_keywords_go_to_the_python_function(bound):
    fn, seen, slow_calls, _, _ = bound
    assert fn(torch.zeros(2).as_subclass(Sub), 0, 0, 0, 1, 0.5, 1) == "slow"
    with pytest.raises(TypeError):
        fn(0, 0, 0, 0, 1, 0.5, n=1)
    assert not seen


def test_a_return_code_raises(bound):
    fn, seen, _, rc, _ = bound
    rc[0] = 2
    with pytest.raises(capi.SagerError) as e:
        fn(0, 0, 0, 0, 1, 0.5, 1)
    assert e.value.code == 2 and len(seen) == 1


@pytest.mark.parametrize("module", ["missing", "older"])
def test_without_the_module_or_its_function_the_python_function_is_the_launcher(monkeypatch, module):
    class Older:
        setup, bind = staticmethod(_fastcall.setup), staticmethod(lambda *a: None)      # (what bind says to a list it does not have)

    monkeypatch.setattr(ops, "_fast", None)
    monkeypatch.delattr(sager_b200, "_fastcall")
    monkeypatch.setitem(sys.modules, "sager_b200._fastcall", None if module == "missing" else Older)
    if module == "older":
        monkeypatch.setattr(sager_b200, "_fastcall", Older, raising=False)
    fn = ops._bind("gemv_q4_k_q8")
    assert type(fn) is type(ops.call) and fn.__name__ == "gemv_q4_k_q8"
    monkeypatch.setattr(ops, "_raw_stream", lambda dev: 0)
    monkeypatch.setattr(ops, "_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    assert fn(16, 16, 16, 0, 2048) is None                             # empty: nothing to do
    with pytest.raises(capi.SagerError) as e:
        fn(None, None, None, 8, 2048)
    assert e.value.code == 1


def test_the_module_is_this_interpreters_and_follows_its_sources(monkeypatch, tmp_path):
    assert build.FASTCALL.endswith(sysconfig.get_config_var("EXT_SUFFIX")) and os.path.samefile(_fastcall.__file__, build.FASTCALL)
    copy = tmp_path / "module"
    copy.write_bytes(b"")
    monkeypatch.setattr(build, "FASTCALL", str(copy))
    newest = max(os.path.getmtime(p) for p in build.headers() + [os.path.join(build.CSRC, "fastcall.c"), os.path.join(build.HERE, "capi.py")])
    os.utime(copy, (newest, newest))
    assert not build.needs_fastcall()
    os.utime(copy, (newest, os.path.getmtime(os.path.join(build.HERE, "capi.py")) - 1))
    assert build.needs_fastcall()
    os.remove(copy)
    assert build.needs_fastcall()


def test_every_launcher_has_one():
    calls = build.fastcall_calls()
    for name, proto in capi.prototypes().items():
        kinds = capi.kinds_of(proto)
        if kinds is not None:
            assert f"call_{kinds}(" in calls, name
            assert _fastcall.bind(kinds, 1, None, None, name) is not None
    assert _fastcall.bind(KINDS, 1, None, None, "unknown list") is None
    assert not isinstance(ops.gemv_q4_k_q8, type(ops.call)) and ops.gemv_q4_k_q8.__name__ == "gemv_q4_k_q8"
