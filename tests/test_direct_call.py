"""The direct call's checks of its inputs, in native code and in Python: what is refused
goes the general way (no GPU: a stand-in takes the launch)."""

import ctypes
import subprocess
import sys

import pytest
import torch

from mlc_compiler_b200.executor import _DirectCall
from mlc_compiler_b200.runtime import native_call

SHAPE, WRITTEN = (4, 8), (0x10000, 0x10040)

_SETUP = """
import ctypes, torch
from mlc_compiler_b200.runtime import native_call
launched = []
LAUNCH = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32,
                          ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64, ctypes.c_uint32)
stand_in = LAUNCH(lambda *a: launched.append(a) or 0)
address = ctypes.cast(stand_in, ctypes.c_void_p).value
word = ctypes.c_uint32(0)
def fail(code):
    raise RuntimeError(f"code {code}")
def make(inputs, ptrs=(0, 64)):
    return native_call()(address, 0, 1, 32, 0, 0, 0, list(ptrs), inputs, [(0x10000, 0x10040)], "out", fail,
                         ctypes.addressof(word))
half = torch.empty(0, dtype=torch.float16)
call = make([((4, 8), half, 64, (0,))])
"""


def native(code: str) -> str:
    """Run ``code`` in a process of its own: at an entry without a guard a C++ exception
    ends the process."""
    if native_call() is None:
        pytest.skip("_mlcb_call.so is not built")
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", _SETUP + code], capture_output=True, text=True,
                       cwd=str(__import__("conftest").ROOT))
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.strip()


def in_python():
    """The Python form with the same input, on a launch that records."""
    d = _DirectCall.__new__(_DirectCall)
    d.native, d.index, d.launch, d.out, d.flags, d._last = None, 0, object(), "out", 0, None
    d.specs = [(torch.Size(SHAPE), torch.float16, 64, (0,))]
    d.written, d.fault, d.proved = [WRITTEN], None, True
    d.args = (0, 1, 32, 0, (ctypes.c_uint64 * 64)(), 2)
    d.run = lambda *a: pytest.fail("launched")
    return d


def test_an_input_without_memory_is_refused():
    got = native("""
from torch._subclasses import FakeTensorMode
with FakeTensorMode():
    t = torch.empty(4, 8, dtype=torch.float16, device="cuda:0")
print(call((t,)), call.last, launched)
""")
    assert got == "None None []"
    from torch._subclasses import FakeTensorMode
    with FakeTensorMode():
        t = torch.empty(*SHAPE, dtype=torch.float16, device="cuda:0")
    d = in_python()
    d._last = (t,)
    assert d((t,)) is None and d.last is None


def test_a_tensor_that_answers_with_an_exception_is_refused():
    """A batched tensor has no data pointer to give: asking for it throws."""
    got = native("""
from torch._subclasses import FakeTensorMode
seen = []
def one(x):
    try:
        x.data_ptr()
        seen.append("has one")
    except RuntimeError:
        pass
    seen.append(call((x,)))
    return x
with FakeTensorMode():
    torch.func.vmap(one)(torch.empty(3, 4, 8, dtype=torch.float16, device="cuda:0"))
print(seen, call.last, launched)
""")
    assert got == "[None] None []"


def test_arguments_a_call_cannot_be_made_of_raise():
    """Nothing a constructor or a call is given ends the process."""
    got = native("""
for what in (lambda: make([((4, 8), 3, 64, (0,))]), lambda: make([((4, 8), half, 64, (2,))]),
             lambda: make([((4, 8), half, 64, (-1,))]), lambda: make([((4, "x"), half, 64, (0,))]),
             lambda: make([], ["x"]), lambda: make([], [0] * 65), lambda: call(1), lambda: call()):
    try:
        what()
        print("accepted")
    except (TypeError, ValueError) as e:
        print(type(e).__name__)
print(call(()), call((1,)), call((torch.zeros(4, 8),)), launched)
""")
    assert got.splitlines() == ["TypeError", "ValueError", "ValueError", "TypeError", "TypeError", "ValueError",
                                "TypeError", "TypeError", "None None None []"]


def test_a_negated_view_is_refused():
    """Its memory holds the values before the sign."""
    d = in_python()
    d.index = -1                                       # host memory stands in for the device's
    ran = []
    d.run = lambda *a: ran.append(a) or 0
    x = torch.ones(SHAPE, dtype=torch.float16)
    torch._C._cuda_getCurrentRawStream, real = (lambda index: 0), getattr(torch._C, "_cuda_getCurrentRawStream", None)
    try:
        assert d((x,)) == "out" and len(ran) == 1 and d.args[4][0] == x.data_ptr()
        assert d((torch._neg_view(x),)) is None and len(ran) == 1
    finally:
        if real is None:
            del torch._C._cuda_getCurrentRawStream
        else:
            torch._C._cuda_getCurrentRawStream = real


def test_a_wait_that_ran_out_is_reported_at_the_next_call():
    got = native("""
print(call((torch.zeros(4, 8),)))
word.value = 1
try:
    call((torch.zeros(4, 8),))
    print("not reported")
except RuntimeError as e:
    print(e)
""")
    assert got.splitlines() == ["None", "code 0"]
    from mlc_compiler_b200.runtime import BackendError, LoadedModule

    loaded = LoadedModule.__new__(LoadedModule)
    loaded.handle, loaded.word = None, ctypes.c_uint32(1)
    with pytest.raises(BackendError, match="ran out"):
        loaded.check()
    loaded.check()                                     # reported once


def test_a_direct_call_needs_no_buffers_for_its_inputs():
    """They exist from the first call that copies an input; results stay where they are."""
    from mlc_compiler_b200 import Config
    from mlc_compiler_b200.executor import _Executable
    from perf import cases

    s = cases.rows_schedule("gelu", 8, 64, "float16")
    form = _Executable.__new__(_Executable)
    form.cfg, form.device = Config(), torch.device("cpu")
    form._bind_form(s, s, {"bias": torch.zeros(64, dtype=torch.float16)}, relaxed=False)
    first = dict(form._storage())
    assert "y" in first and not {"x", "res"} & set(first)
    x, res = torch.ones(8, 64), torch.zeros(8, 64, dtype=torch.float16)
    after = form._resident_buffers([x, res])
    assert torch.equal(after["x"], torch.ones(512, dtype=torch.float16)) and after["y"] is first["y"]
    assert form._resident_buffers([x * 2, res])["x"] is after["x"] and int(after["x"][0]) == 2
