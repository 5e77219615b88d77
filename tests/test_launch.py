"""The native launch path of the binding: every argument of every entry point's signature reaches the C function."""
import ctypes as C
import subprocess
import sys

import numpy as np
import pytest

from paddock_b200 import _launch
from paddock_b200 import pack as packmod

SIGS = sorted(set(packmod._SIGS.values()) | set(packmod._EXTRA_SIGS.values()))
_CTYPE = {"p": "void*", "u": "uint32_t", "U": "uint64_t", "f": "float"}


@pytest.fixture(scope="module")
def echo(tmp_path_factory):
    """One C function per signature that leaves its arguments, as doubles, in `seen`."""
    src = "#include <stdint.h>\ndouble seen[32];\n"
    for i, sig in enumerate(SIGS):
        args = "".join(f"{_CTYPE[c]} a{j}, " for j, c in enumerate(sig))
        body = "".join(f"seen[{j}] = (double){'(uintptr_t)' if c == 'p' else ''}a{j}; " for j, c in enumerate(sig))
        src += f"int echo{i}({args}void* st) {{ {body}seen[{len(sig)}] = (double)(uintptr_t)st; return {i % 3}; }}\n"
    d = tmp_path_factory.mktemp("echo")
    (d / "echo.c").write_text(src)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", str(d / "libecho.so"), str(d / "echo.c")])
    return C.CDLL(str(d / "libecho.so"))


class _Tensor:
    def __init__(self, addr):
        self.addr = addr

    def data_ptr(self):
        return self.addr


@pytest.mark.parametrize("i", range(len(SIGS)), ids=SIGS)
def test_arguments_arrive(echo, i):
    sig = SIGS[i]
    addr = C.cast(getattr(echo, f"echo{i}"), C.c_void_p).value
    slow = []
    caller = _launch.Caller(lambda name: _launch.Entry(addr, sig, name), lambda *a, **k: slow.append((a, k)) or 7, None)
    args, want = [], []
    for j, c in enumerate(sig):
        v = {"p": 0x7f0000001000 + 64 * j, "u": 0xfffffff0 + j % 8, "U": (1 << 40) + j, "f": 0.5 + j}[c]
        args.append(_Tensor(v) if c == "p" and j % 2 else v)
        want.append(float(v))
    assert caller("x", *args, stream=0x1234) == i % 3
    assert list((C.c_double * 32).in_dll(echo, "seen")[:len(sig) + 1]) == want + [float(0x1234)]
    if "p" in sig:                           # None is a null pointer; a ctypes array takes the slow route
        at = sig.index("p")
        assert caller("x", *(None if c == "p" else a for c, a in zip(sig, args))) == i % 3
        assert (C.c_double * 32).in_dll(echo, "seen")[at] == 0.0 and not slow
        args[at] = (C.c_uint8 * 4)()
        assert caller("x", *args, stream=5) == 7 and slow == [(("x", *args), {"stream": 5})]
    with pytest.raises(TypeError):
        caller("x", *args[:-1])


def test_errors(echo):
    addr = C.cast(echo.echo1, C.c_void_p).value
    call = _launch.Caller(lambda name: _launch.Entry(addr, SIGS[1], name), None, packmod.LaunchError)
    with pytest.raises(packmod.LaunchError) as e:
        call("some_slot", *[0] * len(SIGS[1]))
    assert e.value.status == 1 and "some_slot" in str(e.value)
    with pytest.raises(ValueError):
        _launch.Entry(addr, "pfpfpf", "no such signature")
    with pytest.raises(TypeError):
        call("some_slot", *[0] * len(SIGS[1]), flow=1)


def test_what_ctypes_takes_goes_through_ctypes(echo):
    """The stream as a ctypes pointer, numbers as ctypes or numpy scalars: the slow route, nothing refused and nothing read."""
    sig = "pppppufu"
    i = SIGS.index(sig)
    addr = C.cast(getattr(echo, f"echo{i}"), C.c_void_p).value
    slow = []
    caller = _launch.Caller(lambda name: _launch.Entry(addr, sig, name), lambda *a, **k: slow.append((a, k)) or 7, None)
    args = [64, 128, 192, 256, 320, 3, 0.5, 9]
    assert caller("x", *args, stream=None) == i % 3 and not slow
    st = C.c_void_p(0x77)
    assert caller("x", *args, stream=st) == 7 and slow.pop() == (("x", *args), {"stream": st})
    for at, v in ((5, np.int64(3)), (5, C.c_uint32(3)), (6, np.float32(0.5)), (6, C.c_float(0.5)), (6, _Tensor(4096))):
        odd = [*args[:at], v, *args[at + 1:]]
        assert caller("x", *odd, stream=5) == 7 and slow.pop() == (("x", *odd), {"stream": 5})


@pytest.mark.parametrize("native", [True, False])
def test_pack_calls_with_and_without_the_extension(native):
    """The package (file formats included) imports and calls the library without _launch as well; a tensor in a number's
    place is refused either way.  In its own process: the extension is blocked before the first import."""
    code = f"""
import sys, ctypes as C
if not {native}:
    sys.modules['paddock_b200._launch'] = None
import numpy as np
from paddock_b200 import KernelPack, LaunchError, Open, formats, pack
assert (pack._launch is not None) == {native}
try:
    KernelPack.load('/nonexistent/pack.so')
    raise SystemExit('loaded')
except Open:
    pass
p = KernelPack.load()
args = lambda k, n, st=0: ('f8row_gemm', 0, 0, 0, 0, 0, k, n, 1)
assert p.call(*args(16, 0)) is None and p.status(*args(16, 0), stream=C.c_void_p(0)) == 0     # no rows: nothing to do
assert p.status(*args(3, 4)) == 1 and p.status(*args(np.uint32(3), 4)) == 1                  # K not a multiple of 16
try:
    p.call(*args(3, 4))
    raise SystemExit('not refused')
except LaunchError as e:
    assert e.status == 1
class Tensor:
    def data_ptr(self): return 16
for bad in (args(Tensor(), 4), args(16, 0)[:-1]):
    for f in (p.call, p.status):
        try:
            f(*bad)
            raise SystemExit('taken')
        except TypeError:
            pass
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=packmod.os.path.dirname(packmod._PKG))
