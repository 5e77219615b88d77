"""The native launch path of the binding: every argument of every entry point's signature reaches the C function."""
import ctypes as C
import subprocess

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
