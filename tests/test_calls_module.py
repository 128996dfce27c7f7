"""The per-op entry points as an extension module (csrc/calls.c): every argument arrives as it does through ctypes."""

import ctypes
import subprocess
import sys

import numpy as np
import pytest

from yule_b200 import _lib

NAMES = [f"yule_cuda_{n}" for n in ("add", "copy_buffer", "copy_buffer_offset", "copy_from_device", "element_mul", "multihead_attention", "quantized_matmul",
                                    "quantized_matmul_batched", "rms_norm", "rope", "silu")]
pytestmark = pytest.mark.usefixtures("native_libs")


class Whole:
    def __index__(self):
        return 7


def test_every_function_is_one_of_the_library():
    assert sorted(n for n in dir(_lib.calls()) if n.startswith("yule_cuda_")) == NAMES and set(NAMES) <= set(_lib._SIGNATURES)


@pytest.mark.parametrize("name", NAMES)
def test_arguments_as_ctypes_takes_them(name):
    fast, slow = getattr(_lib.calls(), name), getattr(_lib.cuda_lib(), name)
    types = _lib._SIGNATURES[name]
    zeros = [None] + [0.0 if t is _lib.f32 else 0 for t in types[1:]]
    assert fast(*zeros) == slow(*zeros) != 0  # a null context is refused
    for at in range(1, len(types)):
        if types[at] is _lib.vp:
            continue  # (the wrappers pass addresses)
        for value in (True, -1, 2 ** 70, np.int64(5), np.uint32(6), Whole(), 1.5, np.float32(2), "3", b"4", None, [5]):
            args = list(zeros)
            args[at] = value
            got = []
            for f in (fast, slow):
                try:
                    got.append(f(*args))
                except ctypes.ArgumentError:
                    got.append("refused")
            assert got[0] == got[1], (at, value, got)


class Parameter:
    def __init__(self, value):
        self._as_parameter_ = value


class Odd:
    def __index__(self):
        raise ValueError("no number")


@pytest.mark.parametrize("name", NAMES)
def test_arguments_that_only_ctypes_knows(name):
    """Numbers of ctypes' types and objects that stand for another one, in every place, the context's and the host pointer's among them."""
    fast, slow = getattr(_lib.calls(), name), getattr(_lib.cuda_lib(), name)
    types = _lib._SIGNATURES[name]
    zeros = [None] + [0.0 if t is _lib.f32 else 0 for t in types[1:]]
    assert fast(*[t(0) for t in types]) == slow(*zeros) != 0
    taken = 0
    for at in range(len(types)):
        for value in (ctypes.c_uint32(5), ctypes.c_uint64(5), ctypes.c_int32(5), ctypes.c_size_t(5), ctypes.c_float(2), ctypes.c_void_p(0), Parameter(0), Parameter(types[at](0)), Parameter(Parameter(0)),
                      Parameter("x"), Odd()):
            args = list(zeros)
            args[at] = value
            if at == 0 and (not isinstance(value, (ctypes.c_void_p, Parameter)) or getattr(value, "_as_parameter_", 0) == "x"):
                continue  # (an address that is none, or a text's)
            got = []
            for f in (fast, slow):
                try:
                    got.append(f(*args))
                except ctypes.ArgumentError:
                    got.append("refused")
            assert got[0] == got[1], (at, value, got)
            taken += got[0] != "refused"
    assert taken >= 2 * len(types)


@pytest.mark.parametrize("name", NAMES)
def test_the_number_of_arguments(name):
    with pytest.raises(TypeError):
        getattr(_lib.calls(), name)(None)


def test_values_arrive(tmp_path):
    """Against a library of the same names that writes down what it is given."""
    src, so = tmp_path / "fake.c", tmp_path / "libyule_cuda.so"
    body = "#include <stdint.h>\n#include <stddef.h>\n#include <stdio.h>\n"
    for name in NAMES:
        types = _lib._SIGNATURES[name]
        c = {_lib.vp: "void *", _lib.u64: "uint64_t", _lib.u32: "uint32_t", _lib.f32: "float", _lib.size_t: "size_t"}
        args = ", ".join(f"{c[t]} a{i}" for i, t in enumerate(types))
        shown = "".join("%g " if t is _lib.f32 else "%llu " for t in types)
        values = ", ".join(f"a{i}" if t is _lib.f32 else f"(unsigned long long)(uintptr_t)a{i}" for i, t in enumerate(types))
        body += f'int32_t {name}({args}) {{ printf("{shown}\\n", {values}); fflush(stdout); return {len(types)}; }}\n'
    src.write_text(body)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)])
    from yule_b200 import build
    script = ["import importlib.util, sys", f"spec = importlib.util.spec_from_file_location('_calls', {build.CALLS_SO!r})",
              "m = importlib.util.module_from_spec(spec)", "spec.loader.exec_module(m)"]
    want = []
    for name in NAMES:
        types = _lib._SIGNATURES[name]
        args, shown = [], []
        for i, t in enumerate(types):
            v = 0.5 + i if t is _lib.f32 else (1 << 40) + i if t in (_lib.vp, _lib.u64, _lib.size_t) else (1 << 33) + 3000000000 + i
            args.append(v)
            shown.append("%g" % v if t is _lib.f32 else str(v % 2 ** 32 if t is _lib.u32 else v))
        script.append(f"assert m.{name}(*{tuple(args)!r}) == {len(types)}")
        want.append(" ".join(shown) + " ")
    out = subprocess.run([sys.executable, "-c", "\n".join(script)], env={"LD_PRELOAD": str(so), "PATH": "/usr/bin"}, stdout=subprocess.PIPE, text=True, check=True).stdout
    assert out.splitlines() == want
