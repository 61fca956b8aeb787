"""The callables that launchers are called through, against ctypes: every kind of argument in every place.  No GPU."""
import ctypes
import random
import subprocess
from ctypes import c_double, c_float, c_int, c_longlong, c_ulonglong, c_void_p

import numpy as np
import pytest
import torch

from lgml_b200 import csrc, host

C_NAMES = {c_void_p: "void *", c_int: "int", c_longlong: "long long", c_ulonglong: "unsigned long long", c_float: "float", c_double: "double"}


def signatures():
    rng = random.Random(5)
    yield []
    yield [c_float]
    yield [c_void_p, c_int, c_void_p, c_void_p, c_int, c_int, c_float, c_float, c_void_p]
    yield [c_double] * 8 + [c_int] * 40
    for n in (3, 7, 8, 15, 22, 31, 44):
        kinds = [c_void_p, c_int, c_longlong, c_ulonglong] * 5 + [c_float, c_double]
        got = [rng.choice(kinds) for _ in range(n)]
        while not n - 40 <= sum(t in (c_float, c_double) for t in got) <= 8:
            got = [rng.choice(kinds) for _ in range(n)]
        yield got


def test_callers_pass_what_ctypes_passes(tmp_path):
    sigs = list(signatures())
    lines = ["#include <string.h>", "static unsigned long long h;", "static void in(const void *p, int n) { for (int i = 0; i < n; ++i) h = h * 1099511628211ULL + ((const unsigned char *)p)[i]; }"]
    for i, sig in enumerate(sigs):
        args = ", ".join(f"{C_NAMES[t]} a{j}" for j, t in enumerate(sig)) or "void"
        body = " ".join(f"in(&a{j}, sizeof(a{j}));" for j in range(len(sig)))
        lines.append(f"int f{i}({args}) {{ h = 7; {body} return (int)(h ^ (h >> 32)); }}")
    (tmp_path / "f.c").write_text("\n".join(lines))
    subprocess.run([csrc.find_cc(), "-O2", "-shared", "-fPIC", str(tmp_path / "f.c"), "-o", str(tmp_path / "f.so")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "f.so"))
    rng = random.Random(9)
    for i, sig in enumerate(sigs):
        fn = getattr(lib, f"f{i}")
        fn.argtypes, fn.restype = sig, c_int
        fast = host.caller(fn)
        assert fast is not fn
        for _ in range(20):
            args = []
            for t in sig:
                if t is c_void_p:
                    args.append(rng.choice([None, 0, rng.randrange(1 << 47)]))
                elif t in (c_float, c_double):
                    args.append(rng.choice([rng.uniform(-1e9, 1e9), -1.0, 0, 3, float("inf")]))
                elif t is c_int:
                    args.append(rng.choice([-1, True, rng.randrange(-2 ** 31, 2 ** 31)]))
                else:
                    args.append(rng.choice([-1 if t is c_longlong else 2 ** 64 - 1, rng.randrange(2 ** 63)]))
            assert fast(*args) == fn(*args)
        if sig and sig[0] is c_void_p:                       # what is no number goes through ctypes, and so do its errors
            assert fast(ctypes.c_void_p(77), *args[1:]) == fast(77, *args[1:])
            with pytest.raises(ctypes.ArgumentError):
                fast(object(), *args[1:])
        if sig:
            with pytest.raises(TypeError):                   # too few
                fast(*args[:-1])


class Index:
    def __index__(self):
        return 7


class Float:
    def __float__(self):
        return 7.0


@pytest.mark.parametrize("name,kind", [("f", c_int), ("g", c_longlong), ("u", c_ulonglong), ("h", c_float), ("d", c_double), ("p", c_void_p)])
def test_callers_take_and_refuse_what_ctypes_does(tmp_path, name, kind):
    """Every sort of value in the place of every kind: the same result, or the same error."""
    (tmp_path / "f.c").write_text("int f(int a) { return a; } int g(long long a) { return (int)(a ^ a >> 32); } int u(unsigned long long a) { return (int)(a ^ a >> 32); }\n"
                                  "int h(float a) { return (int)a; } int d(double a) { return (int)a; } int p(void *a) { return (int)(long)a; }\n")
    subprocess.run([csrc.find_cc(), "-O2", "-shared", "-fPIC", str(tmp_path / "f.c"), "-o", str(tmp_path / "f.so")], check=True)
    fn = getattr(ctypes.CDLL(str(tmp_path / "f.so")), name)
    fn.argtypes, fn.restype = [kind], c_int
    fast = host.caller(fn)
    assert fast is not fn

    def tried(call, value):
        try:
            return call(value)
        except Exception as e:
            return type(e)

    for value in (None, 5, True, -1, 2 ** 31, 2 ** 32 + 5, 2 ** 63 - 1, 2 ** 63, 2 ** 64 - 1, -2 ** 63, 2.5, -1.0, "a", Index(), Float(), np.int64(5), np.int32(-1),
                  np.float32(2.5), np.float64(2.5), np.bool_(True), torch.tensor(5), torch.tensor(2.5), c_int(5), c_void_p(5), c_float(1.5), object()):
        assert tried(fast, value) == tried(fn, value), (name, value)


def test_other_signatures_stay_with_ctypes():
    fn = ctypes.CFUNCTYPE(c_int, ctypes.c_char_p)(lambda s: 3)
    fn.argtypes = [ctypes.c_char_p]
    assert host.caller(fn) is fn
    many = ctypes.CFUNCTYPE(c_int, *[c_float] * 9)(lambda *a: 3)
    many.argtypes = [c_float] * 9
    assert host.caller(many) is many
