"""The automatic counter choice of a counting wave (csrc/wave_route.h), compiled by itself: the tensor
tiles or the CUDA-core tiles, whichever the measured shapes are faster with, and never far from
the lines of the tuning table."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import tensorfim_b200 as tf

CSRC = os.path.join(os.path.dirname(os.path.abspath(tf.__file__)), "csrc")


@pytest.fixture(scope="module")
def route(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("route")
    src, so = d / "route.cpp", d / "route.so"
    src.write_text('#include "wave_route.h"\nextern "C" int on_tensor(long long b, long long d, long long w, float e, int r, int c)'
                   '{ return tfim::wave_on_tensor(b, d, w, e, r, c); }\n'
                   'extern "C" float empty_pieces(const int* s, long long n, long long t) { return tfim::empty_pieces(s, n, t); }\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.on_tensor.argtypes = [ctypes.c_longlong] * 3 + [ctypes.c_float] + [ctypes.c_int] * 2
    lib.empty_pieces.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_longlong]
    lib.empty_pieces.restype = ctypes.c_float

    def supports(data, d, tx):
        if data == "dense":
            return np.random.Generator(np.random.PCG64(5)).integers(1, 16, size=d) * (tx / 16)
        return np.maximum(0.1 * np.arange(1, d + 1) ** -0.9, 0.0005) * tx

    def choose(data, b, d, tx, min_rows=3, min_cols=1):
        s = supports(data, d, tx).astype(np.int32)
        words = (tx + 2047) // 2048 * 64
        return bool(lib.on_tensor(b, d, words, lib.empty_pieces(s.ctypes.data, d, tx), min_rows, min_cols))

    return choose


# microseconds per call: CUDA-core tiles, tensor tiles
@pytest.mark.parametrize("data,d,tx,b,cuda,tensor", [
    ("longtail", 6162, 500_000, 1, 46, 252), ("longtail", 6162, 200_000, 1, 45, 134), ("longtail", 2000, 500_000, 1, 37, 111),
    ("longtail", 6162, 50_000, 1, 43, 69), ("longtail", 6162, 500_000, 2, 156, 250), ("longtail", 4000, 262_144, 2, 98, 125),
    ("longtail", 6162, 1_000_000, 3, 398, 444), ("longtail", 6162, 130_000, 4, 77, 107), ("dense", 16, 1 << 23, 3, 60, 91),
    ("dense", 8, 1 << 23, 4, 50, 83), ("dense", 69, 10_000, 1, 56, 42), ("dense", 69, 1 << 18, 1, 71, 39),
    ("dense", 1024, 1 << 18, 1, 72, 58), ("dense", 271, 1_000_000, 3, 92, 63), ("dense", 1024, 4_000_000, 3, 410, 303),
    ("longtail", 2000, 500_000, 3, 142, 110), ("longtail", 1200, 130_000, 2, 82, 51), ("longtail", 6162, 1_000_000, 16, 608, 447)])
def test_measured_shapes(route, data, d, tx, b, cuda, tensor):
    assert route(data, b, d, tx) == (tensor < cuda)


def test_lines_of_the_table_hold(route):
    """A raised or lowered line moves the choice with it, for short and for long rows."""
    for tx in (1_000, 10_000, 1 << 23):
        for data in ("dense", "longtail"):
            for line in (1, 3, 64, 10_000):
                for d in (1, 16, 700):
                    assert route(data, line + 5, d, tx, line)
                    assert line <= 3 or not route(data, line - 3, d, tx, line)
                    assert not route(data, line + 5, d, tx, line, d + 1)
    assert not any(route("dense", b, 69, 10_000, 0x7fffffff) for b in (1, 2, 4096))
