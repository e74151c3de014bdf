"""CPU tests of the digit the sample histogram is built on (csrc/fftopk_decide.h, compiled by g++): it is
monotone in the radix key, its bins tile the key space without gaps, and a guess made on any bin admits
every element of that bin and above."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import topk_oracle as orc

REPO = Path(__file__).resolve().parent.parent
BINS = 4096


@pytest.fixture(scope="module")
def dh(tmp_path_factory):
    out = tmp_path_factory.mktemp("digit") / "libdecide.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(REPO / "flash-float-jit-kernels_b200" / "csrc"),
                    "-o", str(out), str(REPO / "tests" / "decide_harness.cpp")], check=True)
    lib = ctypes.CDLL(str(out))
    for name in ("dh_sample_digit", "dh_sample_digit_low", "dh_sample_digit_high"):
        getattr(lib, name).restype = ctypes.c_uint32
        getattr(lib, name).argtypes = [ctypes.c_uint32]
    lib.dh_sample_admits_too_much.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_float, ctypes.c_uint32]
    return lib


def test_bins_tile_the_key_space(dh):
    lows = [dh.dh_sample_digit_low(b) for b in range(BINS)]
    assert lows[0] == 0 and all(a < b for a, b in zip(lows, lows[1:]))
    assert [dh.dh_sample_digit_high(b) for b in range(BINS)] == [v - 1 for v in lows[1:]] + [0xffffffff]


def _values():
    rng = np.random.default_rng(3)
    bits = rng.integers(0, 1 << 32, 4000, dtype=np.uint64).astype(np.uint32)
    edges = [np.float32(s * 2.0 ** e) for e in (-149, -126, -17, -16, -15, 0, 15, 16, 17, 127) for s in (-1, 1)]
    near = np.concatenate([np.nextafter(np.float32(v), np.float32(d)).reshape(1) for v in edges for d in (-np.inf, np.inf)])
    some = np.array([0.0, np.inf, -np.inf, 18.4, -18.4], np.float32)
    v = np.concatenate([bits.view(np.float32), np.array(edges, np.float32), near, some, rng.standard_normal(2000).astype(np.float32)])
    return v[~np.isnan(v) & (v.view(np.uint32) != 0x80000000)]  # (where NaN and -0 fall is of no concern)


def test_digit_is_monotone_and_its_bin_holds_the_key(dh):
    v = np.sort(_values())
    digits = [dh.dh_sample_digit(int(b)) for b in v.view(np.uint32)]
    assert all(a <= b for a, b in zip(digits, digits[1:]))
    for d, key in zip(digits, orc.keys_of(v)):
        assert dh.dh_sample_digit_low(d) <= int(key) <= dh.dh_sample_digit_high(d)


@pytest.mark.parametrize("length", [8193, 131072, 1 << 20])
def test_only_hopeless_guesses_are_given_up(dh, length):
    n_s, room = (16384 if length > 262144 else 8192), 16384
    m = 2048 * n_s / length
    rank = int(m + 5 * m ** 0.5 + 14)  # what a row without crowded bins admits, bin rounding included
    assert not dh.dh_sample_admits_too_much(rank + rank // 4, n_s, length, room)
    assert dh.dh_sample_admits_too_much(n_s, n_s, 4 * room, room)
