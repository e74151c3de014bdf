"""CPU test of the rule that allows a call to ask for its rows ahead of time (csrc/fftopk_decide.h, compiled by g++): never for an
address outside the allocation that the rows lie in, whatever their lengths were when the request was sized."""
import ctypes
import subprocess
from pathlib import Path

import pytest
from hypothesis import given, settings, strategies as st

REPO = Path(__file__).resolve().parent.parent
i64, u64 = ctypes.c_int64, ctypes.c_uint64


@pytest.fixture(scope="module")
def inside(tmp_path_factory):
    out = tmp_path_factory.mktemp("prefetch") / "libdecide.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(REPO / "flash-float-jit-kernels_b200" / "csrc"),
                    "-o", str(out), str(REPO / "tests" / "decide_harness.cpp")], check=True)
    fn = ctypes.CDLL(str(out)).dh_rows_inside
    fn.argtypes = [u64, i64, ctypes.c_int32, i64, ctypes.c_int, u64, u64]
    return fn


size = st.one_of(st.integers(0, 300), st.integers(0, 1 << 40), st.integers(0, (1 << 62) - 1))


@settings(max_examples=1000, deadline=None)
@given(base=st.integers(0, 1 << 62), at=size, slack=st.integers(-9, 9), stride=size, B=st.integers(1, (1 << 31) - 1) | st.integers(1, 5),
       L=size, element=st.sampled_from([2, 4]))
def test_exactly_where_all_rows_fit(inside, base, at, slack, stride, B, L, element):
    last = at + ((B - 1) * stride + L) * element  # one past the last byte, from the allocation's first
    for length in {max(last + slack, 0), at, 1 << 30}:
        if length < 1 << 62:
            assert inside(base + at, stride, B, L, element, base, length) == int(last <= length)


def test_rows_whose_storage_ends_with_their_lengths(inside):
    """Eight rows packed one behind the other with a row length L beyond their stride, and a last row that ends with its storage."""
    base, stride, L = 1 << 40, 300000, 400000
    assert not inside(base, stride, 8, L, 4, base, 8 * stride * 4)
    assert inside(base, stride, 8, L, 4, base, (7 * stride + L) * 4)
    assert not inside(base - 16, stride, 1, L, 4, base, 1 << 30) and not inside(base, -stride, 2, L, 4, base, 1 << 30)
