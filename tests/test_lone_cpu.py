"""CPU tests of the rules a lone CTA works by (csrc/fftopk_decide.h, compiled by g++): the digit of a finish round on
32-bit fields, and the layout of its candidate list."""
import ctypes
import subprocess
from pathlib import Path

import pytest
from hypothesis import given, settings, strategies as st

REPO = Path(__file__).resolve().parent.parent
u32 = ctypes.c_uint32


@pytest.fixture(scope="module")
def dh(tmp_path_factory):
    out = tmp_path_factory.mktemp("lone") / "libdecide.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(REPO / "flash-float-jit-kernels_b200" / "csrc"),
                    "-o", str(out), str(REPO / "tests" / "decide_harness.cpp")], check=True)
    lib = ctypes.CDLL(str(out))
    lib.dh_key_digit.restype, lib.dh_key_digit.argtypes = u32, [u32, u32, u32]
    lib.dh_key_bin_range.argtypes = [u32, u32, u32, u32, ctypes.POINTER(u32), ctypes.POINTER(u32)]
    return lib


word = st.integers(0, (1 << 32) - 1)


@settings(max_examples=500, deadline=None)
@given(a=word, b=word, c=word, d=word, e=word)
def test_key_digit_is_monotone_and_its_bins_tile_the_range(dh, a, b, c, d, e):
    lo, x, y, focus, cap = sorted((a, b, c, d, e))
    bins = dh.dh_finish_bins()
    dx, dy = dh.dh_key_digit(lo, focus, x), dh.dh_key_digit(lo, focus, y)
    assert dh.dh_key_digit(lo, focus, lo) == 0 and dx <= dy < bins
    assert dh.dh_key_digit(lo, focus, focus) < bins - 1 and (cap - focus < bins or dh.dh_key_digit(lo, lo, cap) == bins - 1)
    low, high = u32(), u32()
    for v in (x, y, focus, cap):
        dh.dh_key_bin_range(lo, focus, cap, dh.dh_key_digit(lo, focus, v), ctypes.byref(low), ctypes.byref(high))
        assert lo <= low.value <= v <= high.value <= cap
    if low.value > lo:  # (the bin of cap starts where the one below ends)
        assert dh.dh_key_digit(lo, focus, low.value - 1) == dh.dh_key_digit(lo, focus, low.value) - 1


@pytest.mark.parametrize("threads", [256, 512, 1024])
@pytest.mark.parametrize("list_cap", [32, 48, 2048, 4096, 6144, 9216, 16384])
def test_list_of_a_lone_cta(dh, threads, list_cap):
    seg, spill, warps = dh.dh_lone_segment(list_cap, threads), dh.dh_list_spill(list_cap, 1), threads // 32
    assert 0 < seg <= 32 * dh.dh_lone_regs(threads) or list_cap < 2 * warps
    words = warps * seg + (warps * seg) % 2  # indices, then composites on an 8-byte boundary
    assert dh.dh_lone_list_bytes(list_cap, threads) == 4 * words + 8 * spill <= 8 * list_cap + 8
    assert dh.dh_lone_room(list_cap, threads) == warps * seg + spill >= min(list_cap, 4608)


@pytest.mark.parametrize("first", [0, 1, 2, 3])
def test_a_short_row_fits_whole(dh, first):
    """Rows that get 256 threads (up to 4,352 elements): all of a row may pass the filter. In granules of four of the
    aligned view, of which warp w sees [32 w, 32 w + 32) of every 256, and the two at the ends go to warps 0 and 1."""
    seg, count = dh.dh_lone_segment(4096, 256), [0] * 8
    for i in range(4352):
        g = (i + first) // 4
        whole = g * 4 >= first and g * 4 + 4 <= first + 4352
        count[(g - (first > 0)) % 256 // 32 if whole else (0 if g == 0 else 1)] += 1
    assert sum(max(0, c - seg) for c in count) <= dh.dh_list_spill(4096, 1)
