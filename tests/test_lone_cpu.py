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
@pytest.mark.parametrize("list_cap", [32, 48, 2048, 2560, 6144, 9216, 16384])
def test_list_of_a_lone_cta(dh, threads, list_cap):
    seg, warps = dh.dh_lone_segment(list_cap, threads), threads // 32
    assert 0 < seg <= 32 * dh.dh_lone_regs(threads)
    assert dh.dh_lone_room(list_cap, threads) == warps * seg <= 2 * list_cap


def test_a_short_row_fits_whole(dh):
    """Rows that get 256 threads (up to 4,096 elements): all of a row may pass the filter. In granules of four, of which
    warp w sees [32 w, 32 w + 32) of every 256."""
    count = [sum(1 for g in range(1024) if g % 256 // 32 == w) * 4 for w in range(8)]
    assert max(count) <= dh.dh_lone_segment(2560, 256)


@pytest.mark.parametrize("threads,k,length", [(1024, 4096, n) for n in (131072, 220000, 1 << 19, 1 << 20)]
                         + [(512, 4096, n) for n in (65536, 131072, 262144)]
                         + [(512, 2048, n) for n in (262144, 1 << 20, 2000000)] + [(1024, 2048, 2000000)])
def test_a_warp_holds_its_share_of_what_a_guess_admits(dh, threads, k, length):
    """Rows of independent values: a guess made on rank r of n samples admits r L / n elements, give or take its square root
    in samples; they fall on the warps at random. Three and a half deviations more than a warp's share fit its segment."""
    dh.dh_sample_lower_rank.restype, dh.dh_sample_lower_rank.argtypes = u32, [u32, u32, ctypes.c_float]
    n = 8192 << dh.dh_sample_log_batches(length, u32(k))
    rank, warps = dh.dh_sample_lower_rank(k, n, length), threads // 32
    share, each = rank * length / n / warps, length / n / warps
    deviation = (rank * each ** 2 + share) ** 0.5
    assert share + 3.5 * deviation <= dh.dh_lone_segment(6144, threads)


@pytest.mark.parametrize("start", [0, 1, 2, 3])
def test_a_short_row_fits_whole_wherever_it_starts(dh, start):
    """... and rows that are not 16-byte aligned: inner granule i of a row lies with warp i % 256 // 32, the two that its ends
    cut through with the edge warp."""
    for length in range(4096, 4064, -1):
        first = (4 - start) % 4
        inner, last = divmod(length - first, 4)
        count = [sum(4 for i in range(inner) if i % 256 // 32 == w) for w in range(8)]
        count[dh.dh_lone_edge_warp(256)] += first + last
        assert sum(count) == length and max(count) <= dh.dh_lone_segment(2560, 256)
