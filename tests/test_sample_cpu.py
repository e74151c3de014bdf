"""CPU tests of where the selector's sample of a row lies and what a guess made on it admits
(csrc/fftopk_decide.h, compiled by g++)."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

REPO = Path(__file__).resolve().parent.parent
K = 2048
u32, i32, f32 = ctypes.c_uint32, ctypes.c_int, ctypes.c_float


@pytest.fixture(scope="module")
def dh(tmp_path_factory):
    out = tmp_path_factory.mktemp("sample") / "libdecide.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(REPO / "flash-float-jit-kernels_b200" / "csrc"),
                    "-o", str(out), str(REPO / "tests" / "decide_harness.cpp")], check=True)
    lib = ctypes.CDLL(str(out))
    lib.dh_sample_piece_start.restype, lib.dh_sample_piece_start.argtypes = u32, [u32, u32, i32, u32]
    lib.dh_sample_log_batches.argtypes = [i32, u32]
    lib.dh_sample_lower_rank.restype, lib.dh_sample_lower_rank.argtypes = u32, [u32, u32, f32]
    return lib


def sample_pieces(dh, length, n_s, off=0):
    """Row indices of the sample, one line per piece of consecutive granules (row aligned to a granule)."""
    size = dh.dh_sample_piece()
    pieces = n_s // (4 * size)
    first = np.array([dh.dh_sample_piece_start(length // 4, i, pieces.bit_length() - 1, off) for i in range(pieces)], np.int64)
    return 4 * first[:, None] + np.arange(4 * size)[None, :]


LENGTHS = [8 * 1024 + 36, 20000, 32768, 98304, 98308, 131072, 200000, 262144]


@pytest.mark.parametrize("length", LENGTHS + [(1 << 26) + 4, (1 << 31) - 64])
def test_pieces_lie_inside_the_row_one_per_stretch(dh, length):
    size, gi = dh.dh_sample_piece(), length // 4
    for off in range(size):
        pos = sample_pieces(dh, length, 8192, off)
        first, n = pos[:, 0] // 4, len(pos)
        assert np.all((first[1:] + off) % size == 0) and first[0] >= 0 and pos[-1, -1] < 4 * gi
        assert np.diff(first)[1:].min() >= size and first[1] > first[0]
        # piece i in the first four lines of stretch i of n, but for the rounding
        at = first - np.arange(n) * (gi / n)
        assert at.min() >= -(size + 1) and at.max() <= min(3 * size, gi / n - size)


@pytest.mark.parametrize("length", LENGTHS)
def test_a_window_of_winners_does_not_pass_for_the_rank(dh, length):
    """k consecutive winners anywhere in the row: fewer of them are sampled than the rank the guess is made
    on, so the guess lies below all of them and at least k elements pass."""
    hit = np.zeros(length + 1, np.int64)
    hit[sample_pieces(dh, length, 8192).reshape(-1) + 1] = 1
    before = np.cumsum(hit)
    inside = before[K:] - before[:-K]  # sample elements in [o, o + K) for every offset o
    assert inside.max() < dh.dh_sample_lower_rank(K, 8192, length)


def test_a_period_is_seen_at_every_phase(dh):
    """Rows that repeat with a period of up to 128 elements, as with one value per position in a page of keys: the sample
    holds the same share of every position."""
    for length, n_s in ((32768, 4096), (131072, 8192), (1 << 20, 16384)):
        pos = sample_pieces(dh, length, n_s).reshape(-1)
        for period in (16, 64, 128):
            seen = np.bincount(pos % period, minlength=period)
            assert seen.min() == seen.max(), (length, period, seen)


@pytest.mark.parametrize("reach", [64, 256])
@pytest.mark.parametrize("share", [0.5, 0.9])
def test_smooth_rows_are_guessed_like_others(dh, reach, share):
    """Rows of which a share of the variance varies smoothly over `reach` positions (noise through a triangular
    window): the guess admits at least k in most of 150 rows (a row it does not hold for takes a longer way;
    with slabs of 128 consecutive elements up to 25 % fell short)."""
    rng = np.random.default_rng(reach)
    length, short, rows = 98304, 0, 150
    pos, rank = sample_pieces(dh, length, 8192).reshape(-1), dh.dh_sample_lower_rank(K, 8192, length)
    for _ in range(rows):
        c = rng.standard_normal(length + 2 * reach)
        for _ in range(2):
            c = np.cumsum(c)
            c = c[reach:] - c[:-reach]
        smooth = c[:length]
        row = (share ** 0.5 * (smooth - smooth.mean()) / smooth.std() + (1 - share) ** 0.5 * rng.standard_normal(length)).astype(np.float32)
        sample = row[pos]
        guess = np.partition(sample, sample.size - rank)[sample.size - rank]
        short += int((row >= guess).sum() < K)
    assert short <= 0.1 * rows, f"{short} of {rows} rows"


@pytest.mark.parametrize("k", [1, 512, 2048, 4096])
def test_long_rows_leave_room_for_what_the_guess_admits(dh, k):
    """The number of elements expected to pass stays well below what the gather buffer of a cluster holds
    (16384) for rows of any length, and the sample a small part of the row."""
    for length in [8193, 98304, 262144, 262145] + [n + d for n in (1 << e for e in range(19, 31)) for d in (0, 1)] + [(1 << 31) - 9]:
        n_s = 8192 << dh.dh_sample_log_batches(length, k)
        expected = dh.dh_sample_lower_rank(k, n_s, length) * length / n_s
        assert expected <= (9300 if k <= 2048 else 9800), (length, n_s, expected)
        assert n_s <= 8192 or n_s * 16 < length


@pytest.mark.parametrize("ctas", [2, 4, 8, 16])
@pytest.mark.parametrize("cand_cap,list_cap", [(16384, 6144), (6144, 3072)])  # latency plan, throughput plan
def test_the_gather_buffer_takes_what_one_shard_or_two_hold(dh, ctas, cand_cap, list_cap):
    """All candidates in one CTA's shard: as many as its list holds. In two: what the guess is expected to admit of
    rows of up to 1M elements (a cluster by itself) or 256K (sharing its SMs with other calls)."""
    region = dh.dh_gather_region(cand_cap, list_cap, ctas)
    behind = cand_cap - ctas * region
    assert region > 0 and behind > 0
    assert region + behind >= list_cap
    length, n_s = (1 << 20, 16384) if cand_cap == 16384 else (262144, 8192)
    assert 2 * region + behind >= min(1.1 * dh.dh_sample_lower_rank(K, n_s, length) * length / n_s, 2 * list_cap)


@pytest.mark.parametrize("ctas", [2, 4, 8, 16])
def test_regions_fit_buffers_of_any_size(dh, ctas):
    for cand_cap in (32, 48, 256, 2048, 6144, 16384):
        for list_cap in (32, 512, 6144, 16384):
            region = dh.dh_gather_region(cand_cap, list_cap, ctas)
            assert 0 <= region and ctas * region <= cand_cap
