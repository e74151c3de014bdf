"""Which way rows with one CTA each go where the guess admits many: k beyond 2048, long rows, copies of the threshold. All of
them are finished from the candidates of one filter pass. Counted by the checked build (see test_routes_gpu)."""
import importlib.util
import json
import os
import subprocess
import sys

import pytest

import test_routes_gpu as routes

pytestmark = pytest.mark.gpu

# kind, B, L, k, overlap, warm
CASES = [
    ("normal", 100, 160000, 4096, 0, 0),   # 1024 threads
    ("normal", 100, 220000, 4096, 0, 0),
    ("normal", 80, 512000, 4096, 0, 0),
    ("normal", 64, 262144, 4096, 1, 0),    # 512 threads
    ("normal", 40, 2000000, 2048, 1, 0),
]


# rows of 4,096 and fewer elements, most of them equal: all of a row passes the filter, wherever it starts
SHORT = r"""
import ctypes, json, sys
sys.path[:0] = [REPO, REPO + "/flash-float-jit-kernels_b200"]
import numpy as np
import torch
from jit_kernel import _native
from jit_kernel.topk_indexer import fast_topk_v3
from oracle import topk_oracle as orc
res, B = [], 160
for L, start in json.loads(sys.stdin.read()):
    rng = np.random.default_rng(L + start)
    x = np.where(rng.random((B, L)) < 0.7, 0, np.exp(rng.standard_normal((B, L)))).astype(np.float32)
    wide = torch.zeros(B, L + 9 - L % 4, device="cuda")[:, start:start + L]  # (rows start at `start` in turn with the next three)
    wide.copy_(torch.from_numpy(x))
    ln = np.full(B, L, np.int32)
    assert _native.plan(B, L)["threads"] == 256
    counts = (ctypes.c_uint32 * 3)()
    torch.cuda.synchronize()
    _native.lib().fftopk_checked_routes(counts)
    out = fast_topk_v3(wide, torch.from_numpy(ln).cuda(), 2048)
    torch.cuda.synchronize()
    _native.lib().fftopk_checked_routes(counts)
    orc.check_result(x, ln, out.cpu().numpy(), None, 2048, None, f"L={L} start={start}")
    res.append(list(counts))
print("ROUTES " + json.dumps(res))
"""


def run_checked(child, cases):
    spec = importlib.util.spec_from_file_location("_fftopk_build", routes.REPO / "flash-float-jit-kernels_b200" / "build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    env = dict(os.environ, FFTOPK_LIBRARY=str(mod.build_checked_library()))
    res = subprocess.run([sys.executable, "-c", f"REPO = {str(routes.REPO)!r}\n" + child], cwd=routes.REPO, env=env,
                         capture_output=True, text=True, input=json.dumps(cases))
    assert res.returncode == 0, res.stderr[-3000:]
    return json.loads(res.stdout.split("ROUTES ", 1)[1])


@pytest.mark.timeout(600)
def test_no_row_needs_full_histograms():
    # CTAs a row; rows held, beyond a region, by full histograms
    assert run_checked(routes.CHILD, CASES) == [[1, B, 0, 0] for _, B, *_ in CASES]


@pytest.mark.timeout(600)
def test_a_short_row_fits_whole_wherever_it_starts():
    cases = [(L, start) for L in (4096, 4095, 4093, 2049) for start in (0, 1, 2, 3)]
    assert run_checked(SHORT, cases) == [[160, 0, 0]] * len(cases)
