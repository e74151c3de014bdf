"""Which way rows go through the selector: finished from the candidates of one filter pass, with some of them
beyond their CTA's part of the gather buffer, or by full histograms. Every way gives the same result (checked
against the oracle here too); the point is that rows which the filter pass is meant for take it, on the
launch plans that the sizes get.

The checked build counts the ways (fftopk_checked_routes). It runs in a child process because the library is
chosen when the package is first imported."""
import importlib.util
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parent.parent

CHILD = r"""
import ctypes, json, sys
sys.path[:0] = [REPO, REPO + "/flash-float-jit-kernels_b200"]
import numpy as np
import torch
from jit_kernel import _native
from jit_kernel.topk_indexer import fast_topk_general, fast_topk_v3_warm, kernel_status
from oracle import topk_oracle as orc


def rows(kind, B, L):
    rng = np.random.default_rng(B * 1000 + L)
    x = rng.standard_normal((B, L)).astype(np.float32)
    if kind == "recent":        # the newest 6000 keys stand out: the winners are all in the last shard
        x[:, -6000:] += 6
    elif kind == "straddling":  # ... or in two: a window around a shard boundary
        x[:, L // 2 - 3000:L // 2 + 3000] += 6
    elif kind == "window":      # 2048 consecutive winners
        for b in range(B):
            o = int(rng.integers(0, L - 2048))
            x[b, o:o + 2048] += 8
    elif kind == "equal":
        x[:] = 3.25
    elif kind == "negative zeros":
        u = rng.random((B, L))
        x = np.where(u < 0.1, np.float32(-0.0), np.where(u > 0.995, np.float32(1.0), -np.abs(x) - 0.1)).astype(np.float32)
    return x


def routes():
    out = (ctypes.c_uint32 * 3)()
    assert _native.lib().fftopk_checked_routes(out) == 0
    return list(out)


res = []
for kind, B, L, k, overlap, warm in json.loads(sys.stdin.read()):
    x = rows(kind, B, L)
    ln = np.full(B, L, np.int32)
    xd, ld = torch.from_numpy(x).cuda(), torch.from_numpy(ln).cuda()
    thr = torch.zeros(B, dtype=torch.int32, device="cuda")
    if warm:
        fast_topk_v3_warm(xd, ld - 1, k, thr)
    _native.set_overlap(bool(overlap))
    cluster = _native.plan(B, L)["cluster_ctas"]
    torch.cuda.synchronize()
    routes()
    out = fast_topk_v3_warm(xd, ld, k, thr, margin=1 << 18) if warm else fast_topk_general(xd, ld, k)
    torch.cuda.synchronize()
    _native.set_overlap(False)
    orc.check_result(x, ln, out.cpu().numpy(), None, k, None, f"{kind} B={B} L={L}")
    assert kernel_status() == 0, f"{kind} B={B} L={L}: status {kernel_status():#x}"
    res.append([cluster] + routes())
print("ROUTES " + json.dumps(res))
"""


# kind, B, L, k, overlap, warm  ->  CTAs per row, every row by full histograms?, candidates beyond a region?
# (None: either)
CASES = {
    "plain, one row": (("normal", 1, 98305, 2048, 0, 0), 16, False, False),
    "plain, throughput plan, 2 CTAs a row": (("normal", 16, 131072, 2048, 1, 0), 2, False, False),
    "plain, throughput plan, 4 CTAs a row": (("normal", 8, 131072, 2048, 1, 0), 4, False, None),
    "k = 4096, throughput plan": (("normal", 8, 65536, 4096, 1, 0), 4, False, True),
    "window of winners": (("window", 4, 98305, 2048, 0, 0), 16, False, True),
    "window of winners, throughput plan": (("window", 64, 98305, 2048, 1, 0), 1, False, False),
    "recent keys": (("recent", 1, 1 << 20, 2048, 0, 0), 16, False, True),
    "recent keys, 8 CTAs a row": (("recent", 8, 200000, 2048, 0, 0), 8, False, True),
    "recent keys, throughput plan, 2 CTAs a row": (("recent", 16, 40000, 2048, 1, 0), 2, False, True),
    "recent keys, throughput plan, 8 CTAs a row": (("recent", 4, 65536, 2048, 1, 0), 8, False, True),
    "recent keys, throughput plan, warm": (("recent", 4, 65536, 2048, 1, 1), 8, False, True),
    "keys around a shard boundary": (("straddling", 4, 131072, 2048, 1, 0), 8, False, True),
    "4M elements, k = 4096": (("normal", 1, (1 << 22) + 3, 4096, 0, 0), 16, False, True),
    "12M elements": (("normal", 1, 12 << 20, 2048, 0, 0), 16, False, None),
    "copies of -0 at the threshold": (("negative zeros", 2, 131072, 2048, 0, 0), 16, False, True),
    "all equal": (("equal", 2, 65536, 2048, 0, 0), 16, True, False),
}


@pytest.mark.timeout(600)
def test_rows_take_the_way_they_are_meant_for():
    spec = importlib.util.spec_from_file_location("_fftopk_build", REPO / "flash-float-jit-kernels_b200" / "build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    env = dict(os.environ, FFTOPK_LIBRARY=str(mod.build_checked_library()))
    res = subprocess.run([sys.executable, "-c", f"REPO = {str(REPO)!r}\n" + CHILD], cwd=REPO, env=env, capture_output=True,
                         text=True, input=json.dumps([c[0] for c in CASES.values()]))
    assert res.returncode == 0, res.stderr[-3000:]
    got = json.loads(res.stdout.split("ROUTES ", 1)[1])
    wrong = []
    for (name, (args, cluster, full, beyond)), (c, held, extra, by_histograms) in zip(CASES.items(), got):
        rows = args[1]
        want = (cluster, 0 if full else rows, extra if beyond is None else rows if beyond else 0, rows if full else 0)
        if (c, held, extra, by_histograms) != want:
            wrong.append(f"{name}: (CTAs, held, beyond a region, full histograms) {(c, held, extra, by_histograms)}, expected {want}")
    assert not wrong, "\n".join(wrong)
