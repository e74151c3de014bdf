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


@pytest.mark.timeout(600)
def test_no_row_needs_full_histograms():
    spec = importlib.util.spec_from_file_location("_fftopk_build", routes.REPO / "flash-float-jit-kernels_b200" / "build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    env = dict(os.environ, FFTOPK_LIBRARY=str(mod.build_checked_library()))
    res = subprocess.run([sys.executable, "-c", f"REPO = {str(routes.REPO)!r}\n" + routes.CHILD], cwd=routes.REPO, env=env,
                         capture_output=True, text=True, input=json.dumps(CASES))
    assert res.returncode == 0, res.stderr[-3000:]
    got = json.loads(res.stdout.split("ROUTES ", 1)[1])
    assert got == [[1, B, 0, 0] for _, B, *_ in CASES]  # CTAs a row; rows held, beyond a region, by full histograms
