"""The package imports, and finds device and stream, with a torch that has none of the private CUDA names."""
import subprocess
import sys
from pathlib import Path

REPO = Path(__file__).resolve().parent.parent
CHILD = r"""
import sys
sys.path.insert(0, sys.argv[1])
import torch
for name in ("_cuda_getDevice", "_cuda_getCurrentRawStream"):
    if hasattr(torch._C, name):
        delattr(torch._C, name)
torch.cuda.current_device = lambda: 3
from jit_kernel import indexer, topk_indexer
torch.cuda.current_stream = lambda device: type("Stream", (), {"cuda_stream": 40 + device})
assert topk_indexer._current_device() == 3 and topk_indexer._current_stream(2) == 42
"""


def test_a_torch_without_the_private_names():
    res = subprocess.run([sys.executable, "-c", CHILD, str(REPO / "flash-float-jit-kernels_b200")], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
