"""Rows that are asked for ahead of the launch they belong to (chains of calls on long rows): the kernel in front may still
be writing them, and their lengths, when that happens."""
import pytest
import torch

from jit_kernel import _native
from jit_kernel.topk_indexer import fast_topk, fast_topk_general, kernel_status
from oracle import topk_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L,k,dtype", [(1, 300001, 2048, torch.float32), (3, 262145, 4096, torch.float32),
                                         (2, 600003, 1024, torch.bfloat16)])
def test_rows_written_just_before(B, L, k, dtype):
    g = torch.Generator().manual_seed(L)
    rows = [torch.randn(B, L, generator=g).to(dtype) for _ in range(4)]
    lens = [torch.randint(L // 2, L + 1, (B,), generator=g, dtype=torch.int32) for _ in range(4)]
    rows_d, lens_d = [r.cuda() for r in rows], [x.cuda() for x in lens]
    x, ln = torch.zeros(B, L, dtype=dtype, device="cuda"), torch.zeros(B, dtype=torch.int32, device="cuda")
    outs = []
    for r, n in zip(rows_d, lens_d):  # one buffer, rewritten between calls that stand in a chain
        x.copy_(r)
        ln.copy_(n)
        for _ in range(2):
            out = fast_topk_general(x, ln, k)
        outs.append(out)
    torch.cuda.synchronize()
    for r, n, out in zip(rows, lens, outs):
        orc.check_result(r.float().numpy(), n.numpy(), out.cpu().numpy(), None, k, None, f"B={B} L={L}")
    assert kernel_status() == 0


def test_lengths_beyond_the_matrix_and_odd_strides():
    """Lengths are clamped before they size a request; rows may start anywhere, the last one at the end of its storage."""
    L = 262200
    store = torch.randn(2 * 263001 + L + 3, device="cuda")
    x = store[3:].as_strided((3, L), (263001, 1))
    ln = torch.tensor([1 << 30, -5, 262199], dtype=torch.int32, device="cuda")
    out = torch.empty(3, 2048, dtype=torch.int32, device="cuda")
    for _ in range(3):
        fast_topk(x, out, ln)
    torch.cuda.synchronize()
    orc.check_result(x.cpu().numpy(), torch.tensor([L, 0, 262199]).numpy(), out.cpu().numpy(), None, 2048, None, "clamped")
    assert _native.plan(3, L)["cluster_ctas"] > 1 and kernel_status() == 0
