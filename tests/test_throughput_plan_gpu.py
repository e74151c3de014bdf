"""The throughput plan with several CTAs per row (two CTAs of different calls share an SM): rows whose sample is
misleading, short rows among them, k beyond 2048 and a warm start, against the oracle."""
import numpy as np
import pytest
import torch

from jit_kernel import _native
from jit_kernel.topk_indexer import _status_word, fast_topk_general, fast_topk_v3, fast_topk_v3_warm, kernel_status
from oracle import topk_oracle as orc
from test_select_gpu import _awkward_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _clean_status():
    dev = torch.device("cuda", 0)
    _status_word(dev).zero_()
    yield
    _status_word(dev).zero_()  # (a missed guess is reported there, and is no fault)


@pytest.mark.parametrize("L", [9000, 65537, 131072, 262144])
@pytest.mark.parametrize("rows,ctas", [(15, 2), (8, 4), (4, 8)])
def test_awkward_rows_over_several_ctas(L, rows, ctas):
    s = _awkward_rows(L, seed=L + rows)
    s = torch.stack([s[(3 * i) % 15] for i in range(rows)])
    ln = torch.full((rows,), L, dtype=torch.int32)
    ln[1], ln[2] = L - 3, L // 2 + 1
    ln[3] = 1500  # padded with -1
    sd, ld = s.cuda(), ln.cuda()
    thr = torch.zeros(rows, dtype=torch.int32, device="cuda")
    _native.set_overlap(True)
    try:
        assert _native.plan(rows, L)["cluster_ctas"] == min(ctas, 1 << ((L // 2048).bit_length() - 1))
        torch.cuda.synchronize()
        for _ in range(2):
            got = fast_topk_v3(sd, ld, 2048)
            wide = fast_topk_general(sd, ld, 4096)  # (may start before the call in front of it has ended)
            torch.cuda.synchronize()
            warm = fast_topk_v3_warm(sd, ld, 2048, thr)  # no guess yet, then the thresholds of the call before
            torch.cuda.synchronize()
    finally:
        _native.set_overlap(False)
    for k, out in ((2048, got), (4096, wide), (2048, warm)):
        orc.check_result(s.numpy(), ln.numpy(), out.cpu().numpy(), None, k, None, f"L={L} rows={rows} k={k}")
    assert kernel_status() & ~_native.ST_GUESS_MISSED == 0
    keys = orc.keys_of(s.numpy())
    for b in range(rows):  # a threshold key is the k-th largest, or a lower bound of it
        n = int(ln[b])
        kth = np.sort(keys[b, :n])[-2048] if n > 2048 else 0
        assert int(thr[b]) & 0xFFFFFFFF <= kth
