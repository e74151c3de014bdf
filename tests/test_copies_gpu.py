"""Thousands of copies of two neighbouring values at the threshold, with several CTAs per row: the guess is one of the values
(a third look at the sample tells them apart), and the k-th largest element is a copy of it, or a larger one after all."""
import numpy as np
import pytest
import torch

from jit_kernel import _native
from jit_kernel.topk_indexer import _status_word, fast_topk_general, fast_topk_v3_warm, kernel_status
from oracle import topk_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _reset():
    yield
    _native.set_tuning()
    _native.set_overlap(False)
    _status_word(torch.device("cuda", 0)).zero_()


def rows(L, aboves, copies, seed=0):
    rng = np.random.default_rng(seed)
    out = np.empty((len(aboves), L), np.float32)
    for x, above in zip(out, aboves):
        x[:] = -rng.random(L) - 0.1
        at = rng.permutation(L)
        x[at[:above]] = 2 + rng.random(above)
        x[at[above:above + copies]] = np.float32(1.005)
        x[at[above + copies:above + 2 * copies]] = 1.0
    return out


PLANS = {"8 CTAs, overlapping": (True, {}), "16 CTAs": (False, {}), "8 CTAs of 1024": (False, dict(cluster_ctas=8, threads=1024)),
         "2 CTAs of 256": (False, dict(cluster_ctas=2, threads=256, cand_cap=6144)), "2 CTAs, overlapping": (True, dict(cluster_ctas=2))}


@pytest.mark.parametrize("plan", PLANS)
def test_threshold_is_a_copy_or_lies_above(plan):
    L, k = 131073, 1024
    x = rows(L, [1023, 1024, 1100, 900], 2500)
    ln = np.full(4, L, np.int32)
    overlap, tuning = PLANS[plan]
    _native.set_overlap(overlap)
    _native.set_tuning(**tuning)
    xd, ld = torch.from_numpy(x).cuda(), torch.from_numpy(ln).cuda()
    wide, half = fast_topk_general(xd, ld, k), fast_topk_general(xd.to(torch.bfloat16), ld, k)
    torch.cuda.synchronize()
    orc.check_result(x, ln, wide.cpu().numpy(), None, k, None, plan)
    orc.check_result(xd.to(torch.bfloat16).float().cpu().numpy(), ln, half.cpu().numpy(), None, k, None, f"bf16 {plan}")
    assert kernel_status() == 0


@pytest.mark.parametrize("threads", [512, 1024])
def test_the_same_for_a_warm_start(threads):
    L, k = 200001, 2048
    x = rows(L, [2047, 2048, 2100, 1900], 4500, seed=1)
    ln = np.full(4, L, np.int32)
    _native.set_tuning(cluster_ctas=8, threads=threads)
    xd, ld, thr = torch.from_numpy(x).cuda(), torch.from_numpy(ln).cuda(), torch.zeros(4, dtype=torch.int32, device="cuda")
    want = np.array([np.sort(orc.keys_of(r))[-k] for r in x], np.uint32)
    for step in range(3):
        out = fast_topk_v3_warm(xd, ld, k, thr)
        torch.cuda.synchronize()
        orc.check_result(x, ln, out.cpu().numpy(), None, k, None, f"step {step}")
        got = thr.cpu().numpy().view(np.uint32)
        assert np.all(got <= want) and (step == 0 or np.array_equal(got, want))
    assert kernel_status() == 0
