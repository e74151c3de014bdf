"""Rows with one CTA each (256, 512 and 1024 threads), on every way such a CTA takes: a row held in registers, streamed,
its list spilling, copies of the threshold in any number, rows that go through full histograms; against the oracle."""
import pytest
import torch

from jit_kernel import _native
from jit_kernel.topk_indexer import (_status_word, fast_topk, fast_topk_general, fast_topk_transform_fused, fast_topk_v3,
                                     fast_topk_v3_warm, kernel_status)
from oracle import topk_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _reset():
    _native.set_tuning()
    yield
    _native.set_tuning()
    _status_word(torch.device("cuda", 0)).zero_()  # (a missed guess is reported there, and is no fault)


def _rows(L, seed):
    g = torch.Generator().manual_seed(seed)
    n = lambda: torch.randn(L, generator=g)  # noqa: E731
    pos = torch.arange(L)
    out = [n(), n().abs() + 3, -n().abs() - 1, torch.full((L,), 2.5), n().bfloat16().float()]
    out.append(torch.where(torch.rand(L, generator=g) < 0.7, 0.0, n().exp()))
    for copies in (257, 700, 5000):  # of a value near the threshold
        x = n()
        x[torch.randperm(L, generator=g)[:min(copies, L)]] = x.sort(descending=True).values[min(1900, L - 1)]
        out.append(x)
    out.append(n().sort().values)
    x = n()
    x[L // 3:L // 3 + 2100] += 50  # a window of winners
    out.append(x)
    x = n()
    x[torch.rand(L, generator=g) < 0.3] = float("-inf")
    x[::97] = float("nan")
    out.append(x)
    x = torch.full((L,), float("-inf"))
    x[::5] = n()[::5]
    out.append(x)
    x = torch.zeros(L)
    x[::2] = -0.0
    x[::11] = n()[::11]
    out.append(x)
    out.append(torch.where(pos % 64 < 5, n() + 9, n()))
    return torch.stack(out)


@pytest.mark.parametrize("threads", [256, 512, 1024])
@pytest.mark.parametrize("L", [2049, 4093, 4352, 4609, 8190, 8193, 16384, 20001, 33000, 140003])
def test_every_kind_of_row(threads, L):
    s = _rows(L, seed=L)
    B = s.size(0)
    ln = torch.tensor([max(L - 3 * b, 2049) if b % 3 else L for b in range(B)], dtype=torch.int32)
    ln[4] = 2000
    rs = torch.tensor([min(b % 4, L - 2049) for b in range(B)], dtype=torch.int32)  # every alignment
    sd, ld, rd = s.cuda(), ln.cuda(), rs.cuda()
    _native.set_tuning(cluster_ctas=1, threads=threads)
    got, off = fast_topk_v3(sd, ld, 2048), fast_topk_v3(sd, ld, 2048, rd)
    wide = fast_topk_general(sd, ld, 3000)
    keys = torch.empty(B, 2048, dtype=torch.int32, device="cuda")
    shifted = torch.empty_like(keys)
    fast_topk(sd, shifted, ld, keys=keys, idx_offset=7)
    torch.cuda.synchronize()
    x, n = s.numpy(), ln.numpy()
    orc.check_result(x, n, got.cpu().numpy(), None, 2048, None, f"{threads} L={L}")
    orc.check_result(x, n, off.cpu().numpy(), rs.numpy(), 2048, None, f"row_starts {threads} L={L}")
    orc.check_result(x, n, wide.cpu().numpy(), None, 3000, None, f"k=3000 {threads} L={L}")
    back = torch.where(shifted >= 0, shifted - 7, shifted).cpu().numpy()
    orc.check_result(x, n, back, None, 2048, None, f"offset {threads} L={L}")
    every = orc.keys_of(x)
    got_keys = keys.cpu().numpy().view("uint32")
    for b in range(B):
        if n[b] > 2048:
            assert (got_keys[b] == every[b][back[b]]).all()
    assert kernel_status() == 0


@pytest.mark.parametrize("L", [4096, 9000, 70000])
def test_batches_that_choose_it_themselves(L):
    """More rows than SMs: as the launch plan has it, with a page table, a warm start, 16-bit logits."""
    s = _rows(L, seed=L + 1)
    n = s.size(0)
    x = s.repeat(20, 1)[:290].cuda()
    B = x.size(0)
    ln = torch.full((B,), L, dtype=torch.int32, device="cuda")
    assert _native.plan(B, L)["threads"] == (256 if L <= 4096 else 512)
    table = torch.stack([torch.randperm(L, generator=torch.Generator().manual_seed(i)) for i in range(2)]).int().cuda()
    cu = torch.tensor([0, 150, B], dtype=torch.int32, device="cuda")
    got, paged = fast_topk_v3(x, ln, 2048), fast_topk_transform_fused(x, ln, table, cu, 2048)
    half = fast_topk_general(x.to(torch.bfloat16), ln, 2048)
    thr = torch.zeros(B, dtype=torch.int32, device="cuda")
    warm = [fast_topk_v3_warm(x, ln, 2048, thr, margin=m) for m in (0, 0, 1 << 18)]
    torch.cuda.synchronize()
    assert kernel_status() & ~_native.ST_GUESS_MISSED == 0
    orc.check_result(s.numpy(), ln[:n].cpu().numpy(), got[:n].cpu().numpy(), None, 2048, None, f"L={L}")
    orc.check_result(s.to(torch.bfloat16).float().numpy(), ln[:n].cpu().numpy(), half[:n].cpu().numpy(), None, 2048, None, f"bf16 L={L}")
    want = got[:n].sort(dim=1).values
    for out in (got, *warm):
        assert torch.equal(out.sort(dim=1).values, want.repeat(20, 1)[:B])
    req = (torch.arange(B, device="cuda") >= 150).long()
    assert torch.equal(paged.sort(dim=1).values, table[req].gather(1, got.long()).sort(dim=1).values)
