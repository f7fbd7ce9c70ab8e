"""The one-launch selection at the edges of its tiles: one CTA or up to eight that hand each other their counts, 128-row
groups cut off anywhere, and the sizes at which the launch changes (16 Ki and 64 Ki rows).  The lists are whole numbers:
exact against the oracle."""
import pytest
import torch

from oracle import dyllm_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 129, 2047, 2048, 2049, 8192, 12289, 16383, 16384, 16385, 24575, 24577, 40961, 65535,
                                  65536, 65537])
@pytest.mark.parametrize("frac", [0.02, 0.6])
def test_salient_select_tile_edges(cuda_device, rows, frac):
    from dyllm_b200 import _lib, ops

    g = torch.Generator().manual_seed(rows)
    stats = torch.ones(rows, 3)
    stats[:, 0] = torch.where(torch.rand(rows, generator=g) < frac, 0.5, 0.999)
    cuts = torch.sort(torch.randint(0, rows + 1, (9,), generator=g)).values
    cu_q = torch.cat([torch.zeros(1, dtype=torch.int64), cuts, torch.tensor([rows])]).to(torch.int32)
    cu_p = (torch.arange(cu_q.numel()) * 37).to(torch.int32)
    want = orc.salient_select(stats, 0.99, cu_q, cu_p)
    sel = ops.salient_select(stats.to(cuda_device), 0.99, cu_q.to(cuda_device), cu_p.to(cuda_device), want_mask=True)
    n = int(sel.count.item())
    assert n == want["count"]
    assert torch.equal(sel.idx[:n].cpu(), want["idx"])
    assert torch.equal(sel.idx_k[:n].cpu(), want["idx_k"])
    assert torch.equal(sel.cu_salientlens.cpu(), want["cu_salientlens"])
    assert torch.equal(sel.mask.cpu(), want["mask"])
    assert _lib.load().dyllm_device_status() == 0
