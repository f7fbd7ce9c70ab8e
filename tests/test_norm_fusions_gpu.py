"""One-pass forms against the launches they replace: the same roundings, so the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,heads", [(1, 1), (3, 16), (517, 4), (4099, 16)])
def test_head_norm_with_rotation_equals_the_two_launches(cuda_device, rows, heads):
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, heads, 128, generator=g, device="cuda").bfloat16()
    w = torch.randn(128, generator=g, device="cuda").bfloat16()
    table = torch.randn(700, 128, generator=g, device="cuda")
    pos = torch.randint(-2, 703, (rows,), generator=g, device="cuda")      # clamped to the table
    want = ops.rope_neox_(ops.head_rms_norm_(x.clone(), w, 1e-6), pos, table)
    got = ops.head_rms_norm_rope_(x.clone(), w, 1e-6, pos, table)
    assert torch.equal(got, want)


@pytest.mark.parametrize("live", [0, 1, 37, 1100])
def test_norm_of_listed_rows_finds_their_cache_rows(cuda_device, live):
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(live)
    lens = torch.tensor([0, 311, 5, 900], dtype=torch.int32)
    cu = torch.cat([torch.zeros(1, dtype=torch.int32), lens.cumsum(0, dtype=torch.int32)]).cuda()
    rows = int(lens.sum())
    ids, starts = torch.tensor([3, 0, 2, 5], device="cuda"), torch.tensor([40, -1, 2000, 7, -1, 5000], device="cuda")
    idx = torch.sort(torch.randperm(rows, generator=torch.Generator().manual_seed(live))[:1150]).values.cuda()
    x, res = (torch.randn(rows, 512, generator=g, device="cuda").bfloat16() for _ in range(2))
    w = torch.randn(512, generator=g, device="cuda").bfloat16()
    n = torch.tensor([live], dtype=torch.int32, device="cuda")
    dest = torch.full((idx.numel(),), -7, dtype=torch.int32, device="cuda")
    want = ops.add_rms_norm_rows(x, w, 1e-6, res, idx.int(), n)
    got = ops.add_rms_norm_rows(x, w, 1e-6, res, idx.int(), n, dest=(idx, cu, starts, ids, dest))
    assert torch.equal(got[0][:live], want[0][:live]) and torch.equal(got[1], want[1])
    assert torch.equal(dest[:live], ops.cache_dest_rows(idx, cu, starts, ids, n)[:live])
    assert bool((dest[live:] == -7).all())
