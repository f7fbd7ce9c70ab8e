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
