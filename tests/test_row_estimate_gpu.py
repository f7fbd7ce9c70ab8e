"""The host's estimate of the live rows: where it comes from in steps that the host drives, and what follows from it.

The estimate decides into how many parts the k range of a plain product is cut, hence the order of the fp32 sums.  Both
GEMM kernels must cut alike for every estimate and every count on the device, so their results are compared bit for bit.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_estimate_is_the_count_of_the_last_step_with_or_without_timed_regions(cuda_device):
    from dyllm_b200 import profiling
    from dyllm_b200.layers import Attention

    assert not profiling.enabled()
    attn = Attention(4, 128, 128 ** -0.5, 4)
    assert attn._next_hint(torch.tensor([37], dtype=torch.int32, device="cuda"), 1000) == 1000    # nothing known yet
    torch.cuda.synchronize()
    assert attn._next_hint(torch.tensor([5], dtype=torch.int32, device="cuda"), 1000) == 37
    torch.cuda.synchronize()
    assert attn._next_hint(torch.tensor([9], dtype=torch.int32, device="cuda"), 3) == 3           # never above the capacity
    assert attn._next_hint(torch.tensor([9], dtype=torch.int32, device="cuda"), 1000, fixed=128) == 128


def _planned_tile(estimate, n, sms):
    """Tile width that gathered_gemm_kernel takes on its own for a plain product of ``estimate`` rows."""
    tile = 128 if n % 128 == 0 and -(-estimate // 128) * (n // 128) >= sms * 3 // 4 else 64
    if n % 256 == 0 and estimate > 256 and -(-estimate // 256) * (n // 256) >= sms * 3 // 4:
        tile = 256
    return tile


@pytest.mark.parametrize("hint", [0, 46, 128, 300, 500, 900])
@pytest.mark.parametrize("k,n", [(4096, 4096), (2112, 2304), (320, 3072)])
def test_both_kernels_cut_alike(cuda_device, k, n, hint):
    """A bias of zeros, added in fp32, takes the call to the pair kernel whatever its size and changes no value.  k = 2112 cuts
    into parts of an odd number of 64-column steps, k = 320 into four parts of which the last is empty."""
    from dyllm_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(k + hint)
    x = torch.randn(1024, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).bfloat16()
    zero = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tile = _planned_tile(hint or 1024, n, sms)
    for live in (1, 46, 129, 256, 257, 300, 400, 512, 513, 1024):
        count = torch.tensor([live], dtype=torch.int32, device="cuda")
        got = ops.gathered_linear(x, w, num_rows_dev=count, rows_hint=hint, bias=zero, bias_fp32=True)
        want = ops.gathered_linear(x, w, num_rows_dev=count, rows_hint=hint, tile_n=tile)
        assert torch.equal(got[:live], want[:live]), f"{live} rows, estimate {hint}"
        ref = x[:live].double() @ w.double().t()
        # one bf16 rounding (2^-9 of a value at most) of an fp32 sum
        assert ((got[:live].double() - ref).norm() / ref.norm()).item() <= 2.0 ** -8
    assert _lib.load().dyllm_device_status() == 0


@pytest.mark.parametrize("k,n", [(2048, 4096), (4096, 4096), (3584, 3584), (1536, 4096), (3584, 1024), (4096, 2048)])
def test_chosen_kernel_gives_the_pair_kernels_bits(cuda_device, k, n):
    """Counts on both sides of the lines at which the host's own count changes the kernel (64-column tiles, the pair kernel,
    one wave of 128 x 128 tiles, 256 x 256 tiles)."""
    from dyllm_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(k + n)
    x = torch.randn(3000, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).bfloat16()
    zero = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    for rows in (1, 64, 128, 129, 256, 257, 384, 512, 513, 900, 1600, 3000):
        got = ops.gathered_linear(x, w, num_rows=rows)
        want = ops.gathered_linear(x, w, num_rows=rows, bias=zero, bias_fp32=True)
        assert torch.equal(got, want), f"{rows} rows"
    assert _lib.load().dyllm_device_status() == 0
