"""The CTA-pair GEMM at the edges of its tiles: row tiles (1 .. 256 rows in steps of 32, several of them), ragged column
tiles (256 or 512 columns per pair), short and long contractions, tiles cut along k.

The outputs are bf16 roundings (relative error at most 2^-9, rms below it) of fp32 sums, one rounding for a plain product
and two in a row for the FFN (the intermediate rows are bf16 too): relative L2 error at most 2^-8.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
REL_L2 = 2.0 ** -8


def _close(got, want, what):
    assert bool(torch.isfinite(got.float()).all()), what
    rel = ((got.double() - want).norm() / want.norm().clamp_min(1e-30)).item()
    assert rel <= REL_L2, f"{what}: rel-L2 {rel:.3g}"


def _status_ok():
    from dyllm_b200 import _lib

    assert _lib.load().dyllm_device_status() == 0


def _randn(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()


def _pair(x, w, **kw):
    """The product on the pair kernel, whatever its size: a bias takes a call there, and zeros added in fp32 change nothing."""
    from dyllm_b200 import ops

    return ops.gathered_linear(x, w, bias=torch.zeros(w.size(0), dtype=torch.bfloat16, device="cuda"), bias_fp32=True, **kw)


@pytest.mark.parametrize("rows", [1, 31, 33, 96, 128, 129, 160, 256, 257, 513, 1100])
@pytest.mark.parametrize("k,n", [(64, 64), (192, 192), (1024, 576), (12288, 512), (320, 4096), (4096, 4096), (2112, 2304)])
def test_plain_product(cuda_device, rows, k, n):
    """As the package chooses the kernel (the last two sizes are the pair kernel's at any row count), and the pair kernel by
    force: its row tiles, parts of an odd number of k steps (2112), an empty last part (320)."""
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows * 7 + k + n)
    x, w = _randn(g, rows, k), _randn(g, n, k, scale=0.05)
    want = x.double() @ w.double().t()
    for product in (ops.gathered_linear, _pair):
        got = product(x, w)
        again = product(x, w)
        _status_ok()
        _close(got, want, "plain")
        assert torch.equal(got, again), "the sum of a cut tile does not depend on which CTA arrives last"


@pytest.mark.parametrize("rows", [1, 40, 129, 256, 300, 700])
@pytest.mark.parametrize("hidden,inter", [(64, 64), (256, 192), (4096, 320), (512, 1536), (2048, 4096), (2304, 2112)])
def test_swiglu_ffn(cuda_device, rows, hidden, inter):
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows + hidden + inter)
    x = _randn(g, rows, hidden)
    w1, w2 = _randn(g, 2 * inter, hidden, scale=0.05), _randn(g, hidden, inter, scale=0.05)
    got = ops.swiglu_ffn(x, w1, w2)
    _status_ok()
    h = x.double() @ w1.double().t()
    h = torch.nn.functional.silu(h[:, :inter]) * h[:, inter:]
    _close(got, h.bfloat16().double() @ w2.double().t(), "ffn")


@pytest.mark.parametrize("live,ctas", [(0, 0), (1, 40), (200, 40), (255, 7), (257, 40), (900, 0)])
def test_device_count_column_split_and_fewer_ctas(cuda_device, live, ctas):
    """Rows past the live count hold NaN: nothing of them may reach a live row, and their output rows stay as they are."""
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(live)
    x, w = _randn(g, 1024, 1024), _randn(g, 1536, 1024, scale=0.05)
    x[live:] = float("nan")
    out = torch.full((1024, 1024), 5.0, dtype=torch.bfloat16, device="cuda")
    out2 = torch.full((1024, 512), 5.0, dtype=torch.bfloat16, device="cuda")
    ops.gathered_linear(x, w, num_rows=1024, num_rows_dev=torch.tensor([live], dtype=torch.int32, device="cuda"),
                        out=out, out2=out2, split_col=1024, few_rows_ctas=ctas)
    _status_ok()
    if live:
        want = x[:live].double() @ w.double().t()
        _close(out[:live], want[:, :1024], "first columns")
        _close(out2[:live], want[:, 1024:], "second columns")
    assert bool((out[live:] == 5.0).all()) and bool((out2[live:] == 5.0).all())


@pytest.mark.parametrize("rows,experts,top_k,skew", [(200, 8, 8, 0), (1, 8, 2, 0), (33, 64, 8, 0), (300, 8, 1, 1), (700, 16, 4, 1), (1500, 4, 2, 2)])
def test_grouped_experts(cuda_device, rows, experts, top_k, skew):
    """Experts without rows, with a few, and with several row tiles."""
    from dyllm_b200 import ops

    hidden, inter = 256, 192
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = _randn(g, rows, hidden)
    w1, w2 = _randn(g, experts, 2 * inter, hidden, scale=0.05), _randn(g, experts, hidden, inter, scale=0.05)
    weight = torch.arange(experts, device="cuda").float().add(1).pow(-2.0 * skew).expand(rows, -1)
    ids = torch.multinomial(weight, top_k, generator=g).to(torch.int32)
    tw = torch.rand(rows, top_k, generator=g, device="cuda")
    got = ops.moe_ffn(x, w1, w2, tw, ids)
    again = ops.moe_ffn(x, w1, w2, tw, ids)
    _status_ok()
    want = torch.zeros(rows, hidden, dtype=torch.float64, device="cuda")
    for j in range(top_k):
        for e in range(experts):
            m = (ids[:, j] == e).nonzero().flatten()
            h = x[m].double() @ w1[e].double().t()
            h = (torch.nn.functional.silu(h[:, :inter]) * h[:, inter:]).bfloat16().double()
            want[m] += tw[m, j].double().unsqueeze(1) * (h @ w2[e].double().t())
    # a third rounding: every slot's share is bf16 before the slots are added
    rel = ((got.double() - want).norm() / want.norm()).item()
    assert rel <= 1.5 * REL_L2, f"rel-L2 {rel:.3g}"
    assert torch.equal(got, again)


@pytest.mark.parametrize("rows", [5, 130, 700])
def test_bias_equals_a_separate_addition(cuda_device, rows):
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows)
    x, w, bias = _randn(g, rows, 512), _randn(g, 1024, 512, scale=0.05), _randn(g, 1024)
    k = torch.empty(rows, 384, dtype=torch.bfloat16, device="cuda")
    v = torch.empty(rows, 640, dtype=torch.bfloat16, device="cuda")
    ops.gathered_linear(x, w, out=k, out2=v, split_col=384, bias=bias)
    plain = ops.gathered_linear(x, w)
    _status_ok()
    assert torch.equal(k, plain[:, :384] + bias[:384])
    assert torch.equal(v, plain[:, 384:] + bias[384:])
    once = ops.gathered_linear(x, w, bias=bias, bias_fp32=True)
    want = x.double() @ w.double().t() + bias.double()
    # one rounding of an fp32 sum of 512 products: half an ulp and what the sum is off by
    assert bool(((once.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())


@pytest.mark.parametrize("rows", [1, 100, 128, 129, 200, 256, 300, 512, 513])
@pytest.mark.parametrize("k,n", [(320, 256), (4096, 1024), (1088, 4096)])
def test_same_bits_as_the_kernel_with_named_tiles(cuda_device, rows, k, n):
    """The k range is cut into the same parts as by the tile width that the other kernel takes for this many rows, summed in
    the same order."""
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows + k)
    x, w = _randn(g, rows, k), _randn(g, n, k, scale=0.05)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tile = 128 if -(-rows // 128) * (n // 128) >= sms * 3 // 4 else 64
    got, want = _pair(x, w), ops.gathered_linear(x, w, tile_n=tile)
    _status_ok()
    assert torch.equal(got, want)
    _close(got, x.double() @ w.double().t(), "plain")


@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("rows,k,n", [(40, 4096, 1024), (300, 512, 1088)])
def test_bias_at_any_element(cuda_device, rows, k, n, offset):
    """A bias that is a view at an odd offset, in the epilogue of whole tiles (300 rows) and of tiles cut along k (40)."""
    from dyllm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(rows)
    x, w, bias = _randn(g, rows, k), _randn(g, n, k, scale=0.05), _randn(g, n + 8)[offset:offset + n]
    plain = ops.gathered_linear(x, w, bias=torch.zeros_like(bias), bias_fp32=True)
    got = ops.gathered_linear(x, w, bias=bias)
    once = ops.gathered_linear(x, w, bias=bias, bias_fp32=True)
    _status_ok()
    assert torch.equal(got, plain + bias)
    assert torch.equal(once, ops.gathered_linear(x, w, bias=bias.clone(), bias_fp32=True))


@pytest.mark.parametrize("make", [lambda b: b.float(), lambda b: torch.stack([b, b], 1)[:, 0]])
def test_layer_adds_a_bias_that_the_epilogue_cannot(cuda_device, make):
    """fp32 or strided: added to the bf16 result, as an in-place addition does it."""
    from dyllm_b200 import layers

    g = torch.Generator(device="cuda").manual_seed(1)
    lin = layers.ColumnParallelLinear(512, 1024, bias=True).to("cuda", torch.bfloat16)
    lin.weight.data = _randn(g, 1024, 512, scale=0.05)
    bias = _randn(g, 1024)
    x = _randn(g, 70, 512)
    with torch.inference_mode():
        lin.bias = None
        plain = lin.forward_gathered(x, None, 70)
        lin.bias = torch.nn.Parameter(make(bias), requires_grad=False)
        want = plain.clone()
        want += lin.bias
        assert torch.equal(lin.forward_gathered(x, None, 70), want)
        k, v = lin.forward_gathered(x, None, 70, split_col=256)
        assert torch.equal(torch.cat([k, v], 1), want)
        layers.set_projection_backend("tcgen05")
        try:
            assert torch.equal(lin(x), want)
        finally:
            layers.set_projection_backend("cublas")
    _status_ok()
