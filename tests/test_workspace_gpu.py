"""Workspaces of the GEMM calls: nothing is expected of their content, and calls with different ones may overlap."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TICKET_BYTES = 8192


def _up(v, a):
    return -(-v // a) * a


def _linear(x, w, out, ws, tile_n):
    from dyllm_b200._lib import call, ptr, stream_ptr

    rows, k = x.shape
    call("dyllm_gathered_linear", ptr(x), rows, k, k, None, rows, None, rows, ptr(w), w.size(0), ptr(out), w.size(0), None, 0, 0,
         None, None, ptr(ws), ws.numel(), -1, tile_n, stream_ptr(x.device))


@pytest.mark.parametrize("fill", [0x00, 0x01, 0xFF, 0xA5])
@pytest.mark.parametrize("k,n,tile_n", [(4096, 4096, 0), (4096, 1024, 0), (4096, 1024, 64)])
def test_arrival_counters_lie_in_the_workspace_and_need_no_clearing(cuda_device, k, n, tile_n, fill):
    """The pair kernel (4096 columns) and the 64-column kernel, chosen and named; 40 rows are cut along k in all three."""
    from dyllm_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(n + tile_n)
    x = torch.randn(40, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).bfloat16()
    need = _lib.load().dyllm_gathered_linear_workspace_bytes(40, k, n)
    counters = slice(_up(128 * k * 2, 1024), _up(128 * k * 2, 1024) + TICKET_BYTES)
    outs = []
    for byte in (fill, fill, 0x33):
        ws = torch.full((need,), byte, dtype=torch.uint8, device="cuda")
        out = torch.empty(40, n, dtype=torch.bfloat16, device="cuda")
        _linear(x, w, out, ws, tile_n)
        outs.append(out)
        words = ws[counters].view(torch.int64)
        untouched = int.from_bytes(bytes([byte]) * 8, "little", signed=True)
        used = words[words != untouched]
        assert bool((used == 0).all()), "the last arrival leaves a zero"
        assert byte == 0 or used.numel() >= n // 256, "a counter per cut tile at least"
        _linear(x, w, out, ws, tile_n)      # what the first call has left is as good
        outs.append(out)
    assert _lib.load().dyllm_device_status() == 0
    ref = x.double() @ w.double().t()
    assert ((outs[0].double() - ref).norm() / ref.norm()).item() <= 2.0 ** -8      # bf16 rounding of fp32 sums
    assert all(torch.equal(o, outs[0]) for o in outs)


def test_calls_on_two_streams_get_two_workspaces(cuda_device, monkeypatch):
    """Looked up without launching anything: the workspace is the last pointer but one before the sizes."""
    from dyllm_b200 import _lib, ops

    seen = {}
    monkeypatch.setattr(ops, "call", lambda name, *args: seen.setdefault(name, []).append(args))
    x = torch.zeros(64, 256, dtype=torch.bfloat16, device="cuda")
    w1, w2 = torch.zeros(512, 256, dtype=torch.bfloat16, device="cuda"), torch.zeros(256, 256, dtype=torch.bfloat16, device="cuda")
    sizes = {"dyllm_gathered_linear_bias": _lib.load().dyllm_gathered_linear_workspace_bytes(64, 256, 512),
             "dyllm_swiglu_ffn": _lib.load().dyllm_swiglu_ffn_workspace_bytes(64, 256, 256)}
    for stream in (torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            ops.gathered_linear(x, w1)
            ops.swiglu_ffn(x, w1, w2)
    for name, need in sizes.items():
        # the argument before the workspace's size is the workspace
        pointers = [args[next(i for i, a in enumerate(args) if a == need) - 1] for args in seen[name]]
        assert len(pointers) == 2 and pointers[0] != pointers[1], name


def test_cut_products_on_two_streams(cuda_device):
    """Products of few rows, narrow and wide, in flight on two streams at once: the bits of one after the other."""
    from dyllm_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(3)
    sets = []
    for k, n in ((4096, 4096), (4096, 1024), (1536, 4096), (2112, 8192)):
        x = torch.randn(40, k, generator=g, device="cuda").bfloat16()
        w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).bfloat16()
        sets.append((x, w, ops.gathered_linear(x, w)))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for turn in range(20):
        for s, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                x, w, want = sets[(turn + s * 2) % 4]
                got.append((ops.gathered_linear(x, w), want))
    torch.cuda.synchronize()
    assert _lib.load().dyllm_device_status() == 0
    assert all(torch.equal(a, b) for a, b in got)
