"""Hooks on a layer's modules, and modules that a program puts in their place, take part in a step: the shorter ways through
a layer (K and V as two tensors, norm and rotation in one pass, cache rows found by the norm) are for this package's own
methods only.  Runs on the CPU: the parts of the step that need a GPU are replaced."""
import pytest
import torch
from torch import nn

from dyllm_b200 import layers, model
from dyllm_b200.context import get_context, set_context, set_metadata

HID, H, HKV, D, T = 256, 4, 2, 128, 6


class Rotary(nn.Module):
    """Has what a layer needs of a rotary embedding, with the two-argument ``rotate``."""

    def rotate(self, positions, x):
        return x + positions.view(-1, 1, 1).to(x.dtype)

    def forward(self, positions, q, k):
        return self.rotate(positions, q), self.rotate(positions, k)


class Norm(layers.RMSNorm):
    def forward_heads_(self, x, num_rows_dev=None):
        return x * 2


class Caught(nn.Module):
    def forward(self, q, k, v, dv=None):
        self.seen = q, k, v
        return q


class Cache:
    def __init__(self, *args, **kwargs):
        pass

    def reset_full(self, *args, **kwargs):
        pass

    finish = reset_full


@pytest.fixture
def dense_attention(monkeypatch):
    torch.manual_seed(0)
    monkeypatch.setattr(model, "CacheManager", Cache)      # the real ones allocate on a GPU
    monkeypatch.setattr(layers, "CacheManager", Cache)
    attn = model.LLaDAAttention(HID, H, HKV, head_dim=D, max_position=64, rope_theta=1e4, rms_norm_eps=1e-6,
                                rotary_emb=Rotary()).requires_grad_(False)
    for p in attn.parameters():
        nn.init.normal_(p, std=0.05)
    attn.attn = Caught()
    set_metadata([0], [0], [])
    set_context(True, cu_seqlens_q=None, total_seqlen=T)
    yield attn
    set_context(False)


def _expect(attn, x, positions):
    kv = nn.functional.linear(x, attn.kv_proj.weight)
    q = nn.functional.linear(x, attn.q_proj.weight).view(-1, H, D)
    shift = positions.view(-1, 1, 1).float()
    return q + shift, kv[:, : HKV * D].view(-1, HKV, D) + shift, kv[:, HKV * D:].view(-1, HKV, D)


def _run(attn):
    x, positions = torch.randn(T, HID), torch.arange(T)
    attn(positions, x)
    return x, positions


def test_hook_on_the_kv_projection_sees_a_dense_step(dense_attention):
    calls = []
    dense_attention.kv_proj.register_forward_hook(lambda m, args, out: calls.append(out))
    x, positions = _run(dense_attention)
    assert len(calls) == 1 and calls[0].shape == (T, 2 * HKV * D)
    assert all(torch.equal(a, b) for a, b in zip(dense_attention.attn.seen, _expect(dense_attention, x, positions)))


def test_replaced_forward_of_the_kv_projection_is_used(dense_attention):
    kv = dense_attention.kv_proj
    kv.forward = lambda x: nn.functional.linear(x, kv.weight) * 3
    x, positions = _run(dense_attention)
    q, k, v = _expect(dense_attention, x, positions)
    shift = positions.view(-1, 1, 1).float()
    assert torch.equal(dense_attention.attn.seen[2], v * 3)
    assert torch.allclose(dense_attention.attn.seen[1], (k - shift) * 3 + shift, rtol=0, atol=1e-5)


def test_library_backend_covers_the_kv_projection(dense_attention):
    layers.set_projection_backend("cublas")
    try:
        x, positions = _run(dense_attention)
    finally:
        layers.set_projection_backend("default")
    assert all(torch.equal(a, b) for a, b in zip(dense_attention.attn.seen, _expect(dense_attention, x, positions)))


def test_hook_on_the_rotary_embedding_sees_a_dense_step(dense_attention):
    class Own(layers.RotaryEmbedding):
        def rotate(self, positions, x):
            return x + 1

    own, calls = Own(D, D, 64, 1e4), []
    own.register_forward_hook(lambda m, args, out: calls.append(len(args)))
    dense_attention.rotary_emb = own
    layers.set_projection_backend("cublas")
    try:
        _run(dense_attention)
    finally:
        layers.set_projection_backend("default")
    assert calls == [3]


@pytest.mark.parametrize("norm", [None, Norm(D)])
def test_rotary_embedding_with_two_arguments_and_own_head_norm(norm):
    x, positions = torch.randn(T, H, D), torch.arange(T)
    got = model._norm_and_rotate(Rotary(), positions, x, norm)
    assert torch.equal(got, (x * 2 if norm is not None else x) + positions.view(-1, 1, 1))
    assert torch.equal(model._norm_and_rotate(Rotary(), positions, x, norm), got)


def test_replaced_mlp_and_norm_get_the_arguments_they_know():
    class Mlp(nn.Module):
        def forward_salient(self, hidden, staged=False):
            assert staged
            return hidden + 1

    class RowsNorm(nn.Module):
        def forward_rows(self, x, residual, sel_idx32, sel_count_dev=None):
            return x[sel_idx32.long()], residual + x

    layer = nn.Module()
    layer.mlp, layer.post_attention_layernorm = Mlp(), RowsNorm()
    idx = torch.tensor([1, 4], dtype=torch.int32)
    set_metadata([0], [0], [])
    set_context(False, idx_salient_row=idx.long(), idx_salient_row32=idx)
    try:
        assert not get_context().is_full
        x, res = torch.randn(T, HID), torch.randn(T, HID)
        out, residual = model._post_attention(layer, x, res)
    finally:
        set_context(False)
    assert torch.equal(out, x[idx.long()] + 1) and torch.equal(residual, res + x)
