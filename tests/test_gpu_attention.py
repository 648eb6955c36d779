"""Rotary embedding + causal grouped-query attention over packed rows against a plain PyTorch fp64 statement of it, forward
and backward, at the edges of the 64-row tiles, with empty and single-row sequences, both head dimensions, grouped and
ungrouped heads, and more sequences than one launch takes. fp16 results of fp32 sums over fp16 probabilities: the rounding
of P, dS (2^-11 each, relative) and of the rotated q, k and the result give a few 2^-11 in the 2-norm; 3e-3 bounds it."""

import numpy as np
import pytest
import torch

from decentrik_prime_b200 import stack

pytestmark = pytest.mark.gpu
REL = 3e-3


def reference(qkv, lens, nh, nkv, hd, theta, da):
    x = qkv.double().cpu().requires_grad_(True)
    H, KV = nh * hd, nkv * hd
    outs, at = [], 0
    inv = theta ** (-torch.arange(0, hd, 2, dtype=torch.float64) / hd)
    for n in lens:
        ang = torch.arange(n, dtype=torch.float64)[:, None] * inv[None, :]
        cos, sin = torch.cat([ang, ang], 1).cos()[:, None], torch.cat([ang, ang], 1).sin()[:, None]

        def rot(t):
            return t * cos + torch.cat([-t[..., hd // 2:], t[..., :hd // 2]], -1) * sin

        rows = x[at:at + n]
        q, k = rot(rows[:, :H].view(n, nh, hd)), rot(rows[:, H:H + KV].view(n, nkv, hd)).repeat_interleave(nh // nkv, 1)
        v = rows[:, H + KV:].view(n, nkv, hd).repeat_interleave(nh // nkv, 1)
        s = torch.einsum("ihd,jhd->hij", q, k) / hd ** 0.5
        s = s.masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool), 1), float("-inf"))
        outs.append(torch.einsum("hij,jhd->ihd", s.softmax(-1), v).reshape(n, H))
        at += n
    out = torch.cat(outs)
    (dx,) = torch.autograd.grad(out, x, da.double().cpu())
    return out.detach(), dx


def rel(got, ref):
    return float((got.double().cpu() - ref).norm() / ref.norm())


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 64), (3, 1, 128), (2, 2, 128), (11, 1, 64), (7, 1, 128)])
@pytest.mark.parametrize("lens", [[1], [63, 64, 65], [128, 0, 1, 200], [5] * 131 + [70], [331]])
def test_attention_against_fp64(nh, nkv, hd, lens):
    gen = torch.Generator().manual_seed(sum(lens) + nh)
    M = sum(lens)
    qkv = torch.randn(M, (nh + 2 * nkv) * hd, generator=gen).half().cuda()
    da = torch.randn(M, nh * hd, generator=gen).half().cuda()
    att = stack.PackedAttention(nh, nkv, hd, theta=1.0e4)
    a, state = att.forward(qkv, lens)
    dqkv = stack.PackedAttention.backward(state, da)
    ref, dref = reference(qkv, [n for n in lens if n], nh, nkv, hd, 1.0e4, da)
    assert rel(a, ref) <= REL
    H, KV = nh * hd, nkv * hd
    if M > 1:                      # a single row attends to itself: d(q) = d(k) = 0
        assert rel(dqkv[:, :H], dref[:, :H]) <= REL
        assert rel(dqkv[:, H:H + KV], dref[:, H:H + KV]) <= REL
    assert rel(dqkv[:, H + KV:], dref[:, H + KV:]) <= REL
    a2, _ = att.forward(qkv, lens)
    assert torch.equal(a, a2) and torch.equal(dqkv, stack.PackedAttention.backward(state, da))


def test_attention_of_unaligned_rows():
    """Rows that do not start on 16-byte boundaries, and a result gradient of another type, as the PyTorch path takes them."""
    gen = torch.Generator().manual_seed(3)
    wide = torch.randn(70, 4 * 64 + 3, generator=gen).half().cuda()
    da = torch.randn(70, 2 * 64, generator=gen).half().cuda()
    att = stack.PackedAttention(2, 1, 64)
    a, state = att.forward(wide[:, 3:], [30, 40])
    b, state_b = att.forward(wide[:, 3:].contiguous(), [30, 40])
    assert torch.equal(a, b)
    odd = torch.empty(70, 2 * 64 + 1, dtype=torch.half, device="cuda")[:, 1:].copy_(da)
    expected = att.backward(state_b, da)
    assert torch.equal(att.backward(state, odd), expected) and torch.equal(att.backward(state, da.float()), expected)
    with pytest.raises(ValueError):
        att.backward(state, da[:69])


@pytest.mark.parametrize("lens", [np.diff(np.array([0, 30, 31, 70])), torch.tensor([30, 1, 39]), (30, 1, 39)], ids=["numpy", "tensor", "tuple"])
def test_sequence_lengths_of_other_types(lens):
    gen = torch.Generator().manual_seed(4)
    qkv = torch.randn(70, 4 * 64, generator=gen).half().cuda()
    att = stack.PackedAttention(2, 1, 64)
    a, state = att.forward(qkv, lens)
    b, state_b = att.forward(qkv, [30, 1, 39])
    assert torch.equal(a, b) and torch.equal(att.backward(state, a), att.backward(state_b, b))


def test_attention_of_a_packed_view_at_an_odd_offset():
    """Contiguous, but off a 16-byte boundary."""
    gen = torch.Generator().manual_seed(6)
    flat = torch.randn(70 * 4 * 64 + 1, generator=gen).half().cuda()
    odd = flat[1:].view(70, 4 * 64)
    assert odd.is_contiguous() and odd.data_ptr() % 16
    da_odd = torch.randn(70 * 2 * 64 + 3, generator=gen).half().cuda()[3:].view(70, 2 * 64)
    att = stack.PackedAttention(2, 1, 64)
    a, state = att.forward(odd, [30, 40])
    b, state_b = att.forward(odd.clone(), [30, 40])
    assert torch.equal(a, b) and torch.equal(att.backward(state, da_odd), att.backward(state_b, da_odd.clone()))


@pytest.mark.parametrize("nh,nkv,hd,lens,graph", [(28, 4, 128, [3100], False), (12, 2, 128, [2300], True), (14, 2, 64, [4100, 70, 0, 1], True)])
def test_long_sequences(nh, nkv, hd, lens, graph):
    """PyTorch's kernels where they are the faster ones, also in a graph captured of lengths that no call has had before."""
    gen = torch.Generator().manual_seed(nh)
    M = sum(lens)
    qkv = torch.randn(M, (nh + 2 * nkv) * hd, generator=gen).half().cuda()
    da = torch.randn(M, nh * hd, generator=gen).half().cuda()
    att = stack.PackedAttention(nh, nkv, hd)
    assert not att._own_kernels(lens, graph)
    own = stack.PackedAttention(nh, nkv, hd)
    own._own_kernels = lambda lens, capturing: True
    a_own, state = own.forward(qkv, lens)
    assert len(state) > 2
    d_own = own.backward(state, da)
    if graph:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            att.backward(att.forward(qkv[:70], [70])[1], da[:70])
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                a, state = att.forward(qkv, lens)
                d = att.backward(state, da)
            assert len(state) == 2
            att.forward(qkv[:71], [71])
            g.replay()
        side.synchronize()
    else:
        a, state = att.forward(qkv, lens)
        assert len(state) == 2
        d = att.backward(state, da)
    assert rel(a, a_own.double().cpu()) <= REL and rel(d, d_own.double().cpu()) <= REL
