"""Attention whose key blocks are shared out between two halves of a CTA: the shortest sequences that take it, odd and even numbers of
blocks, tiles with a single one beside them. The bound is that of the other attention tests."""

import pytest
import torch

from decentrik_prime_b200 import stack
from tests.test_gpu_attention import REL, reference, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 64), (3, 1, 128)])
@pytest.mark.parametrize("lens", [[192, 1], [193], [256, 0, 63], [257, 64], [449, 3, 128]])
def test_halves_against_fp64(nh, nkv, hd, lens):
    gen = torch.Generator().manual_seed(sum(lens) + nh)
    M = sum(lens)
    # scores large enough for one half to hold all of a row's weight
    qkv = torch.randn(M, (nh + 2 * nkv) * hd, generator=gen).mul_(1.7).half().cuda()
    da = torch.randn(M, nh * hd, generator=gen).half().cuda()
    att = stack.PackedAttention(nh, nkv, hd, theta=1.0e4)
    a, state = att.forward(qkv, lens)
    dqkv = stack.PackedAttention.backward(state, da)
    ref, dref = reference(qkv, [n for n in lens if n], nh, nkv, hd, 1.0e4, da)
    H, KV = nh * hd, nkv * hd
    assert rel(a, ref) <= REL
    for part in (slice(0, H), slice(H, H + KV), slice(H + KV, H + 2 * KV)):
        assert rel(dqkv[:, part], dref[:, part]) <= REL
    a2, _ = att.forward(qkv, lens)
    assert torch.equal(a, a2) and torch.equal(dqkv, stack.PackedAttention.backward(state, da))


@pytest.mark.parametrize("nh,nkv,hd", [(14, 2, 64), (12, 3, 128)])
def test_one_half_where_the_tiles_fill_the_device(nh, nkv, hd):
    """As many tiles as take one half again (forward and dQ), of four blocks and fewer."""
    lens = [200] * 9 + [256, 1, 130]
    gen = torch.Generator().manual_seed(nh)
    qkv = torch.randn(sum(lens), (nh + 2 * nkv) * hd, generator=gen).half().cuda()
    da = torch.randn(sum(lens), nh * hd, generator=gen).half().cuda()
    a, state = stack.PackedAttention(nh, nkv, hd, theta=1.0e4).forward(qkv, lens)
    dqkv = stack.PackedAttention.backward(state, da)
    ref, dref = reference(qkv, lens, nh, nkv, hd, 1.0e4, da)
    assert rel(a, ref) <= REL and rel(dqkv, dref) <= REL


@pytest.mark.parametrize("blocks", [(0,), (1,), (0, 1), (1, 2)])
@pytest.mark.parametrize("n", [100, 256, 300])
def test_keys_that_overflowed_add_nothing(n, blocks):
    """Keys of whole blocks infinite in one coordinate, of which every query's is negative: scores of -inf, wherever a half starts."""
    nh = nkv = 1
    hd, theta = 64, 1.0e4
    qkv = torch.randn(n, 3 * hd, generator=torch.Generator().manual_seed(n)).half()
    first, second = hd // 2 - 1, hd - 1            # the pair that turns slowest: a fraction of a degree per position
    qkv[:, [first, second]] = -1.0
    for b in blocks:
        # from position 1 on, where the rotated second coordinate is infinite too
        qkv[max(1, 64 * b):64 * (b + 1), hd + first] = float("inf")
    qkv = qkv.cuda()
    a, _ = stack.PackedAttention(nh, nkv, hd, theta=theta).forward(qkv, [n])
    ref, _ = reference(qkv, [n], nh, nkv, hd, theta, torch.zeros(n, hd).half().cuda())
    assert ref.isfinite().all() and rel(a, ref) <= REL
