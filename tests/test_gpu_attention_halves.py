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
