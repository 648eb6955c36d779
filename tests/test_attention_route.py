"""Which attention kernels a batch takes, on the measured batches: us of forward + backward of the library's, PyTorch's replayed
from a graph, and PyTorch's issued call by call. No GPU needed."""

import pytest

from decentrik_prime_b200 import stack

MEASURED = [
    (28, 4, 128, [1024], 234, 323, 840), (28, 4, 128, [2048], 655, 557, 840), (28, 4, 128, [3072], 1359, 860, 996), (28, 4, 128, [4096], 2257, 1215, 1342),
    (28, 4, 128, [1024] * 8, 1317, 2578, 2992), (28, 4, 128, [512] * 16, 810, 3294, 4117), (28, 4, 128, [227, 277, 365, 82], 114, 467, 1622),
    (12, 2, 128, [951], 161, 215, 872), (12, 2, 128, [3072], 650, 432, 928), (12, 2, 128, [6144], 2168, 892, 1028),
    (40, 8, 128, [1024], 300, 409, 847), (40, 8, 128, [4096], 3074, 1790, 1937), (40, 8, 128, [2048] * 4, 3172, 3465, 3732),
    (14, 2, 64, [1024], 122, 177, 853), (14, 2, 64, [4096], 647, 424, 887), (14, 2, 64, [6144], 1316, 655, 868), (14, 2, 64, [2048] * 4, 636, 797, 1480),
    (16, 16, 64, [2048], 254, 315, 807), (16, 16, 64, [6144], 1498, 947, 1067), (16, 16, 64, [64] * 64, 60, 4000, 12477),
]


@pytest.mark.parametrize("nh,nkv,hd,lens,own,graph,issued", MEASURED)
def test_the_faster_kernels(nh, nkv, hd, lens, own, graph, issued):
    att = stack.PackedAttention(nh, nkv, hd)
    assert att._own_kernels(lens, True) == (own <= graph)
    assert att._own_kernels(lens, False) == (own <= issued)


def test_short_batches_need_no_model():
    for nh, nkv, hd in ((1, 1, 64), (1, 1, 128), (8, 1, 64), (28, 4, 128), (64, 8, 128), (64, 64, 64), (128, 1, 128), (128, 1, 64)):
        att = stack.PackedAttention(nh, nkv, hd)
        for n in (1, 100, 500, 1000, stack._ATTN_SURELY_OWN_ROWS):
            assert att._own_kernels([n], True) and att._own_kernels([n // 2, n - n // 2], True)
