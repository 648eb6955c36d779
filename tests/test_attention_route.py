"""Which attention kernels a batch takes, on the measured batches: us of forward + backward of the library's, PyTorch's replayed
from a graph, and PyTorch's issued call by call. No GPU needed."""

import pytest

from decentrik_prime_b200 import stack

MEASURED = [
    (28, 4, 128, [1024], 220, 303, 830), (28, 4, 128, [2048], 624, 561, 868), (28, 4, 128, [3072], 1294, 866, 1001),
    (28, 4, 128, [4096], 2158, 1218, 1350), (28, 4, 128, [1024] * 8, 1270, 2518, 2940), (28, 4, 128, [512] * 16, 784, 3315, 4063),
    (28, 4, 128, [227, 277, 365, 82], 106, 431, 1428), (12, 2, 128, [951], 126, 227, 826), (12, 2, 128, [3072], 588, 434, 807),
    (12, 2, 128, [6144], 2057, 876, 1040), (40, 8, 128, [1024], 281, 415, 813), (40, 8, 128, [4096], 2935, 1769, 1939),
    (40, 8, 128, [2048] * 4, 3046, 3436, 3734), (14, 2, 64, [1024], 100, 182, 801), (14, 2, 64, [4096], 625, 429, 836),
    (14, 2, 64, [6144], 1278, 658, 839), (14, 2, 64, [2048] * 4, 620, 799, 1411), (16, 16, 64, [2048], 235, 322, 802),
    (16, 16, 64, [6144], 1467, 945, 1075), (28, 4, 128, [1500], 398, 440, 797),
    (12, 2, 128, [2500], 428, 389, 926), (14, 2, 64, [2048], 228, 248, 794), (14, 2, 64, [3072], 377, 340, 832),
    (12, 2, 128, [2048] * 2, 550, 584, 1004), (28, 4, 128, [200] * 20, 317, 2264, 4429), (8, 2, 64, [2048], 178, 211, 802),
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
