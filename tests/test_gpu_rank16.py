"""The rank-16 passes at the edges of their row and column tiles, against fp64: projections T of one and of two branches over the
same rows, one launch (direct with 16 and 32 rows per CTA, through a cluster with 8, 16 and 32, by atomics), and the gradients dA, dB whose warps each
take sixteen rows of a 64-row stage. fp32 sums of n fp16 products: relative error in the 2-norm below n 2^-24 / sqrt(n), here
1e-5 with the hi + lo split of the fp32 operand (2^-22) included."""

import pytest
import torch

from decentrik_prime_b200 import _lib, linear
from tests.problem import make_problem, to_device

pytestmark = pytest.mark.gpu


def rel(got, ref):
    return ((got.cpu().double() - ref).norm() / ref.norm()).item()


def dropped(x, mask, ks):
    return (x.float() * ks).half().double() * mask if mask is not None else x.double()


def variant(M, C, n):
    """How lora_down_launch (csrc/nf4ll_lora.cu) combines the parts of a row's sum, and the rows of a CTA, on a B200's 148 SMs."""
    sms = 148
    groups = {r: -(-M // r) for r in (8, 16, 32)}
    if groups[16] * 4 >= 3 * sms:
        return "direct", 16
    units = -(-C // 256)
    ks = max(1, min(2 * sms // (groups[32] * n), units))
    if ks > 8 and M * C <= 1 << 21:
        ks = 8
    per = -(-units // ks)
    ks = -(-C // (per * 256))
    if ks == 1:
        return "direct", 32
    if ks > 8:
        return "atomic", 32
    aside = M > 16 and C > 16384
    return "cluster", next((r for r in (8, 16) if not aside and groups[r] * ks * n <= 2 * sms), 32)


CASES = [(1, 512, "cluster", 8), (7, 5120, "cluster", 8), (8, 1536, "cluster", 8), (9, 512, "cluster", 8), (17, 2048, "cluster", 8),
         (31, 320, "cluster", 8), (64, 4096, "cluster", 8), (65, 1536, "cluster", 8), (187, 1536, "cluster", 8), (300, 512, "cluster", 8),
         (2300, 512, "direct", 16), (333, 3584, "cluster", 16), (511, 3584, "cluster", 32), (63, 27648, "cluster", 32),
         (701, 256, "direct", 32), (187, 18944, "atomic", 32)]


@pytest.mark.parametrize("M,K,combined,rows", CASES)
def test_projections_of_two_branches(M, K, combined, rows):
    assert torch.cuda.get_device_properties(0).multi_processor_count != 148 or variant(M, K, 2) == (combined, rows)
    parts = (128, 128, 256)
    pr = make_problem(sum(parts), K, M, seed=M + K, lora=False)
    d = to_device(pr)
    g = torch.Generator().manual_seed(M)
    lora = [((torch.randn(16, K, generator=g) / K ** 0.5).half(), (torch.randn(n, 16, generator=g) * 0.02).half()) for n in parts]
    masks = [(torch.rand(M, K, generator=g) >= 0.1).to(torch.uint8), None, (torch.rand(M, K, generator=g) >= 0.1).to(torch.uint8)]
    ks = [1.0 / 0.9, 1.0, 1.0 / 0.9]
    for on in ((0, 2), (0, 1, 2), (1,)):
        segs = [(n, (lora[i][0].cuda(), lora[i][1].cuda(), 2.0) if i in on else None, masks[i].cuda() if i in on and masks[i] is not None else None, ks[i])
                for i, n in enumerate(parts)]
        before = _lib.lib().nf4ll_launch_count()
        _, t = linear.forward_multi(d.w, d.x, segs)
        launches = _lib.lib().nf4ll_launch_count() - before
        linear.check_status()
        with_t = [(*s, ti) if ti is not None else s for s, ti in zip(segs, t)]
        before = _lib.lib().nf4ll_launch_count()
        linear.forward_multi(d.w, d.x, with_t)
        launches -= _lib.lib().nf4ll_launch_count() - before
        # two branches in a launch but where a CTA has whole rows: the choice between them costs those kernels a fifth of their speed
        assert launches == (len(on) if combined == "direct" else (len(on) + 1) // 2)
        for i in on:
            assert rel(t[i], dropped(pr.x, masks[i], ks[i]) @ lora[i][0].double().t()) < 1e-5, (on, i)


@pytest.mark.parametrize("N,K", [(64, 256), (576, 512), (2048, 1216)])
@pytest.mark.parametrize("M", [1, 15, 16, 17, 63, 64, 65, 130, 700])
@pytest.mark.parametrize("dropout", [0.0, 0.1])
def test_gradients(N, K, M, dropout):
    g = torch.Generator().manual_seed(N + M)
    x, dy = torch.randn(M, K, generator=g).half(), torch.randn(M, N, generator=g).half()
    t, u = torch.randn(M, 16, generator=g), torch.randn(M, 16, generator=g)
    mask = (torch.rand(M, K, generator=g) >= dropout).to(torch.uint8) if dropout else None
    ks = 1.0 / (1.0 - dropout)
    dA, dB = linear.lora_grads(dy.cuda(), x.cuda(), t.cuda(), u.cuda(), 2.0, mask=None if mask is None else mask.cuda(), keep_scale=ks)
    assert rel(dA, u.double().t() @ dropped(x, mask, ks)) < 1e-5
    assert rel(dB, 2.0 * dy.double().t() @ t.double()) < 1e-5
