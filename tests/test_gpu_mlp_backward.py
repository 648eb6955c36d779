"""The joined backward of an MLP block: gated-SiLU backward with what LoRA branches take from its matrices, the LoRA terms of dx
expanded for two dropout masks, the factors' gradients of several projections in one launch, at the edges of their tiles."""

import pytest
import torch

from decentrik_prime_b200 import k_nf4, linear
from decentrik_prime_b200.blocks import GradBucket, MlpBlock

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rand(*shape, scale=1.0, seed=0):
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=gen) * scale).to(DEV)


# stages of 16 rows, row ranges of several of them, warps of 32 and CTAs of 128 columns, 16-byte pieces of the mask
@pytest.mark.parametrize("M,I", [(1, 8), (5, 24), (9, 32), (15, 40), (20, 120), (16, 128), (33, 136), (16, 256), (17, 264), (33, 2056), (187, 1000),
                                 (600, 8960), (4801, 520)])
@pytest.mark.parametrize("masked,accumulate", [(True, True), (False, False)])
def test_gated_backward_with_lora(M, I, masked, accumulate):
    gu, dh = rand(M, 2 * I, seed=1).half(), rand(M, I + 8, seed=2).half()[:, :I]
    Bg, Bu = (rand(16, I, scale=0.05, seed=3 + i).half() for i in range(2))
    tg, tu, ud = (rand(M, 16, seed=5 + i) for i in range(3))
    mask = (rand(M, (I + 15) // 16 * 16, seed=8) > -1.0).to(torch.uint8)[:, :I] if masked else None
    grads = [rand(*s, seed=9) for s in ((I, 16), (I, 16), (16, I))]
    before = [x.double() if accumulate else 0.0 for x in grads]
    g, u = gu[:, :I], gu[:, I:]
    dg, du = linear.swiglu_backward(g, u, dh, inplace=False)
    h = linear.swiglu_forward(g, u)
    h = h if mask is None else (h.float() * mask * 1.25).half()
    ug, uu = linear.gated_backward(g, u, dh, mask, 1.25, tg, tu, ud, (Bg, 2.0), (Bu, 0.5), *grads, accumulate)
    assert torch.equal(gu, torch.cat((dg, du), 1))
    # exact products in fp32 sums: a unit in the last place of the absolute sum per addition
    for d, b, s, got in ((dg, Bg, 2.0, ug), (du, Bu, 0.5, uu)):
        bound = s * d.double().abs() @ b.double().abs().t()
        assert ((got.double() - s * d.double() @ b.double().t()).abs() <= (I / 16 + 16) * 2.0 ** -23 * bound + 1e-12).all()
    # and the sides in two fp16 parts (22 bits)
    for d, side, s, got, old in ((dg, tg, 2.0, grads[0], before[0]), (du, tu, 0.5, grads[1], before[1]), (h, ud, 1.0, grads[2].t(), before[2])):
        old = old.t() if got is not grads[0] and got is not grads[1] and accumulate else old
        ref, bound = s * d.double().t() @ side.double() + old, s * d.double().abs().t() @ side.double().abs()
        assert ((got.double() - ref).abs() <= (M / 16 + 16) * 2.0 ** -22 * (bound + abs(old))).all()


@pytest.mark.parametrize("M,K", [(1, 8), (15, 56), (16, 64), (17, 72), (65, 136), (187, 1536), (3001, 200)])
@pytest.mark.parametrize("masked", [(), (0,), (1,), (0, 1)])
@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("size", [1.0, 2.0 ** -20, 2.0 ** 20])
def test_expanded_lora_terms(M, K, masked, n, size):
    """`size`: of u in every third row, beyond fp16's range and far below it, beside an lora_A that brings the terms back to it."""
    ldm = (K + 15) // 16 * 16
    u = [rand(M, 16, scale=0.3, seed=i) for i in range(n)]
    for t in u:
        t[::3] *= size
    A = [(rand(16, K, scale=0.2, seed=5 + i) * size ** -0.5).half() for i in range(n)]
    masks = [(rand(M, ldm, seed=9 + i) > -1.0).to(torch.uint8)[:, :K] if i in masked else None for i in range(n)]
    out = torch.full((M, K + 8), 7.0, dtype=torch.float16, device=DEV)
    linear.lora_expand([(u[i], A[i], masks[i], 1.25) for i in range(n)], out[:, :K])
    ref, bound = 0.0, 0.0
    for i in range(n):
        keep = 1.0 if masks[i] is None else masks[i].double() * 1.25
        ref = ref + keep * (u[i].double() @ A[i].double())
        bound = bound + 1.25 * (u[i].double().abs() @ A[i].double().abs())
    # u in two fp16 parts (22 bits of every rank that counts) and fp32 sums, then one rounding to fp16
    assert ((out[:, :K].double() - ref).abs() <= 2.0 ** -11 * ref.abs() + 2.0 ** -20 * bound + 2.0 ** -24).all()
    assert (out[:, K:] == 7.0).all()


def test_an_infinite_factor_reaches_its_row_only():
    M, K = 20, 96
    A, u = rand(16, K, seed=4).half(), rand(M, 16, seed=5)
    u[3, 7], u[13, 0] = float("inf"), float("nan")
    out = linear.lora_expand([(u, A, None, 1.0)], torch.empty(M, K, dtype=torch.float16, device=DEV))
    rest = torch.ones(M, dtype=torch.bool, device=DEV)
    rest[3] = rest[13] = False
    assert out[rest].isfinite().all() and out[13].isnan().all()
    assert torch.equal(out[3], torch.where(A[7] > 0, float("inf"), float("-inf")).half())


@pytest.mark.parametrize("M", [1, 64, 187, 2048])
@pytest.mark.parametrize("accumulate", [False, True])
def test_gradients_of_three_projections(M, accumulate):
    """Against one call each: the row ranges differ (fp32 sums of M terms in another order)."""
    list_, want = [], []
    for i, (N, K) in enumerate(((72, 200), (8, 1536), (1536, 64))):
        dy, x, t, u = rand(M, N, seed=i).half(), rand(M, K, seed=10 + i).half(), rand(M, 16, seed=20 + i), rand(M, 16, seed=30 + i)
        mask = (rand(M, (K + 15) // 16 * 16, seed=40 + i) > -1.0).to(torch.uint8)[:, :K] if i != 1 else None
        dA, dB = rand(16, K, seed=50 + i), rand(N, 16, seed=60 + i)
        want.append(linear.lora_grads(dy, x, t, u, 0.5, mask=mask, keep_scale=1.25, dA=dA.clone(), dB=dB.clone(), accumulate=accumulate))
        list_.append((dy, x, t, u, 0.5, mask, 1.25, dA, dB))
    linear.lora_grads_batch(list_, accumulate)
    for (dy, x, t, u, s, _, ks, dA, dB), (wA, wB) in zip(list_, want):
        tol = (M / 16 + 16) * 2.0 ** -22
        assert ((dA - wA).abs() <= tol * (ks * (u.abs().t() @ x.float().abs()) + wA.abs() + 1)).all()
        assert ((dB - wB).abs() <= tol * (s * (dy.float().abs().t() @ t.abs()) + wB.abs() + 1)).all()


@pytest.mark.parametrize("M", [1, 24, 187])
@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_joined_and_separate_backward(M, mode):
    """Both orders of the block's backward round dx twice to fp16: each within two half-ulps of the exact sum."""
    H, I = 256, 512
    x, dy = rand(M, H, seed=1).half(), rand(M, H, seed=2).half()
    masks = [(rand(M, k, seed=3 + i) > -1.3).to(torch.uint8) for i, k in enumerate((H, H, I))]
    block = MlpBlock(H, I, 0, DEV)
    got = []
    with mode():
        for joined in (True, False):
            block.forward(x, masks, 1.1)
            if not joined:
                g, u = block._saved
                dx = block._backward_each(g, u, dy, True, False, None)
            else:
                dx = block.backward(dy)
            got.append((dx, [t.clone() for p in block.projections for t in (p.dA, p.dB)]))
    (dx1, gr1), (dx2, gr2) = got
    scale = dx2.float().abs().max()
    assert ((dx1.float() - dx2.float()).abs() <= 2.0 ** -11 * 4 * scale).all()
    for a, b in zip(gr1, gr2):
        assert ((a - b).norm() / b.norm()) < 1e-3          # u of the joined order from fp32 sums in another order


def block_reference(block, x, masks, ks, dy):
    """fp64 over the fp16 weights and factors: dx and dA, dB of gate, up, down. The forward's g, u and h are the block's own."""
    flat = torch.empty(block.layer.numel, dtype=torch.float16, device=DEV)
    k_nf4.dequant_layer(block.layer, block.code2, None, flat)
    at, W = 0, []
    for p in block.projections:
        W.append(flat[at:at + p.w.N * p.w.K].view(p.w.N, p.w.K).double())
        at += p.w.N * p.w.K
    (Ag, Bg), (Au, Bu), (Ad, Bd) = ((p.A16.double(), p.B16.double()) for p in block.projections)
    s = block.gate.scale
    (g, u), h, x, dy = (t.double() for t in block._saved), block.down._saved[0].double(), x.double(), dy.double()
    keep = [m.double() * ks for m in masks]
    ud = s * dy @ Bd
    dh = dy @ W[2] + keep[2] * (ud @ Ad)
    sig = torch.sigmoid(g)
    dg, du = dh * u * sig * (1 + g * (1 - sig)), dh * g * sig
    ug, uu = s * dg @ Bg, s * du @ Bu
    dx = dg @ W[0] + keep[0] * (ug @ Ag) + du @ W[1] + keep[1] * (uu @ Au)
    xg, xu, hd = (keep[i] * t for i, t in enumerate((x, x, h)))
    grads = [ug.t() @ xg, s * dg.t() @ (xg @ Ag.t()), uu.t() @ xu, s * du.t() @ (xu @ Au.t()), ud.t() @ hd, s * dy.t() @ (hd @ Ad.t())]
    return dx, grads


@pytest.mark.parametrize("M", [24, 187])
@pytest.mark.parametrize("side_stream", [False, True])
@pytest.mark.parametrize("with_bucket", [False, True])
@pytest.mark.parametrize("out", ["new", "given", "dy", "none"])
def test_block_backward_over_its_options(M, side_stream, with_bucket, out):
    """dx into a new tensor, a given one, dy itself, or left out; gradients written, then added up by a second backward."""
    H, I = 256, 512
    x, dy = rand(M, H, seed=1).half(), rand(M, H, seed=2).half()
    masks = [(rand(M, k, seed=3 + i) > -1.3).to(torch.uint8) for i, k in enumerate((H, H, I))]
    bucket = GradBucket(MlpBlock.grad_numel(H, I), torch.device(DEV)) if with_bucket else None
    block = MlpBlock(H, I, 0, DEV, bucket=bucket)
    if side_stream:
        block.use_grad_stream()
    for p in block.projections:
        p.dA.fill_(3.0)                               # overwritten by the first backward
        p.dB.fill_(3.0)
    for times in (1, 2):
        block.forward(x, masks, 1.1)
        if times == 1:
            dx_ref, grads_ref = block_reference(block, x, masks, 1.1, dy)
        given = {"given": torch.full_like(dy, 7.0), "dy": dy.clone()}.get(out)
        dx = block.backward(given if out == "dy" else dy, need_dx=out != "none", accumulate_grads=times == 2, out=given)
        assert (dx is None) == (out == "none") and (given is None or dx is given)
        # fp16 activations on the way: a rounding (2^-12 in the 2-norm) each of dy . W_down, dg and du, dx twice
        if dx is not None:
            assert (dx.double() - dx_ref).norm() <= 6 * 2.0 ** -12 * dx_ref.norm()
        for got, ref in zip((t for p in block.projections for t in (p.dA, p.dB)), grads_ref):
            assert (got.double() - times * ref).norm() <= 6 * 2.0 ** -12 * times * ref.norm()
