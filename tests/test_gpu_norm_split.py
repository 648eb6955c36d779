"""The norms with a group of eight rows shared out over a cluster: rows past the end, parts and chunks that do not divide the row, LoRA
factors far from 1, against fp64."""

import pytest
import torch

from decentrik_prime_b200 import k_norm

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rand(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def mask_of(M, D, seed):
    return (rand(M, (D + 15) // 16 * 16, seed=seed) > -1.3).to(torch.uint8)[:, :D]


# 1, 2, .. 8 CTAs of 1 .. 4 chunks per warp, and rows that take a CTA each: D / 32 chunks, (M + 7) / 8 groups
@pytest.mark.parametrize("M,D", [(1, 8), (9, 264), (8, 520), (3, 1000), (15, 1544), (300, 1544), (1100, 1544), (333, 3584), (17, 4096), (600, 4088), (1185, 1016), (2000, 72)])
@pytest.mark.parametrize("branches", ["", "q", "v", "qv"])
def test_split_norms(M, D, branches):
    check_norms(M, D, branches, 0)


# ranks of u that fall by a factor of 2 each beside rows of lora_A that rise by it: every rank counts for as much in the result
@pytest.mark.parametrize("M,D", [(9, 264), (300, 1544), (600, 4088)])
def test_ranks_of_unlike_size(M, D):
    check_norms(M, D, "qv", 1)


def check_norms(M, D, branches, fall):
    x, delta, w = rand(M, D, seed=1), rand(M, D, seed=2).half(), rand(D, seed=3)
    rank = 2.0 ** (fall * torch.arange(16, device=DEV, dtype=torch.float32))
    A = {b: (rand(16, D, seed=4 + i, scale=0.05) * rank[:, None]).half() for i, b in enumerate("qv") if b in branches}
    m = {"q": mask_of(M, D, 6)} if "q" in branches else {}          # v without dropout
    t = {b: torch.empty(M, 16, device=DEV) for b in A}
    y, rstd, xo = torch.empty(M, D + 8, device=DEV).half(), torch.empty(M, device=DEV), torch.empty(M, D, device=DEV)
    y_view = y.view(-1)[:M * D].view(M, D)
    ks = 1.25
    k_norm.rms_forward(x, w, y_view, rstd, 1e-6, delta=delta, xout=xo, aq=A.get("q"), av=A.get("v"), tq=t.get("q"), tv=t.get("v"), mq=m.get("q"),
                       keep_scale=ks)
    xs = x + delta.float()
    assert torch.equal(xo, xs)
    r = ((xs.double() ** 2).mean(1) + 1e-6).rsqrt()
    assert (rstd.double() / r - 1).abs().max() < 1e-5 * (D / 1000 + 1) ** 0.5
    ref = w.double() * xs.double() * rstd.double()[:, None]
    assert ((y_view.double() - ref).abs() <= 2.0 ** -11 * 1.01 * ref.abs() + 2.0 ** -24).all()
    for b in A:
        d = ref if b not in m else ref * ks * m[b]
        # a rounding of each dropped-out value to fp16, exact products, fp32 sums
        bound = d.abs() @ A[b].double().abs().t()
        assert ((t[b].double() - d @ A[b].double().t()).abs() <= (2.0 ** -11 + D / 16 * 2.0 ** -23) * 1.05 * bound + 1e-7).all()

    u = {b: rand(M, 16, seed=8 + i) for i, b in enumerate(A)}
    scales = (1.0, 1e-9, 1e7)
    for i, b in enumerate(u):
        u[b] *= torch.tensor([scales[(row + i) % 3] for row in range(M)], device=DEV)[:, None] / rank
    dy, dres = rand(M, D, seed=10).half(), rand(M, D, seed=11)
    out, o16 = dres.clone(), torch.empty(M, D, device=DEV).half()
    k_norm.rms_backward(dy, 0.5, x, w, rstd, out, dres=out, uq=u.get("q"), uv=u.get("v"), aq=A.get("q"), av=A.get("v"), mq=m.get("q"), keep_scale=ks,
                        out16=o16, delta=delta)
    g, size = dy.double() * 0.5, dy.double().abs() * 0.5
    for b in u:
        keep = m[b].double() * ks if b in m else 1.0
        g = g + keep * (u[b].double() @ A[b].double())
        size = size + keep * (u[b].double().abs() @ A[b].double().abs())
    xhat, wd, rd = xs.double() * rstd.double()[:, None], w.double(), rstd.double()[:, None]
    ref = (g * wd - xhat * (g * wd * xhat).mean(1, keepdim=True)) * rd + dres.double()
    # fp32: a few roundings of each term, of the factors' sixteen products and of the row's sum
    size, rough = size * wd.abs(), (size * (wd * xhat).abs()).mean(1, keepdim=True)
    assert ((out.double() - ref).abs() <= 2.0 ** -24 * ((20 * size + (24 + D / 64) * xhat.abs() * rough) * rd + 2 * ref.abs() + 2 * dres.double().abs())).all()
    assert torch.equal(o16, out.half())


def test_an_infinite_factor_reaches_its_row_only():
    M, D = 16, 1536
    x, w, rstd, dy = rand(M, D, seed=1), rand(D, seed=2), torch.ones(M, device=DEV), rand(M, D, seed=3).half()
    A, u = rand(16, D, seed=4).half(), rand(M, 16, seed=5)
    u[3, 7], u[5, 0] = float("inf"), float("nan")
    out = torch.empty(M, D, device=DEV)
    k_norm.rms_backward(dy, 1.0, x, w, rstd, out, uq=u, aq=A)
    bad = ~torch.isfinite(out).all(1)
    assert bad[3] and bad[5] and bad.sum() == 2
