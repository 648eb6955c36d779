"""The kernel for middling batches (csrc/nf4ll_mid.cu) against the CPU oracle O1 (fp64), at the sizes where its cutting can go
wrong: row tiles, contractions and token tiles with remainders, blocks that do not come in aligned pairs (K a multiple of 64
only), every cluster size, several units in a row per cluster with one accumulator and with two, and both directions with LoRA, mask, bias and accumulation.
Its weights are the bit-exact fp16 ones and every output is one fp32 sum rounded once, so the path's tolerance applies:
max-abs-err <= 2e-2 and rel-L2 <= 1e-3."""

import pytest
import torch

from decentrik_prime_b200 import _lib, linear
from oracle import nf4_oracle
from tests.problem import make_problem, mid, oracle_weight, to_device

pytestmark = pytest.mark.gpu
MAX_ABS, REL_L2 = 2e-2, 1e-3


def assert_close(name, got, ref):
    err, rel = nf4_oracle.errors(got, ref)
    assert err <= MAX_ABS and rel <= REL_L2, f"{name}: max-abs {err:.3e} rel-L2 {rel:.3e}"


def launches(f):
    n0 = _lib.lib().nf4ll_launch_count()
    out = f()
    return out, _lib.lib().nf4ll_launch_count() - n0


def taken():
    return _lib.lib().nf4ll_test_mid_calls()


# (N, K): whole tiles; half a row tile and K of 6 steps; K of 21 steps (blocks in no pairs); K of 10 steps (pairs, no quads)
@pytest.mark.parametrize("N,K", [(256, 512), (320, 384), (1280, 1344), (1024, 640)])
@pytest.mark.parametrize("M,rb,nt,cl", [(1, 1, 16, 1), (17, 1, 32, 2), (33, 2, 48, 1), (100, 1, 64, 3), (129, 2, 80, 2), (187, 1, 192, 2),
                                        (256, 1, 208, 1), (300, 2, 112, 1)])
def test_forward_and_backward(N, K, M, rb, nt, cl):
    if (N * K) % 16384:
        N *= 2
    pr = make_problem(N, K, M, seed=N + M, lora=True, dropout=0.05, bias=True)
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x, pr.dy, pr.bias, pr.A16, pr.B16, pr.scale, pr.mask, pr.keep_scale)
    d = to_device(pr)
    before = taken()
    with mid(rb, nt, min(cl, -(-K // 256), N // 128)):                 # a cluster's CTAs take 256 steps forward, 128 backward at least
        (y, _), n = launches(lambda: linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale))
        dx, _ = linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)
        old = torch.randn(M, K).half()
        acc, _ = linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, out=old.cuda(), accumulate=True)
        plain = linear.forward(d.w, d.x)[0]
    linear.check_status()
    assert n == 2 and taken() - before == 4       # rank-16 projection and the product
    assert_close("y", y, ref["y"])
    assert_close("dx", dx, ref["dx"])
    assert_close("dx accumulated", acc, ref["dx"] + old.double())
    assert_close("y without LoRA", plain, pr.x.double() @ oracle_weight(pr).double().t())


@pytest.mark.parametrize("cl", range(1, 9))
def test_cluster_sizes_give_the_same_bits_every_time(cl):
    """Many units per cluster (3000 tokens in tiles of 32), the sums of the slices exchanged between the CTAs: compared with the
    oracle on some rows, and bit for bit between repeated calls that race with one another."""
    pr = make_problem(1024, 2048, 3000, seed=cl, lora=True, dropout=0.05)
    d = to_device(pr)
    rows = [0, 31, 32, 1501, 2999]
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x[rows], pr.dy[rows], None, pr.A16, pr.B16, pr.scale, pr.mask[rows], pr.keep_scale)

    def both():
        return (linear.forward(d.w, d.x, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0],
                linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0])
    with mid(1, 32, cl):
        first = both()
        again = [both() for _ in range(10)]
    linear.check_status()
    assert_close("y", first[0][rows], ref["y"])
    assert_close("dx", first[1][rows], ref["dx"])
    for other in again:
        assert torch.equal(other[0], first[0]) and torch.equal(other[1], first[1])


# Units beyond the 148 CTAs or 74 pairs that a B200 holds at once. `accumulators`: how many of a unit's columns tensor memory has room for,
# beside the slots of weights (forward) or the masked rank-16 product (backward).
@pytest.mark.parametrize("backward,N,K,M,rb,nt,cl,mask,accumulators", [(False, 2304, 512, 3000, 2, 176, 1, False, 1), (False, 1024, 512, 3000, 2, 64, 1, False, 2),
                                                                       (False, 1024, 512, 2600, 2, 64, 2, False, 2), (False, 1280, 768, 3100, 2, 96, 2, True, 1),
                                                                       (True, 512, 1536, 3000, 2, 112, 1, True, 1), (True, 512, 1536, 3000, 2, 112, 1, False, 2),
                                                                       (True, 512, 1536, 1650, 2, 64, 2, True, 2), (True, 256, 1408, 3000, 1, 224, 1, True, 1),
                                                                       (True, 512, 1280, 3500, 1, 128, 2, True, 2)])
def test_several_units_in_a_row(backward, N, K, M, rb, nt, cl, mask, accumulators):
    beside = rb * nt if backward and mask else 0 if backward else 256
    assert accumulators == (2 if 2 * rb * nt + beside <= 512 else 1)
    pr = make_problem(N, K, M, seed=N + nt, lora=True, dropout=0.05 if mask else 0.0, bias=not backward)
    d = to_device(pr)
    rows = sorted({0, nt - 1, nt, M // 2, M - nt, M - 1})
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x[rows], pr.dy[rows], pr.bias, pr.A16, pr.B16, pr.scale,
                                    pr.mask[rows] if mask else None, pr.keep_scale)
    blocks = -(-(K if backward else N) // (128 * rb))
    assert blocks * -(-M // nt) > {1: 148, 2: 74}[cl]

    def run():
        if backward:
            return linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0]
        return linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0]
    before = taken()
    with mid(rb, nt, cl):
        first = run()
        again = [run() for _ in range(5)]
    linear.check_status()
    assert taken() - before == 6
    assert_close("dx" if backward else "y", first[rows], ref["dx" if backward else "y"])
    assert all(torch.equal(a, first) for a in again)


def test_gate_up_with_several_units_in_a_row():
    """2 x 1152 rows, 3000 tokens in tiles of 176: 162 units on 148 CTAs, one accumulator, two slots of weights, LoRA on both halves."""
    I, K, M = 1152, 512, 3000
    pr = make_problem(2 * I, K, M, seed=I, lora=False)
    g = torch.Generator().manual_seed(M)
    lora = [((torch.randn(16, K, generator=g) / K ** 0.5).half(), (torch.randn(I, 16, generator=g) * 0.02).half(), 2.0) for _ in range(2)]
    d = to_device(pr)
    dev = [(a.cuda(), b.cuda(), s) for a, b, s in lora]
    before = taken()
    with mid(2, 176, 1):
        first = linear.forward_gate_up(d.w, d.x, lora_gate=dev[0], lora_up=dev[1])[:3]
        again = [linear.forward_gate_up(d.w, d.x, lora_gate=dev[0], lora_up=dev[1])[:3] for _ in range(5)]
    linear.check_status()
    assert taken() - before == 6
    rows = [0, 175, 176, 1500, 2999]
    x, w = pr.x[rows].double(), oracle_weight(pr).double()
    for i in range(2):
        assert_close(f"half {i}", first[i][rows], x @ w[i * I:(i + 1) * I].t() + 2.0 * (x @ lora[i][0].double().t()) @ lora[i][1].double().t())
    assert torch.equal(first[2], linear.swiglu_forward(first[0].contiguous(), first[1].contiguous()))
    assert all(torch.equal(a, b) for other in again for a, b in zip(other, first))


@pytest.mark.parametrize("I,K,M,nt,cl", [(256, 512, 20, 32, 1), (320, 1024, 130, 80, 2), (1088, 1024, 300, 112, 3), (256, 512, 187, 192, 1)])
def test_gate_up(I, K, M, nt, cl):
    """A branch whose rank-16 product is not finite does not reach the other one's columns."""
    pr = make_problem(2 * I, K, M, seed=I, lora=False)
    w = oracle_weight(pr).double()
    g = torch.Generator().manual_seed(M)
    lora = [((torch.randn(16, K, generator=g) / K ** 0.5).half(), (torch.randn(I, 16, generator=g) * 0.02).half(), 2.0) for _ in range(2)]
    d = to_device(pr)
    dev = [(a.cuda(), b.cuda(), s) for a, b, s in lora]
    before = taken()
    with mid(2, nt, cl):
        gate, up, h, _, _ = linear.forward_gate_up(d.w, d.x, lora_gate=dev[0], lora_up=dev[1])
        bad = (torch.full_like(dev[0][0], float("inf")), dev[0][1], 2.0)
        _, up_beside, _, _, _ = linear.forward_gate_up(d.w, d.x, lora_gate=bad, lora_up=dev[1])
    linear.check_status()
    assert taken() - before == 2
    for i, got in enumerate((gate, up)):
        t = pr.x.double() @ lora[i][0].double().t()
        assert_close(f"half {i}", got, pr.x.double() @ w[i * I:(i + 1) * I].t() + 2.0 * t @ lora[i][1].double().t())
    hg, hu = gate.cpu().double(), up.cpu().double()
    assert_close("h", h, hg * torch.sigmoid(hg) * hu)
    assert torch.equal(up_beside, up)


def test_stacked_projections():
    """Row tiles of 128 or 256 over segments of 128-row multiples, a branch on the first and on the last."""
    K, M, parts = 512, 70, (384, 128, 256)
    pr = make_problem(sum(parts), K, M, seed=5, lora=False, bias=True)
    w = oracle_weight(pr).double()
    g = torch.Generator().manual_seed(3)
    lora = [((torch.randn(16, K, generator=g) / K ** 0.5).half(), (torch.randn(n, 16, generator=g) * 0.02).half(), 2.0) for n in parts]
    d = to_device(pr)
    segs = [(n, None if i == 1 else (lora[i][0].cuda(), lora[i][1].cuda(), 2.0), None, 1.0) for i, n in enumerate(parts)]
    ref = pr.x.double() @ w.t() + pr.bias.double()
    at = 0
    for i, n in enumerate(parts):
        if i != 1:
            ref[:, at:at + n] += 2.0 * (pr.x.double() @ lora[i][0].double().t()) @ lora[i][1].double().t()
        at += n
    for rb in (1, 2):
        before = taken()
        with mid(rb, 0, 2):
            y, _ = linear.forward_multi(d.w, d.x, segs, bias=d.bias)
        assert taken() - before == 1
        assert_close(f"y, {rb} row blocks", y, ref)
    linear.check_status()


def test_values_that_are_not_finite_stay_in_their_rows():
    """Padding tokens, rows past the weight and steps past the contraction contribute nothing, whatever the neighbours hold."""
    pr = make_problem(320, 384 * 2, 50, seed=9, lora=False)
    d = to_device(pr)
    x = d.x.clone()
    x[7] = float("inf")
    x[9, 3] = float("nan")
    before = taken()
    with mid(1, 64, 2):
        clean, y = linear.forward(d.w, d.x)[0], linear.forward(d.w, x)[0]
    assert taken() - before == 2
    keep = [i for i in range(50) if i not in (7, 9)]
    assert torch.equal(y[keep], clean[keep])
    assert not torch.isfinite(y[[7, 9]]).any()
    linear.check_status()


@pytest.mark.parametrize("M,rb,nt,cl", [(1, 1, 16, 1), (9, 2, 16, 2), (17, 1, 32, 3), (33, 2, 48, 1), (40, 1, 16, 1), (64, 1, 64, 4), (64, 2, 64, 2)])
def test_short_batches_keep_the_rank16_product_in_32_bits(M, rb, nt, cl):
    """Up to 64 rows, with a branch that is nearly all of the output. In two fp16 parts the product is off by 2^-22, and so little
    moves a result to its other neighbour in fp16 (steps of 2^-11 to 2^-10) with a probability of some 2^-11 per term; the fp32
    sums' own error (about 2^-22 of a result) as much: 1 % allowed. A product rounded to fp16 (2^-12) moves two fifths of them.
    A token whose scaled product fp16 cannot hold is finite and as close to fp64 as any; one that is not finite stays alone."""
    N, K = 640, 1024                              # four groups of 256: as many CTAs in a cluster at most
    pr = make_problem(N, K, M, seed=M + nt, lora=False, w_std=1e-3)
    w = oracle_weight(pr).double()
    g = torch.Generator().manual_seed(nt)
    A, B = (torch.randn(16, K, generator=g) / K ** 0.5).half(), torch.randn(N, 16, generator=g).half()
    d = to_device(pr)

    def check(x, B, scale, rows):
        before = taken()
        with mid(rb, nt, cl):
            y, _ = linear.forward(d.w, x.cuda(), lora=(A.cuda(), B.cuda(), scale))
            multi, _ = linear.forward_multi(d.w, x.cuda(), [(256, None, None, 1.0), (384, (A.cuda(), B[:384].contiguous().cuda(), scale), None, 1.0)])
        linear.check_status()
        assert taken() - before == 2
        ref = x.double() @ w.t() + scale * (x.double() @ A.double().t()) @ B.double().t()
        assert (y.cpu()[rows] != ref.half()[rows]).sum() <= 0.01 * N * len(rows)
        ref2 = x.double() @ w[256:].t() + scale * (x.double() @ A.double().t()) @ B[:384].double().t()
        assert (multi.cpu()[rows, 256:] != ref2.half()[rows]).sum() <= 0.01 * 384 * len(rows)
        return y.cpu()
    every = list(range(M))
    check(pr.x, B, 2.0, every)
    x = pr.x.clone()
    x[M // 2] = (x[M // 2].float() * 2.0 ** 12).half()                # its product, times the scale: 2^17 and more
    check(x, (B.float() * 2.0 ** -12).half(), 48.0, every)
    x[M - 1, 5] = float("inf")
    y = check(x, (B.float() * 2.0 ** -12).half(), 48.0, every[:-1])
    assert not torch.isfinite(y[-1]).all()


@pytest.mark.parametrize("N,K,M", [(1536, 1536, 24), (4096, 4096, 64), (8960, 1536, 187)])
@pytest.mark.parametrize("flags", [1, 8, 9])
def test_flags_about_other_kernels_do_not_keep_it_out(N, K, M, flags):
    """Bit 0 (no cooperative reduction) and bit 3 (no dequantisation): the same kernel as without them, bit for bit."""
    d = to_device(make_problem(N, K, M, seed=M, lora=True, dropout=0.05, bias=True))

    def both():
        return (linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0],
                linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0])
    default = both()
    with mid():
        assert all(torch.equal(a, b) for a, b in zip(default, both()))
    with linear.tune_override(flags=flags):
        assert all(torch.equal(a, b) for a, b in zip(default, both()))
    linear.check_status()


@pytest.mark.parametrize("N,K,M,backward", [(5120, 5120, 2300, False), (5120, 5120, 1800, True)])
def test_it_takes_what_the_dense_gemm_would_where_the_workspace_is_too_small(N, K, M, backward):
    """Calls for which the models put the dense GEMM first and this kernel second: with the least workspace, this one. The order
    of the sums, the rank-16 branch's place in it included, tells the three ways apart."""
    h = _lib.lib()
    d = to_device(make_problem(N, K, M, seed=1, lora=True, dropout=0.0, device="cuda"))
    sizes = [h.nf4ll_workspace_bytes(M, N, K, 16), h.nf4ll_workspace_bytes_fast(M, N, K, 16)]
    assert sizes[0] < 2 * N * K <= sizes[1]
    least, fast = (torch.empty(n, dtype=torch.uint8, device="cuda") for n in sizes)

    def run(ws):
        return (linear.backward_dx(d.w, d.dy, lora=d.lora, workspace=ws) if backward else linear.forward(d.w, d.x, lora=d.lora, workspace=ws))[0]
    with mid():
        own = run(least)
    with mid(on=-1):
        tiles = run(least)
    with linear.tune_override(flags=16):
        dense = run(fast)
    assert not torch.equal(own, dense) and not torch.equal(own, tiles)
    assert torch.equal(run(fast), dense) and torch.equal(run(least), own)
    linear.check_status()


def test_plans_of_a_layer_are_searched_for_once():
    """The products of a small layer, forward and backward with and without a mask, at a hundred batch sizes: a second pass over
    the same sizes finds every plan of a batch size it has just made."""
    h = _lib.lib()
    ds = [to_device(make_problem(N, K, 600, seed=N + K, lora=True, dropout=0.05, device="cuda")) for N, K in ((512, 512), (1024, 512), (512, 1024), (768, 512))]

    def layer(M):
        for d in ds:
            x, dy, mask = d.x[:M], d.dy[:M], d.mask[:M]
            linear.forward(d.w, x, lora=d.lora, mask=mask, keep_scale=d.keep_scale)
            linear.forward(d.w, x)
            linear.backward_dx(d.w, dy, lora=d.lora, mask=mask, keep_scale=d.keep_scale)
            linear.backward_dx(d.w, dy)
    for M in range(17, 600, 6):
        layer(M)
        before = h.nf4ll_test_mid_searches()
        layer(M)
        assert h.nf4ll_test_mid_searches() == before, M
    linear.check_status()


# us of the streaming kernel / this one; the first two and the last differ by 2 %, the others by 5 % and more
@pytest.mark.parametrize("N,K,M,gate_up,lora,taken", [
    (5120, 27648, 9, False, False, True), (27648, 5120, 16, False, False, True),      # 40.9 / 40.1, 34.4 / 35.3
    (9344, 11008, 9, False, False, True), (5120, 27648, 12, False, True, True),       # 32.9 / 27.9, 50.4 / 42.8
    (28672, 4096, 9, True, False, True), (27648, 1024, 16, True, False, True),        # 35.0 / 32.0, 15.5 / 12.2
    (28672, 4096, 16, True, True, True), (27648, 5120, 8, False, False, False),       # 41.4 / 34.5, 21.2 / -
    (18944, 3584, 9, True, False, False), (27648, 5120, 16, True, False, False),      # 18.6 / 21.0, 36.7 / 38.7
    (3584, 3584, 16, False, False, False), (10240, 2560, 9, False, False, False),     # 7.9 / 10.7, (streamed by far)
    (11008, 2048, 9, True, False, False), (4096, 4096, 12, True, True, False),        # 10.9 / 13.5, 13.5 / 16.9
    (1536, 8960, 9, False, True, False), (27648, 5120, 9, True, False, False)])       # 11.4 / 14.1, 36.3 / 38.4
def test_nine_to_sixteen_rows_take_the_faster_kernel(N, K, M, gate_up, lora, taken):
    """The default gives one kernel's bits or the other's."""
    d = to_device(make_problem(N, K, M, seed=N + M, lora=lora, device="cuda"))

    def run():
        if not gate_up:
            return linear.forward(d.w, d.x, lora=d.lora)[0]
        half = (d.lora[0], d.lora[1][:N // 2].contiguous(), d.lora[2]) if lora else None
        return linear.forward_gate_up(d.w, d.x, half, None, half, None)[0]
    with mid():
        own = run()
    with mid(on=-1):
        streamed = run()
    assert not torch.equal(own, streamed)
    assert torch.equal(run(), own if taken else streamed)
    linear.check_status()


@pytest.mark.parametrize("M,taken", [(951, True), (1024, False), (1025, True)])
def test_long_chains_with_two_token_slots_are_left_to_the_tiles_where_those_are_ahead(M, taken):
    """2048 x 11008 forward: 144 units of 112 tokens and four slots, 128 units of 128 tokens and two slots, and one row more, for
    which the tiles take another round."""
    d = to_device(make_problem(2048, 11008, M, seed=M, lora=True, dropout=0.0, device="cuda"))
    ws = torch.empty(_lib.lib().nf4ll_workspace_bytes(M, 2048, 11008, 16), dtype=torch.uint8, device="cuda")      # no room for the dense GEMM
    t = d.x.float() @ d.A16.float().t()

    def run():                                        # the rank-16 product given: its sum over a row uses atomics here
        return linear.forward_multi(d.w, d.x, [(2048, d.lora, None, 1.0, t)], workspace=ws)[0]
    with mid():
        own = run()
    with mid(on=-1):
        tiles = run()
    assert not torch.equal(own, tiles)
    assert torch.equal(run(), own if taken else tiles)
    linear.check_status()
