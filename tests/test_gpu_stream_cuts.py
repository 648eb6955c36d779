"""How the streaming kernel cuts a call up, at its edges: rows of one quantisation block and of as many as one CTA holds and one more
(a cluster), tiles that go round teams, stages and buffers several times, clusters whose last CTA has fewer blocks, absmax codes off a
16-byte boundary, gate|up with its product in the launch and behind it. Against the fp64 oracle, with the tolerance of every forward."""

import pytest
import torch

from decentrik_prime_b200 import _lib, linear
from oracle import nf4_oracle
from tests.problem import make_problem, oracle_weight, tiles_only, to_device
from tests.test_gpu_linear import assert_close

pytestmark = pytest.mark.gpu
COPIES, CLUSTER_SUMS = 1, 3


def reference(pr):
    return nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x, None, pr.bias, pr.A16, pr.B16, pr.scale, pr.mask, pr.keep_scale)["y"]


def forward(d, w=None):
    y = linear.forward(w or d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0]
    linear.check_status()
    return y


# 84 blocks to a CTA up to 8 tokens (5376 weights), 60 beyond (3840); 9728 rows: five tiles for some CTAs, four for others
@pytest.mark.parametrize("N,K", [(256, 64), (256, 448), (192, 5376), (256, 5440), (256, 8128), (192, 3840), (256, 3904), (9728, 512), (19456, 64),
                                 (1024, 8192), (1152, 5376)])      # the last two leave SMs to the rank-16 projection
@pytest.mark.parametrize("M", [1, 5, 8, 9, 16])
def test_edges(N, K, M):
    pr = make_problem(N, K, M, seed=N + K + M, lora=True, dropout=0.05, bias=True, device="cuda" if N * K > 1 << 22 else "cpu")
    with tiles_only():
        assert_close("y", forward(to_device(pr)), reference(pr))


# warps of a team | CTAs of a cluster | teams (beyond 8 tokens two at most): every size of a cluster, parts of one to seven blocks
@pytest.mark.parametrize("np,cl,teams", [(12, 1, 1), (2, 1, 4), (3, 1, 2), (6, 1, 2), (1, 2, 1), (5, 3, 2), (2, 4, 2), (4, 5, 1), (1, 6, 4), (7, 7, 1), (2, 8, 1), (3, 2, 4)])
@pytest.mark.parametrize("M", [3, 13])
def test_forced_cuts(np, cl, teams, M):
    pr = make_problem(9728, 832, M, seed=np + cl + teams, lora=True, dropout=0.05, bias=True, device="cuda")      # 13 blocks a row, 608 tiles
    d = to_device(pr)
    with linear.tune_override(splits=np | cl << 8 | teams << 16, flags=2):
        y = forward(d)
    assert_close("y", y, reference(pr))


# rows that eight CTAs hold and one block more, that sixteen do, and longer ones: all without scratch
@pytest.mark.parametrize("N,K", [(128, 43008), (256, 43072), (384, 65536), (1024, 45056), (256, 86016), (256, 90112)])
@pytest.mark.parametrize("M", [1, 5, 8, 11])
def test_long_rows(N, K, M):
    pr = make_problem(N, K, M, seed=N + M, lora=False, bias=True, device="cuda")
    d = to_device(pr)
    y = linear.forward(d.w, d.x, bias=d.bias, workspace=torch.empty(256, dtype=torch.uint8, device="cuda"))[0]
    linear.check_status()
    assert_close("y", y, reference(pr))


def test_long_rows_of_gate_and_up():
    inter, K, M = 256, 43072, 3
    pr = make_problem(2 * inter, K, M, seed=5, lora=False, device="cuda")
    d = to_device(pr)
    g, u, h, _, _ = linear.forward_gate_up(d.w, d.x, workspace=torch.empty(256, dtype=torch.uint8, device="cuda"))
    linear.check_status()
    y = reference(pr)
    assert_close("g", g, y[:, :inter])
    assert_close("u", u, y[:, inter:])
    assert torch.equal(h, linear.swiglu_forward(g, u))


@pytest.mark.parametrize("on", [(0, 1, 2, 3), (1, 3), (2,)])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
def test_four_projections(M, on):
    """As many segments as a call may have, each with a rank-16 branch of its own or none."""
    rows, K = (256, 128, 384, 128), 1536
    pr = make_problem(sum(rows), K, M, seed=M, lora=False, bias=True)
    d = to_device(pr)
    gen = torch.Generator().manual_seed(M)
    A, B = [torch.randn(16, K, generator=gen).mul_(0.03).half() for _ in rows], [torch.randn(r, 16, generator=gen).mul_(0.05).half() for r in rows]
    scales = (2.0, 0.5, 1.0, 3.0)
    segments = [(r, (A[i].cuda(), B[i].cuda(), scales[i]) if i in on else None, None, 1.0) for i, r in enumerate(rows)]
    with tiles_only():
        y, t = linear.forward_multi(d.w, d.x, segments, bias=d.bias)
    linear.check_status()
    base, at = reference(pr), 0
    for i, r in enumerate(rows):
        ref = base[:, at:at + r]
        if i in on:
            ref = ref + (scales[i] * (pr.x.double() @ A[i].double().t()) @ B[i].double().t()).to(ref.dtype)
        assert (t[i] is not None) == (i in on)
        assert_close(f"y{i}", y[:, at:at + r], ref)
        at += r


@pytest.mark.parametrize("K", [512, 5440])
def test_absmax_codes_off_a_boundary(K):
    d = to_device(make_problem(256, K, 6, seed=K, lora=True, dropout=0.05, bias=True))
    room = torch.empty(d.w.qabs.numel() + 16, dtype=torch.uint8, device="cuda")
    room[4:4 + d.w.qabs.numel()] = d.w.qabs
    shifted = linear.Nf4Weight(d.w.packed, room[4:4 + d.w.qabs.numel()], d.w.scale2, d.w.offset2, d.w.code2, d.w.N, d.w.K)
    assert shifted.qabs.data_ptr() % 16 == 4
    assert torch.equal(forward(d, shifted), forward(d))


# halves of 640 and 9472 rows; in one launch up to 8 tokens, beyond only where a CTA holds a row
@pytest.mark.parametrize("inter,K,launches", [(640, 512, (1, 1)), (9472, 256, (1, 1)), (640, 5632, (1, 2))])
@pytest.mark.parametrize("M", [1, 8, 11])
def test_gate_up(inter, K, launches, M):
    gate, up = (make_problem(inter, K, M, seed=inter + K + i, lora=True, dropout=0.05, device="cuda") for i in (0, 1))
    d = [to_device(p) for p in (gate, up)]
    stacked = [torch.cat([getattr(e.w, n) for e in d]) for n in ("packed", "qabs", "scale2", "offset2")]
    w = linear.Nf4Weight(*stacked, d[0].w.code2, 2 * inter, K)
    h = _lib.lib()
    with tiles_only():
        linear.forward_gate_up(w, d[0].x)      # (its scratch)
    _lib.lib().nf4ll_test_mid(-1, 0, 0, 0)
    try:
        before = h.nf4ll_launch_count()
        linear.forward_gate_up(w, d[0].x)
        assert h.nf4ll_launch_count() - before == launches[M > 8]
        g, u, product, _, _ = linear.forward_gate_up(w, d[0].x, d[0].lora, d[0].mask, d[1].lora, d[1].mask, gate.keep_scale)
    finally:
        _lib.lib().nf4ll_test_mid(0, 0, 0, 0)
    linear.check_status()
    up.x = gate.x
    assert_close("g", g, reference(gate))
    assert_close("u", u, reference(up))
    assert torch.equal(product, linear.swiglu_forward(g.contiguous(), u.contiguous()))


@pytest.mark.parametrize("what,K,M,words", [(COPIES, 512, 1, {0x0801, 0x0802, 0x0806}), (COPIES, 512, 16, {0x0801, 0x0802, 0x0806}),
                                            (COPIES, 6144, 8, {0x0801, 0x0802, 0x0806, 0x0807}), (CLUSTER_SUMS, 6144, 8, {0x0807, 0x0804, 0x0806})])
def test_expired_waits(what, K, M, words):
    """Copies that are never asked for, sums of a cluster that are never announced (nf4ll_test_mid_withhold; limit 20 ms): the kernel
    ends, the status word holds a wait that depends on them, and the same call gives the same bits again."""
    d = to_device(make_problem(4096, K, M, seed=K + M, lora=True, dropout=0.05, bias=True, device="cuda"))
    with tiles_only():
        good = forward(d).clone()
        _lib.lib().nf4ll_test_mid_withhold(what, 20000)
        linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)
        with pytest.raises(_lib.Nf4llError) as info:
            linear.check_status()
        assert "wait" in str(info.value)
        word = int(linear.status_word(d.x.device).item())
        linear.status_word(d.x.device).zero_()
        assert word in words, hex(word)
        for _ in range(3):
            assert torch.equal(forward(d), good)
