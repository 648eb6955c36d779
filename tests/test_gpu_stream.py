"""The weight-streaming forward of decode-sized batches, and the kernel for middling batches for gate|up: single, stacked (Q|K|V) and
gate|up calls against the fp64 oracle of each projection, at rows of a whole and of an odd number of four quantisation
blocks, at the edges of the token tiles, with and without the rank-16 branch (behind whose kernel the weight stream starts
early). Tolerance as for every forward: fp16 outputs of fp32 sums."""

import pytest
import torch

from decentrik_prime_b200 import k_nf4, linear, quantize
from oracle import nf4_oracle
from tests.problem import make_problem, oracle_weight, to_device
from tests.test_gpu_linear import assert_close, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(64, 256), (256, 576), (1024, 2048), (256, 5184)])
@pytest.mark.parametrize("M,lora", [(1, True), (7, False), (8, True), (9, False), (16, True)])
def test_single_projection(N, K, M, lora):
    run_case(N, K, M, lora=lora, bias=True, seed=N + K + M)


@pytest.mark.parametrize("K", [512, 576, 3456])
@pytest.mark.parametrize("M", [1, 8, 13])
@pytest.mark.parametrize("team", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12])
def test_every_split_of_a_unit(K, M, team):
    """So many warps to a tile of 16 rows, of 8, 9 and 54 quantisation blocks: at most one to a block, and as many as hold the row with
    seven blocks each, beyond eight tokens five (two of the shorter rows; eight and eleven of the longest)."""
    pr = make_problem(256, K, M, seed=K + M + team, lora=True, dropout=0.05, bias=True)
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x, None, pr.bias, pr.A16, pr.B16, pr.scale, pr.mask, pr.keep_scale)
    d = to_device(pr)
    with linear.tune_override(splits=team, flags=2):
        y, _ = linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)
    linear.check_status()
    assert_close("y", y, ref["y"])


def _group(rows, K, seed):
    names = ("q_proj", "k_proj", "v_proj")[:len(rows)]
    lin = {n: quantize.random_nf4_weight(r, K, seed=seed + i, device="cuda") for i, (n, r) in enumerate(zip(names, rows))}
    layer, code2 = k_nf4.repack_layer(lin, torch.device("cuda"), names=names)
    w16 = [nf4_oracle.dequant_weight(k_nf4.PackedLayer(layer.flat.cpu(), layer.offsets, layer.n_qblocks, layer.segments), n, code2.cpu()) for n in names]
    return linear.Nf4Weight.from_layer_group(layer, names, code2), w16


def _branch(gen, n, K, M):
    A, B = (torch.randn(16, K, generator=gen) * 0.05).half(), (torch.randn(n, 16, generator=gen) * 0.05).half()
    return A, B, (torch.rand(M, K, generator=gen) >= 0.05).to(torch.uint8)


@pytest.mark.parametrize("K", [512, 576])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("with_lora", [(0, 2), (), (1,)])
def test_stacked(K, M, with_lora):
    rows, ks, gen = (512, 256, 256), 1.0 / 0.95, torch.Generator().manual_seed(K + M)
    w, w16 = _group(rows, K, seed=7)
    x, bias = torch.randn(M, K, generator=gen).half(), (torch.randn(sum(rows), generator=gen) * 0.1).half()
    br = [_branch(gen, r, K, M) if i in with_lora else None for i, r in enumerate(rows)]
    segs = [(r, None, None, 1.0) if b is None else (r, (b[0].cuda(), b[1].cuda(), 2.0), b[2].cuda(), ks) for r, b in zip(rows, br)]
    y, ts = linear.forward_multi(w, x.cuda(), segs, bias=bias.cuda())
    ready = [s if t is None else (*s, t) for s, t in zip(segs, ts)]
    y2, _ = linear.forward_multi(w, x.cuda(), ready, bias=bias.cuda())
    linear.check_status()
    assert torch.equal(y, y2)
    at = 0
    for i, (r, b) in enumerate(zip(rows, br)):
        A, B, m = b if b is not None else (None, None, None)
        ref = nf4_oracle.lora_linear_o1(w16[i], x, None, bias[at:at + r], A, B, 2.0, m, ks)
        assert_close(f"segment {i}", y[:, at:at + r], ref["y"])
        at += r


# M = 20 and 33 on two weights of 2^24 elements: one launch of the kernel for middling batches
@pytest.mark.parametrize("I,K,M", [(256, K, M) for K in (512, 576) for M in (1, 8, 9, 16)] + [(8192, 2048, 20), (4096, 4096, 33)])
def test_gate_up(I, K, M):
    gen = torch.Generator().manual_seed(K + M)
    w, w16 = _group((I, I), K, seed=9)
    x = torch.randn(M, K, generator=gen).half()
    A, B, m = _branch(gen, I, K, M)
    for lora_up in (None, (A.cuda(), B.cuda(), 2.0)):
        g, u, h, _, _ = linear.forward_gate_up(w, x.cuda(), None, None, lora_up, None if lora_up is None else m.cuda(), 1.0 / 0.95)
        linear.check_status()
        assert_close("g", g, nf4_oracle.lora_linear_o1(w16[0], x)["y"])
        up = nf4_oracle.lora_linear_o1(w16[1], x, None, None, A, B, 2.0, m, 1.0 / 0.95) if lora_up else nf4_oracle.lora_linear_o1(w16[1], x)
        assert_close("u", u, up["y"])
        assert torch.equal(h, linear.swiglu_forward(g.contiguous(), u.contiguous()))
