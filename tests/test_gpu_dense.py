"""The large-batch path (one dequantisation pass, then the dense tcgen05 GEMM), forced through the tuning hook at the
sizes where it can go wrong: rows around the 512-row tile and its 128-row quarters, columns around the 256-column tile,
contractions of one to a few 64-wide steps, tiles cut into 2, 3 and 4 parts of the contraction (clusters), alone and behind
whole waves, stacked segments whose boundaries fall inside a tile, gate|up tiles, accumulation into dx. Launch counts show
that the path ran. Against the fp64 oracle at the path's
tolerance: max-abs-err <= 2e-2 and rel-L2 <= 1e-3."""

import pytest
import torch

from decentrik_prime_b200 import _lib, k_nf4, linear, quantize
from oracle import nf4_oracle
from tests.problem import make_problem, oracle_weight, to_device

pytestmark = pytest.mark.gpu
MAX_ABS, REL_L2 = 2e-2, 1e-3
DENSE = 16


def assert_close(name, got, ref):
    err, rel = nf4_oracle.errors(got, ref)
    assert err <= MAX_ABS and rel <= REL_L2, f"{name}: max-abs {err:.3e} rel-L2 {rel:.3e}"


def workspace(M, N, K):
    return torch.empty(2 * N * K + 192 * M + 32 * N + 2048, dtype=torch.uint8, device="cuda")


WHOLE, BOTH = 1, 16      # what nf4ll_test_dense_plan says: whole tiles, and whole waves before the cut ones


def launches(f):
    before = _lib.lib().nf4ll_launch_count()
    r = f()
    return r, _lib.lib().nf4ll_launch_count() - before


# One to five k-blocks; rows around the tile and its quarters; 192 and 320 columns: ragged tiles. Then the plans, forward and
# backward: short waves cut into 2, 3 and 4 parts, in both directions
@pytest.mark.parametrize("N,K,M,plans", [(256, 64, 1, (WHOLE, WHOLE)), (256, 128, 127, (WHOLE, WHOLE)), (256, 192, 129, (WHOLE, WHOLE)),
                                         (256, 320, 256, (WHOLE, WHOLE)), (512, 512, 257, (WHOLE, WHOLE)), (320, 1024, 511, (WHOLE, WHOLE)),
                                         (192, 256, 512, (WHOLE, WHOLE)), (1536, 1536, 513, (3, 3)), (1024, 4864, 600, (4, WHOLE)),
                                         (768, 7168, 1025, (4, WHOLE)), (2048, 768, 700, (WHOLE, 4)), (2048, 1536, 1500, (2, 3)),
                                         (1536, 2048, 1500, (3, 2)), (1600, 2560, 300, (4, 3))])
@pytest.mark.parametrize("lora,dropout,bias", [(True, 0.05, True), (True, 0.0, False), (False, 0.0, True)])
def test_tile_edges(N, K, M, plans, lora, dropout, bias):
    assert (_lib.lib().nf4ll_test_dense_plan(M, N, K), _lib.lib().nf4ll_test_dense_plan(M, K, N)) == plans
    pr = make_problem(N, K, M, seed=N + K + M, lora=lora, dropout=dropout, bias=bias)
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x, pr.dy, pr.bias, pr.A16, pr.B16, pr.scale, pr.mask, pr.keep_scale)
    d = to_device(pr)
    ws = workspace(M, N, K)
    with linear.tune_override(flags=DENSE):
        (y, t), n = launches(lambda: linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, want_t=lora, workspace=ws))
        assert n == (3 if lora else 2)           # (the rank-16 projection,) the dequantisation pass, the GEMM
        (dx, u), n = launches(lambda: linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, want_u=lora, workspace=ws))
        assert n == (4 if lora else 2)           # lora_B is transposed too
        linear.check_status()
        assert_close("y", y, ref["y"])
        assert_close("dx", dx, ref["dx"])
        again, _ = linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, out=dx.clone(), accumulate=True, workspace=ws)
        y2, _ = linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, workspace=ws)
        linear.check_status()
    if not lora:      # (the rank-16 product of a few hundred rows may be summed with atomics)
        assert torch.equal(y, y2)
    assert_close("dx + dx", again, 2 * ref["dx"])
    if lora:
        assert_close("t", t, ref["t"])
        assert_close("u", u, ref["u"])


@pytest.mark.parametrize("N,K,M,fwd,bwd", [(2048, 2048, 5000, BOTH + 4, BOTH + 4), (4096, 2112, 2560, BOTH + 3, WHOLE), (2112, 4096, 2560, WHOLE, BOTH + 3)])
@pytest.mark.parametrize("dropout", [0.05, 0.0])
def test_more_tiles_than_pairs(N, K, M, fwd, bwd, dropout):
    """Pairs that take several tiles, whole waves and then a short one cut in two launches, with everything fused. The oracle
    computes the rows around the tiles' edges; the kernels that decode give all of them."""
    assert (_lib.lib().nf4ll_test_dense_plan(M, N, K), _lib.lib().nf4ll_test_dense_plan(M, K, N)) == (fwd, bwd)
    pr = make_problem(N, K, M, seed=7, lora=True, dropout=dropout, bias=True)
    rows = torch.tensor(sorted({r for e in range(0, M + 1, 512) for r in (e - 1, e, e + 127, e + 128, e + 300) if 0 <= r < M} | {M - 1}))
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x[rows], pr.dy[rows], pr.bias, pr.A16, pr.B16, pr.scale,
                                    None if pr.mask is None else pr.mask[rows], pr.keep_scale)
    d = to_device(pr)
    ws = workspace(M, N, K)

    def forward():
        return linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, workspace=ws)[0]

    def backward(out=None):
        return linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, out=out, accumulate=out is not None, workspace=ws)[0]

    with linear.tune_override(flags=DENSE):
        y, n = launches(forward)
        assert n == (4 if fwd > BOTH else 3)
        dx, n = launches(backward)
        assert n == (5 if bwd > BOTH else 4)
        twice = backward(dx.clone())
    with linear.tune_override(flags=8):
        ws = None
        y_decoded, dx_decoded = forward(), backward()
    linear.check_status()
    for name, got, want, full in (("y", y, ref["y"], y_decoded), ("dx", dx, ref["dx"], dx_decoded), ("dx + dx", twice, 2 * ref["dx"], 2 * dx_decoded.float())):
        assert_close(name, got[rows.cuda()], want)
        assert_close(name, got, full.double().cpu())


def test_stacked_projections_cut_into_parts():
    """Q|K|V with LoRA on q and v whose boundary lies inside a tile, in tiles cut into parts of the contraction."""
    M, rows, K = 700, (1408, 384, 256), 1536
    N = sum(rows)
    assert _lib.lib().nf4ll_test_dense_plan(M, N, K) == 3
    pr = make_problem(N, K, M, seed=12, lora=True, dropout=0.05, bias=True)
    d = to_device(pr)
    w16, at, segments, branches = oracle_weight(pr), 0, [], []
    for i, r in enumerate(rows):
        l = None if i == 1 else (pr.A16 * (i + 1), pr.B16[at:at + r].contiguous(), 2.0)
        branches.append((at, r, l))
        segments.append((r, None if l is None else (l[0].cuda(), l[1].cuda(), l[2]), None if l is None else d.mask, pr.keep_scale))
        at += r
    with linear.tune_override(flags=DENSE):
        (y, _), n = launches(lambda: linear.forward_multi(d.w, d.x, segments, bias=d.bias, workspace=workspace(M, N, K)))
    linear.check_status()
    assert n == 4                                  # two projections, the dequantisation pass, the GEMM
    for at, r, l in branches:
        A, B, s = (None, None, 1.0) if l is None else l
        ref = nf4_oracle.lora_linear_o1(w16[at:at + r], pr.x, None, pr.bias[at:at + r], A, B, s, None if l is None else pr.mask, pr.keep_scale if l else 1.0)
        assert_close(f"rows {at}", y[:, at:at + r], ref["y"])


@pytest.mark.parametrize("M,H,KV,I", [(300, 512, 128, 1024), (1100, 384, 128, 896)])
def test_stacked_and_gate_up(M, H, KV, I):
    """Q|K|V with segment boundaries inside a 256-column tile (LoRA on q and v), and gate|up with one and two branches."""
    names = k_nf4.LAYER_WEIGHTS
    shapes = {"q_proj": (H, H), "k_proj": (KV, H), "v_proj": (KV, H), "o_proj": (H, H), "gate_proj": (I, H), "up_proj": (I, H), "down_proj": (H, I)}
    lin = {n: quantize.random_nf4_weight(*shapes[n], seed=700 + i, device="cuda") for i, n in enumerate(names)}
    layer, code2 = k_nf4.repack_layer(lin, torch.device("cuda"))
    gen = torch.Generator().manual_seed(M)
    x = torch.randn(M, H, generator=gen).half()
    ks = float(1.0 / torch.tensor(0.95, dtype=torch.float32))

    def branch(n):
        return ((torch.randn(16, H, generator=gen) * 0.05).half(), (torch.randn(n, 16, generator=gen) * 0.05).half(), 2.0)

    def mask():
        return (torch.rand(M, H, generator=gen) >= 0.05).to(torch.uint8)

    def dev(l):
        return None if l is None else (l[0].cuda(), l[1].cuda(), l[2])

    def oracle(name, l, m, bias=None):
        A, B, s = (None, None, 1.0) if l is None else l
        return nf4_oracle.lora_linear_o1(nf4_oracle.dequant_weight(layer, name, code2), x, None, bias, A, B, s, m, ks if m is not None else 1.0)

    qkv = ("q_proj", "k_proj", "v_proj")
    rows = [shapes[n][0] for n in qkv]
    bias = [(torch.randn(r, generator=gen) * 0.1).half() for r in rows]
    loras, masks = [branch(rows[0]), None, branch(rows[2])], [mask(), None, mask()]
    wg = linear.Nf4Weight.from_layer_group(layer, qkv, code2)
    with linear.tune_override(flags=DENSE):
        y, ts = linear.forward_multi(wg, x.cuda(), [(r, dev(l), None if m is None else m.cuda(), ks) for r, l, m in zip(rows, loras, masks)],
                                     bias=torch.cat(bias).cuda(), workspace=workspace(M, wg.N, wg.K))
        linear.check_status()
    at = 0
    for n, r, b, l, m, t in zip(qkv, rows, bias, loras, masks, ts):
        ref = oracle(n, l, m, b)
        assert_close(n, y[:, at:at + r], ref["y"])
        if l is not None:
            assert_close(n + " t", t, ref["t"])
        at += r
    w = linear.Nf4Weight.from_layer_group(layer, ("gate_proj", "up_proj"), code2)
    for lg, lu in ((branch(I), branch(I)), (None, branch(I)), (None, None)):
        mg, mu = (mask() if lg else None), (mask() if lu else None)
        with linear.tune_override(flags=DENSE):
            g, u, h, tg, tu = linear.forward_gate_up(w, x.cuda(), dev(lg), None if mg is None else mg.cuda(), dev(lu),
                                                     None if mu is None else mu.cuda(), ks, workspace=workspace(M, w.N, w.K))
            linear.check_status()
        assert_close("g", g, oracle("gate_proj", lg, mg)["y"])
        assert_close("u", u, oracle("up_proj", lu, mu)["y"])
        assert torch.equal(h, linear.swiglu_forward(g.contiguous(), u.contiguous()))


@pytest.mark.parametrize("bad", [float("inf"), float("nan"), 3.0e4])      # 3e4: the product overflows where it is rounded to fp16
def test_branches_do_not_mix(bad):
    """Two branches in one 256-column tile: a product that is not finite stays in its own branch's columns."""
    M, H, KV, I = 200, 384, 128, 384
    shapes = {"q_proj": (H, H), "k_proj": (KV, H), "v_proj": (KV, H), "gate_proj": (I, H), "up_proj": (I, H)}
    lin = {n: quantize.random_nf4_weight(*s, seed=40 + i, device="cuda") for i, (n, s) in enumerate(shapes.items())}
    layer, code2 = k_nf4.repack_layer(lin, torch.device("cuda"), names=tuple(shapes))
    gen = torch.Generator().manual_seed(5)
    x = torch.randn(M, H, generator=gen).half().cuda()

    def branch(n, ill=False):
        A = torch.randn(16, H, generator=gen) * 0.05
        if ill:
            A[3] = bad
        return A.half().cuda(), (torch.randn(n, 16, generator=gen) * 0.05).half().cuda(), 2.0

    wq = linear.Nf4Weight.from_layer_group(layer, ("q_proj", "k_proj", "v_proj"), code2)
    wg = linear.Nf4Weight.from_layer_group(layer, ("gate_proj", "up_proj"), code2)
    ws = workspace(M, wg.N, wg.K)
    for ill, well, multi in (((0,), (1, 2), (True, False, True)), ((2,), (0, 1), (True, False, True)), ((0,), (1, 2), (True, True, True)),
                             ((2,), (0, 1), (False, False, True))):
        loras = [branch(n, i in ill) if has else None for i, (n, has) in enumerate(zip((H, KV, KV), multi))]
        with linear.tune_override(flags=DENSE):
            y, _ = linear.forward_multi(wq, x, [(n, l, None, 1.0) for n, l in zip((H, KV, KV), loras)], workspace=ws)
        linear.check_status()
        parts = y.split((H, KV, KV), dim=1)
        for i in well:
            A, B, s = (None, None, 1.0) if loras[i] is None else (loras[i][0].cpu(), loras[i][1].cpu(), loras[i][2])
            ref = nf4_oracle.lora_linear_o1(nf4_oracle.dequant_weight(layer, ("q_proj", "k_proj", "v_proj")[i], code2), x.cpu(), None, None, A, B, s, None, 1.0)
            assert_close(f"segment {i}", parts[i], ref["y"])
        assert not all(bool(torch.isfinite(parts[i]).all()) for i in ill)
    for ill in (0, 1):
        for other in (True, False):
            loras = [branch(I, True), branch(I) if other else None][::1 if ill == 0 else -1]
            with linear.tune_override(flags=DENSE):
                g, u, h, _, _ = linear.forward_gate_up(wg, x, loras[0], None, loras[1], None, 1.0, workspace=ws)
            linear.check_status()
            l = loras[1 - ill]
            A, B, s = (None, None, 1.0) if l is None else (l[0].cpu(), l[1].cpu(), l[2])
            ref = nf4_oracle.lora_linear_o1(nf4_oracle.dequant_weight(layer, ("up_proj", "gate_proj")[ill], code2), x.cpu(), None, None, A, B, s, None, 1.0)
            assert_close("other half", (u, g)[ill], ref["y"])
            assert not torch.isfinite((g, u)[ill]).all()


@pytest.mark.parametrize("N,K,M,rows,dense", [(768, 26496, 5884, None, False),            # 36 tiles of 414 steps
                                              (3584, 3584, 3100, None, True),
                                              (1280, 1024, 2604, (1024, 128, 128), False),  # stacked with odd boundaries: 128-wide tiles
                                              (2176, 1664, 2943, (1664, 256, 256), True)])
def test_large_batches_take_the_way_that_the_model_puts_ahead(N, K, M, rows, dense):
    w = to_device(make_problem(N, K, 1, seed=N, lora=False)).w
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(0)).half().cuda()

    def run(flags):
        with linear.tune_override(flags=flags):
            if rows is None:
                return linear.forward(w, x, workspace=ws)[0]
            return linear.forward_multi(w, x, [(r, None, None, 1.0) for r in rows], workspace=ws)[0]

    def route(flags):
        before = _lib.lib().nf4ll_launch_count()
        y = run(flags)
        return _lib.lib().nf4ll_launch_count() - before, y

    ws = torch.empty(max(2 * N * K + 192 * M + 32 * N + 2048, _lib.lib().nf4ll_workspace_bytes(M, N, K, 0)), dtype=torch.uint8, device="cuda")
    decoded, dequantised = route(8), route(DENSE)
    assert decoded[0] != dequantised[0] or not torch.equal(decoded[1], dequantised[1])      # launches or the order of sums tell them apart
    taken = dequantised if dense else decoded
    for workspace_given in (True, False):             # the call's own workspace takes the same way
        if not workspace_given:
            ws = None
        n, y = route(0)
        assert n == taken[0] and torch.equal(y, taken[1])
    linear.check_status()
