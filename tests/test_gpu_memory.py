"""Scratch memory. Calls whose fast route wants an fp16 copy of the weight, on a GPU without that much memory left for this process: they take
the route that decodes inside the GEMM, as they do with a workspace of nf4ll_workspace_bytes."""

import pytest
import torch

from decentrik_prime_b200 import _lib, linear
from oracle import nf4_oracle
from tests.problem import make_problem, oracle_weight, to_device

pytestmark = pytest.mark.gpu


def test_the_smaller_route_when_memory_is_short():
    N = K = 4096
    M = 2048
    pr = make_problem(N, K, M, seed=3, lora=True, dropout=0.05, bias=True)
    d = to_device(pr)
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x, pr.dy, pr.bias, pr.A16, pr.B16, pr.scale, pr.mask, pr.keep_scale)
    h = _lib.lib()
    fast, least = h.nf4ll_workspace_bytes_fast(M, N, K, 16), h.nf4ll_workspace_bytes(M, N, K, 16)
    assert fast > 2 * N * K > 4 * least
    y = torch.empty(M, N, dtype=torch.float16, device="cuda")
    dx = torch.empty(M, K, dtype=torch.float16, device="cuda")
    with linear.tune_override(flags=8):
        plain, _ = linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)
    side = torch.cuda.Stream()                 # a stream without a workspace yet
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    room = torch.cuda.memory_reserved() + max(least, 2 << 20) + (16 << 20)
    try:
        torch.cuda.set_per_process_memory_fraction(room / total)
        with torch.cuda.stream(side):
            with pytest.raises(torch.OutOfMemoryError):
                torch.empty(fast, dtype=torch.uint8, device="cuda")
            for _ in range(2):
                linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, out=y)
                linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, out=dx)
        side.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    linear.check_status()
    assert torch.equal(y, plain)
    for name, got in (("y", y), ("dx", dx)):
        err, rel = nf4_oracle.errors(got, ref[name])
        assert err <= 2e-2 and rel <= 1e-3, (name, err, rel)


@pytest.mark.parametrize("room_for", [1000, 40])
def test_the_gated_backward_takes_fewer_rows_at_a_time(room_for):
    """The parts of its rank-16 products: of 8960 columns 9 KB a row. Every row's parts are added up in the same order."""
    M, I = 2200, 8960
    gen = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    g, u, dh = (rand(M, I).half() for _ in range(3))
    t, B, mask = [rand(M, 16) for _ in range(3)], [(rand(16, I) * 0.05).half() for _ in range(2)], (rand(M, I) > -1.0).to(torch.uint8)

    def run(g, u, grads):
        return linear.gated_backward(g, u, dh, mask, 1.25, *t, (B[0], 2.0), (B[1], 0.5), *grads)

    inputs = [(g.clone(), u.clone(), [torch.empty(s, device="cuda") for s in ((I, 16), (I, 16), (16, I))]) for _ in range(2)]
    want = run(*inputs[0])
    h = _lib.lib()
    full, part = h.nf4ll_gated_backward_bytes(M, I), h.nf4ll_gated_backward_bytes(room_for, I)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.cuda.memory_reserved() + (4 << 20) + (part >> 21 << 21)      # the results, and large blocks in steps of 2 MB
    try:
        torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
        holes = []                                  # of segments that something else keeps
        with pytest.raises(torch.OutOfMemoryError):
            while True:
                holes.append(torch.empty(full, dtype=torch.uint8, device="cuda"))
        got = run(*inputs[1])
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(want + inputs[0][:2], got + inputs[1][:2]):
        assert torch.equal(a, b)
    # fp32 sums of M terms in another order, each term an fp16 product with the side's 22 bits
    for a, b in zip(inputs[0][2], inputs[1][2]):
        assert (a - b).norm() <= M / 16 * 2.0 ** -22 * a.norm()


def test_a_first_call_that_needs_no_scratch():
    """A contraction too short to be split, without LoRA: the first call on a stream, issued and captured."""
    pr = make_problem(256, 64, 130, seed=4, lora=False)
    d = to_device(pr)
    assert _lib.lib().nf4ll_workspace_bytes_fast(130, 256, 64, 0) == 0
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x)
    torch.cuda.synchronize()
    for capture in (False, True):
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            if capture:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=side):
                    y, _ = linear.forward(d.w, d.x)
                graph.replay()
            else:
                y, _ = linear.forward(d.w, d.x)
        side.synchronize()
        err, rel = nf4_oracle.errors(y, ref["y"])
        assert err <= 2e-2 and rel <= 1e-3, (capture, err, rel)
