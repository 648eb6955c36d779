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
