"""A captured call's scratch belongs to its graph: a replay neither writes to memory that has gone to somebody else since, nor
meets the scratch of eager calls on the same stream."""

import contextlib

import pytest
import torch

from decentrik_prime_b200 import linear
from oracle import nf4_oracle
from tests.problem import make_problem, oracle_weight, tiles_only, to_device

pytestmark = pytest.mark.gpu


def calls(pr, d):
    y, t = linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale, want_t=False)
    dx, _ = linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)
    return y, dx


@pytest.mark.parametrize("warm", [True, False])
@pytest.mark.parametrize("N,K,M,way", [(512, 2048, 70, tiles_only), (4096, 4096, 24, contextlib.nullcontext),      # split tiles, middling batches,
                                       (1024, 2048, 3100, contextlib.nullcontext)])                               # fp16 weight
def test_replay_after_the_workspace_has_grown(N, K, M, way, warm):
    pr = make_problem(N, K, M, seed=N + M, lora=True, dropout=0.05, bias=True)
    d = to_device(pr)
    ref = nf4_oracle.lora_linear_o1(oracle_weight(pr), pr.x, pr.dy, pr.bias, pr.A16, pr.B16, pr.scale, pr.mask, pr.keep_scale)
    big = to_device(make_problem(2048, 4096, 3200, seed=1, lora=True, dropout=0.0))
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        with way():
            if warm:
                calls(pr, d)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                y, dx = calls(pr, d)
        big_y, _ = linear.forward(big.w, big.x, lora=big.lora)      # grows the stream's workspace
        expected = big_y.clone()
        # memory of every size class, so that whatever has been released is somebody's now
        kept = [torch.full((n << 18,), 0x5A, dtype=torch.uint8, device="cuda") for n in (80, 40, 24, 16, 12, 8, 6, 5, 4, 2, 1) for _ in range(12)]
        for _ in range(3):
            y.fill_(float("nan"))
            dx.fill_(float("nan"))
            graph.replay()
            big_y2, _ = linear.forward(big.w, big.x, lora=big.lora)
    side.synchronize()
    linear.check_status()
    for name, got in (("y", y), ("dx", dx)):
        err, rel = nf4_oracle.errors(got, ref[name])
        assert err <= 2e-2 and rel <= 1e-3, (name, err, rel)
    assert torch.equal(big_y2, expected)
    assert all(bool((k == 0x5A).all()) for k in kept)
