"""Failure detection on the device: a bounded wait that runs out must end the kernel with an error status
the host can read, leave the CUDA context usable and not disturb later calls. The failures are staged
without faulting anything, by hooks of the library: a split contraction launched one split short (with a short poll
limit), so that the wait of every CTA on its tile's other splits can never be satisfied, and something in the kernel for middling
batches that is never signalled."""

import pytest
import torch

from decentrik_prime_b200 import _lib, linear
from tests.problem import make_problem, tiles_only, to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("direction", ["forward", "backward"])
def test_expired_wait_is_reported_and_the_next_call_is_correct(direction):
    # 1536 x 1536 at M = 2048 on the tile kernels: 48 output tiles, so the plan splits the contraction three
    # ways and the 144 CTAs share the reduction (single-CTA kernel forward, CTA-pair kernel backward)
    pr = make_problem(1536, 1536, 2048, seed=71, lora=True, dropout=0.05, bias=True)
    d = to_device(pr)
    dev = d.x.device
    h = _lib.lib()

    def run():
        with tiles_only():
            if direction == "forward":
                return linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0]
            return linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0]

    good = run().clone()
    linear.check_status()
    h.nf4ll_test_expire_wait(2000)
    run()
    with pytest.raises(_lib.Nf4llError) as info:
        linear.check_status()
    assert "wait" in str(info.value)
    word = int(linear.status_word(dev).item())
    assert word == 0x0306, hex(word)             # "a split gave up waiting for its tile's counter"
    linear.status_word(dev).zero_()              # the library never clears the word itself
    # the hook was one-shot, the context is alive, and the tile counters left behind do no harm
    again = run()
    linear.check_status()
    assert torch.equal(again, good)


CODES, RANK16, SUMS = 1, 2, 3


@pytest.mark.parametrize("direction", ["forward", "backward"])
@pytest.mark.parametrize("what,M,rb,nt,cl,words", [(CODES, 40, 1, 48, 1, {0x0705, 0x0707, 0x0708, 0x0709, 0x070a, 0x070d}),
                                                   (CODES, 300, 2, 112, 2, {0x0702, 0x0705, 0x0707, 0x0708, 0x0709, 0x070a, 0x070b, 0x070c}),
                                                   (RANK16, 40, 1, 48, 1, {0x0706, 0x070a, 0x070d}),
                                                   (RANK16, 300, 1, 112, 3, {0x0703, 0x0706, 0x0708, 0x070a, 0x070b, 0x070c}),
                                                   (SUMS, 40, 1, 48, 3, {0x070b, 0x070c}),
                                                   (SUMS, 2000, 1, 32, 2, {0x070b, 0x070c})])       # seven units one after another
def test_expired_waits_of_the_kernel_for_middling_batches(direction, what, M, rb, nt, cl, words):
    """Something that its warps or the other CTAs of a cluster wait for is never signalled (nf4ll_test_mid_withhold; limit 20 ms):
    the kernel ends, the status word holds a wait that depends on it, and the same call gives the same bits again."""
    pr = make_problem(1024, 2048, M, seed=M + cl, lora=True, dropout=0.05, bias=True)
    d = to_device(pr)
    h = _lib.lib()

    def run():
        if direction == "forward":
            return linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0]
        return linear.backward_dx(d.w, d.dy, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)[0]
    h.nf4ll_test_mid(1, rb, nt, cl)
    try:
        good = run().clone()
        linear.check_status()
        h.nf4ll_test_mid_withhold(what, 20000)
        run()
        with pytest.raises(_lib.Nf4llError) as info:
            linear.check_status()
        assert "wait" in str(info.value)
        word = int(linear.status_word(d.x.device).item())
        linear.status_word(d.x.device).zero_()
        assert word in words, hex(word)
        for _ in range(3):
            assert torch.equal(run(), good)
        linear.check_status()
    finally:
        h.nf4ll_test_mid(0, 0, 0, 0)


def test_the_hooks_are_forgotten_after_a_call_that_they_do_not_concern():
    d = to_device(make_problem(512, 512, 64, seed=3, lora=True))
    h = _lib.lib()
    good = linear.forward(d.w, d.x, lora=d.lora)[0].clone()
    h.nf4ll_test_expire_wait(2000)
    h.nf4ll_test_mid_withhold(RANK16, 20000)
    linear.forward(d.w, d.x[:1], lora=d.lora)                 # the weight-streaming kernel has no such waits
    assert torch.equal(linear.forward(d.w, d.x, lora=d.lora)[0], good)      # in the order of the kernel for middling batches
    linear.check_status()
