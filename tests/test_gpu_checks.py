"""Tensors that are shorter than the call they come with are refused on the host, before anything is launched; longer ones are
taken, as ever."""

import pytest
import torch

from decentrik_prime_b200 import k_nf4, k_norm, linear, stack
from tests.problem import make_problem, to_device

pytestmark = pytest.mark.gpu
M, N, K = 40, 256, 128


@pytest.fixture(scope="module")
def d():
    return to_device(make_problem(N, K, M, seed=2, lora=True, dropout=0.05, bias=True))


def zeros(*shape, dtype=torch.float16):
    return torch.zeros(*shape, dtype=dtype, device="cuda")


def f32(*shape):
    return zeros(*shape, dtype=torch.float32)


def mask(*shape):
    return zeros(*shape, dtype=torch.uint8)


A, B = (16, K), (N, 16)
SHORT = {
    "out rows": lambda d: linear.forward(d.w, d.x, out=zeros(M - 1, N)),
    "bias": lambda d: linear.forward(d.w, d.x, bias=zeros(N - 8)),
    "bias type": lambda d: linear.forward(d.w, d.x, bias=f32(N)),
    "bias stride": lambda d: linear.forward(d.w, d.x, bias=zeros(2 * N)[::2]),
    "lora_A": lambda d: linear.forward(d.w, d.x, lora=(zeros(16, K - 8), zeros(*B), 1.0)),
    "lora_B": lambda d: linear.forward(d.w, d.x, lora=(zeros(*A), zeros(N - 8, 16), 1.0)),
    "lora on the host": lambda d: linear.forward(d.w, d.x, lora=(zeros(*A).cpu(), zeros(*B), 1.0)),
    "mask rows": lambda d: linear.forward(d.w, d.x, lora=d.lora, mask=mask(M - 1, K)),
    "mask columns": lambda d: linear.forward(d.w, d.x, lora=d.lora, mask=mask(M, K - 16)),
    "mask of one row": lambda d: linear.forward(d.w, d.x, lora=d.lora, mask=mask(K)),
    "mask on the host": lambda d: linear.forward(d.w, d.x, lora=d.lora, mask=mask(M, K).cpu()),
    "workspace on the host": lambda d: linear.forward(d.w, d.x, workspace=torch.empty(1 << 22, dtype=torch.uint8)),
    "multi out rows": lambda d: linear.forward_multi(d.w, d.x, [(N, None, None, 1.0)], out=zeros(M - 1, N)),
    "multi bias": lambda d: linear.forward_multi(d.w, d.x, [(N, None, None, 1.0)], bias=zeros(N - 8)),
    "multi lora_B": lambda d: linear.forward_multi(d.w, d.x, [(128, (zeros(*A), zeros(64, 16), 1.0), None, 1.0), (128, None, None, 1.0)]),
    "multi mask": lambda d: linear.forward_multi(d.w, d.x, [(N, d.lora, mask(M - 1, K), 1.0)]),
    "gate|up lora_B": lambda d: linear.forward_gate_up(d.w, d.x, lora_up=(zeros(*A), zeros(64, 16), 1.0)),
    "gate|up mask": lambda d: linear.forward_gate_up(d.w, d.x, lora_gate=(zeros(*A), zeros(128, 16), 1.0), mask_gate=mask(M - 1, K)),
    "dx rows": lambda d: linear.backward_dx(d.w, d.dy, out=zeros(M - 1, K)),
    "dx mask": lambda d: linear.backward_dx(d.w, d.dy, lora=d.lora, mask=mask(M - 1, K)),
    "dx lora_B": lambda d: linear.backward_dx(d.w, d.dy, lora=(zeros(*A), zeros(N - 8, 16), 1.0)),
    "grads dy rows": lambda d: linear.lora_grads(d.dy[:-1], d.x, f32(M, 16), f32(M, 16), 1.0),
    "grads t": lambda d: linear.lora_grads(d.dy, d.x, f32(M - 1, 16), f32(M, 16), 1.0),
    "grads t type": lambda d: linear.lora_grads(d.dy, d.x, zeros(M, 16), f32(M, 16), 1.0),
    "grads u": lambda d: linear.lora_grads(d.dy, d.x, f32(M, 16), f32(M - 1, 16), 1.0),
    "grads dA": lambda d: linear.lora_grads(d.dy, d.x, f32(M, 16), f32(M, 16), 1.0, dA=f32(16, K - 8)),
    "grads dB": lambda d: linear.lora_grads(d.dy, d.x, f32(M, 16), f32(M, 16), 1.0, dB=f32(N - 8, 16)),
    "grads mask": lambda d: linear.lora_grads(d.dy, d.x, f32(M, 16), f32(M, 16), 1.0, mask=mask(M - 1, K)),
    "swiglu u": lambda d: linear.swiglu_forward(zeros(M, K), zeros(M - 1, K)),
    "swiglu out": lambda d: linear.swiglu_forward(zeros(M, K), zeros(M, K), out=zeros(M - 1, K)),
    "swiglu dh": lambda d: linear.swiglu_backward(zeros(M, K), zeros(M, K), zeros(M - 1, K)),
    "norm lora_A": lambda d: k_norm.rms_forward(f32(M, K), f32(K), zeros(M, K), f32(M), 1e-6, aq=zeros(16, K - 64), tq=f32(M, 16)),
    "norm mask": lambda d: k_norm.rms_forward(f32(M, K), f32(K), zeros(M, K), f32(M), 1e-6, aq=zeros(*A), tq=f32(M, 16), mq=mask(M - 1, K)),
    "dequant codes": lambda d: k_nf4.dequant_tensors(mask(31 * 4), mask(4), f32(1), f32(1), d.code2, 4, NF4(), zeros(256)),
    "dequant absmax": lambda d: k_nf4.dequant_tensors(mask(32 * 300), mask(299), f32(2), f32(2), d.code2, 300, NF4(), zeros(300 * 64)),
    "dequant scale2": lambda d: k_nf4.dequant_tensors(mask(32 * 300), mask(300), f32(1), f32(2), d.code2, 300, NF4(), zeros(300 * 64)),
    "dequant code2": lambda d: k_nf4.dequant_tensors(mask(32), mask(1), f32(1), f32(1), f32(255), 1, NF4(), zeros(64)),
}


def NF4():
    return torch.tensor(k_nf4.NF4_CODE, dtype=torch.float32, device="cuda")


@pytest.mark.parametrize("what", SHORT)
def test_short_tensors_are_refused(d, what):
    with pytest.raises(ValueError):
        SHORT[what](d)


def test_autograd_linear_refuses_short_factors_and_masks(d):
    a, b = f32(*A).requires_grad_(True), f32(*B).requires_grad_(True)
    for lora, m in (((f32(16, K - 8), b, 1.0), None), ((a, f32(N - 8, 16), 1.0), None), ((a, b, 1.0), mask(M - 1, K)), ((a, b, 1.0), mask(K))):
        with pytest.raises(ValueError):
            linear.nf4_lora_linear(d.x, d.w, lora=lora, mask=m)
    with pytest.raises(ValueError):
        linear.nf4_lora_linear(d.x, d.w, bias=zeros(N - 8))


def test_attention_backward_refuses_another_call_s_state():
    att = stack.PackedAttention(2, 1, 64)
    qkv = zeros(70, 4 * 64)
    a, state = att.forward(qkv, [30, 40])
    short, short_state = att.forward(qkv[:69], [30, 39])
    for i, part in enumerate(short_state):
        if torch.is_tensor(part) and part.shape[:1] == (69,):
            with pytest.raises(ValueError):
                att.backward(tuple(part if j == i else s for j, s in enumerate(state)), a)


def test_longer_tensors_are_taken(d):
    y, _ = linear.forward(d.w, d.x, bias=d.bias, lora=d.lora, mask=d.mask, keep_scale=d.keep_scale)
    out = zeros(M + 3, N)
    tall = torch.cat([d.mask, mask(5, K)])
    got, _ = linear.forward(d.w, d.x, bias=torch.cat([d.bias, zeros(8)]), lora=d.lora, mask=tall, keep_scale=d.keep_scale, out=out)
    assert got is out and torch.equal(out[:M], y) and not out[M:].any()
    assert linear.forward(d.w, d.x[:0], lora=d.lora, mask=mask(0))[0].shape == (0, N)      # nothing is read
    one, _ = linear.forward(d.w, d.x[:1], lora=d.lora, mask=d.mask[0], keep_scale=d.keep_scale)
    two, _ = linear.forward(d.w, d.x[:1], lora=d.lora, mask=d.mask[:1], keep_scale=d.keep_scale)
    assert torch.equal(one, two)


def test_rank_16_products_off_a_16_byte_boundary_are_refused(d):
    """They are read four floats at a time. Gradients may lie anywhere in a flat bucket."""
    t, odd = f32(M, 16), f32(M * 16 + 1)[1:].view(M, 16)
    for call in (lambda: linear.forward_multi(d.w, d.x, [(N, d.lora, None, 1.0, odd)]),
                 lambda: linear.lora_grads(d.dy, d.x, odd, t, 1.0), lambda: linear.lora_grads(d.dy, d.x, t, odd, 1.0)):
        with pytest.raises(ValueError):
            call()
    flat = f32(16 * K + 16 * N + 1)
    linear.lora_grads(d.dy, d.x, t + 1, t + 1, 1.0, dA=flat[1:1 + 16 * K].view(16, K), dB=flat[1 + 16 * K:].view(N, 16))
    dA, dB = linear.lora_grads(d.dy, d.x, t + 1, t + 1, 1.0)
    assert torch.allclose(flat[1:1 + 16 * K].view(16, K), dA, rtol=1e-4, atol=1e-3) and torch.allclose(flat[1 + 16 * K:].view(N, 16), dB, rtol=1e-4, atol=1e-3)
