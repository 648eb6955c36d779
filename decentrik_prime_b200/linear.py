"""The NF4 + LoRA linear as Python calls: raw forward / backward_dx / lora_grads for a hand-written
backward (the reference's model is one autograd node with its own backward,
solution/fast_qwen.py:1527-1543) and `nf4_lora_linear`, an autograd function (a C++ node of the host extension) for ordinary
modules. All compute happens in libnf4ll.so (include/nf4ll.h); PyTorch only owns the memory and
the streams. Tensors must be CUDA tensors: nothing here runs on the CPU.

Call-site mapping to the reference (solution/fast_qwen.py):
  forward      <- _ws_use + torch.mm/addmm on the fp16 workspace (947, 1037, 1080-1098, 1112) and the
                  LoRA GEMMs + add (943-946; k_rope.py:39-45, 56-58)
  backward_dx  <- torch.mm(dy, W) (1310, 1320-1327, 1350, 1364), `daq`/`lqx` (1370-1377) and the
                  masked add in k_norm.py:64-71
  lora_grads   <- d_bq / d_aq / d_bv / d_av (1369-1374)
"""

import contextlib
import ctypes
import threading

import torch

from . import _lib
from .k_nf4 import PackedLayer

RANK = 16


class Nf4Weight:
    """One NF4 weight W[N, K] on the GPU: views into a PackedLayer's sections plus the shared
    second-level code table."""

    def __init__(self, packed, qabs, scale2, offset2, code2, rows, cols):
        for t in (packed, qabs, scale2, offset2, code2):
            if not t.is_cuda:
                raise ValueError("NF4 weights must live on the GPU")
        if code2.dtype != torch.float32 or code2.numel() != 256:
            raise ValueError("code2 must be 256 fp32 entries")
        self.packed, self.qabs, self.scale2, self.offset2, self.code2 = packed, qabs, scale2, offset2, code2
        self.N, self.K = int(rows), int(cols)
        self.device = packed.device
        self._c = _lib.Nf4Mat(packed.data_ptr(), qabs.data_ptr(), scale2.data_ptr(), offset2.data_ptr(),
                              code2.data_ptr(), self.N, self.K)
        self._addr = ctypes.addressof(self._c)       # what the host extension reads

    @classmethod
    def from_layer(cls, layer: PackedLayer, name, code2):
        return cls(*layer.weight(name)[:4], code2, *layer.weight(name)[4:])

    @classmethod
    def from_layer_group(cls, layer: PackedLayer, names, code2):
        """Several consecutive weights of a layer as one stacked matrix (for forward_multi); the rows
        of each are kept in `.rows_each`."""
        packed, qabs, scale2, offset2, rows, cols, rows_each = layer.weight_group(names)
        w = cls(packed, qabs, scale2, offset2, code2, rows, cols)
        w.rows_each = list(rows_each)
        return w

    @property
    def nbytes(self):
        """Algorithmic bytes of the weight stream: nibbles + absmax codes + scale2 + offset2."""
        n = self.N * self.K
        return n // 2 + n // 64 + 2 * 4 * (n // 16384)


class _DeviceState(threading.local):
    def __init__(self):
        self.status = {}


_state = _DeviceState()


@contextlib.contextmanager
def tune_override(bm_tiles=0, bn=0, splits=0, flags=0):
    """Testing / tuning hook: force the tile shape (bm_tiles 1|2, bn 128|256, 512 = CTA-pair kernel) and the
    split count for this thread's calls inside the block; flags bit 0 keeps split contractions off the
    cooperative reduction. Workspaces allocated inside the block are sized for the forced plan."""
    h, host = _lib.lib(), _lib.host()
    h.nf4ll_tune_override(bm_tiles, bn, splits, flags)
    host.set_tune(bm_tiles, bn, splits)
    try:
        yield
    finally:
        h.nf4ll_tune_override(0, 0, 0, 0)
        host.set_tune(0, 0, 0)


def status_word(device):
    """The device status word kernels write when a bounded wait expires (zero = healthy)."""
    st = _state.status.get(device.index)
    if st is None:
        st = torch.zeros(1, dtype=torch.int32, device=device)
        _state.status[device.index] = st
    return st


def check_status(device=None):
    """Synchronise the current stream and raise if any kernel reported an expired wait."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else device
    st = status_word(device)
    _lib.check(_lib.lib().nf4ll_read_status(st.data_ptr(), _lib.current_stream(device)))


# Each function below is one call into the host extension (csrc/torch_host.cpp), which checks the tensors, allocates the
# results and finds the calling thread's workspace for the current device and stream (grown on demand; calls on different
# streams of one thread use different ones, `workspace=` replaces it). A call captured by torch.cuda.graph takes its scratch
# from the graph's own memory.
def forward(w: Nf4Weight, x, bias=None, lora=None, mask=None, keep_scale=1.0, out=None, want_t=False,
            workspace=None):
    """y = x . W^T (+ bias) + scale * (drop(x) . A^T) . B^T. `lora` = (A16 [16,K], B16 [N,16], scale) or
    (A16, B16, scale, B16t [16,N]) when the caller keeps a transposed shadow of lora_B for the backward.
    Returns (y, t) with t = drop(x) . A^T in fp32 [M,16] when want_t, else None."""
    return _lib.host().forward(w._addr, x, bias, lora, mask, keep_scale, out, want_t, workspace)


def forward_multi(w: Nf4Weight, x, segments, bias=None, out=None, workspace=None):
    """One launch for several projections that share x and are stacked row-wise in `w` (Q|K|V,
    gate|up; the reference's fused W_qkv GEMM, solution/fast_qwen.py:405-413, 947).
    `segments`: one (rows, lora, mask, keep_scale) per projection, lora as in forward() or None; a fifth element,
    when given, is the projection's ready-made rank-16 product t fp32 [M,16] (k_norm.rms_forward wrote it while
    producing x), which the call then reads instead of computing.
    Returns (y [M, sum rows], [t per segment or None])."""
    return _lib.host().forward_multi(w._addr, x, segments, bias, out, workspace)


def forward_gate_up(w: Nf4Weight, x, lora_gate=None, mask_gate=None, lora_up=None, mask_up=None, keep_scale=1.0,
                    workspace=None):
    """(g, u, h, t_gate, t_up) of an MLP's first half in one launch: `w` is gate_proj and up_proj stacked
    ([2I, K], Nf4Weight.from_layer_group), h = silu(g) * u is formed in the kernel's epilogue (reference:
    two GEMMs + gated_silu, solution/fast_qwen.py:1080-1108). g and u are views of one [M, 2I] buffer."""
    return _lib.host().forward_gate_up(w._addr, x, lora_gate, mask_gate, lora_up, mask_up, keep_scale, workspace)


def backward_dx(w: Nf4Weight, dy, lora=None, mask=None, keep_scale=1.0, out=None, accumulate=False,
                want_u=False, workspace=None):
    """dx (+)= dy . W + keep_scale * mask (.) ((scale * dy . B) . A). Returns (dx, u) with
    u = scale * dy . B in fp32 [M,16] when want_u, else None."""
    return _lib.host().backward_dx(w._addr, dy, lora, mask, keep_scale, out, accumulate, want_u, workspace)


def lora_grads(dy, x, t, u, scale, mask=None, keep_scale=1.0, dA=None, dB=None, accumulate=False):
    """dA[16,K] (+)= u^T . drop(x), dB[N,16] (+)= scale * dy^T . t, both fp32. dA / dB may be views
    into a flat gradient bucket; missing ones are allocated (zero-initialised by the call)."""
    return _lib.host().lora_grads(dy, x, t, u, scale, mask, keep_scale, dA, dB, accumulate)


def lora_u(dy, B16t, scale):
    """u fp32 [M,16] = scale * dy . B, the rank-16 factor of the LoRA branch's backward (reference
    solution/fast_qwen.py:1370, 1373 `daq`, `dav`), from the transposed fp16 shadow B16t [16, N]."""
    return _lib.host().lora_u(dy, B16t, scale)


def lora_grads_batch(projections, accumulate=False):
    """lora_grads of up to three projections over as many rows each, in one launch: (dy, x, t, u, scale, mask, keep_scale,
    dA, dB) of each, dA or dB None to leave it out."""
    _lib.host().lora_grads_batch(projections, accumulate)


def lora_expand(branches, out):
    """out[M,K] = fp16(sum over one or two branches (u, A16, mask, keep_scale) of keep_scale * mask (.) (u . A)): the LoRA
    terms of d(input) of projections that share an input (reference solution/fast_qwen.py:1376-1377), to which one
    backward_dx(..., out=out, accumulate=True) over the stacked weight adds the rest."""
    _lib.host().lora_expand(branches, out)
    return out


def nf4_lora_linear(x, w: Nf4Weight, bias=None, lora=None, mask=None, keep_scale=1.0):
    """Differentiable y = NF4Linear(x) + LoRA(x). `lora` = (A fp32 [16,K], B fp32 [N,16], scale) with
    A and B ordinary parameters: they receive fp32 gradients; W is frozen (no dW)."""
    A, B, scale = (None, None, 1.0) if lora is None else lora
    return _lib.host().linear(x, A, B, w, w._addr, bias, scale, mask, keep_scale)


def swiglu_forward(g, u, out=None):
    """h = fp16(silu(g) * u) in fp32 math (reference solution/k_mlp.py:21-29)."""
    return _lib.host().swiglu_forward(g, u, out)


def swiglu_backward(g, u, dh, inplace=True):
    """(dg, du) from dh; with inplace=True they overwrite g and u, as the reference overwrites its
    fused [gate | up] buffer (solution/k_mlp.py:32-47)."""
    dg = g if inplace else torch.empty_like(g)
    du = u if inplace else torch.empty_like(u)
    _lib.host().swiglu_backward(g, u, dh, dg, du)
    return dg, du


def gated_backward(g, u, dh, mask, keep_scale, t_gate, t_up, u_down, gate, up, dB_gate, dB_up, dA_down, accumulate=False):
    """swiglu_backward in place (g becomes dg, u becomes du), and in the same pass what LoRA branches on gate, up and down take
    from the matrices it holds: returns (u_gate, u_up), fp32 [M,16] = scale * dg . B (lora_u would read dg again for it), and
    writes dB_gate, dB_up (scale * dg^T . t) and dA_down (u_down^T . drop(silu(g) * u)). `gate`, `up`: (B16t, scale) of each."""
    return _lib.host().gated_backward(g, u, dh, g, u, mask, keep_scale, t_gate, t_up, u_down, gate[0], up[0], gate[1], up[1],
                                      dB_gate, dB_up, dA_down, accumulate)
