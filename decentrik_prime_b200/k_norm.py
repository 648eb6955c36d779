"""Fused residual add + RMSNorm around the NF4 + LoRA projections: same role, argument names and meaning as the
reference's solution/k_norm.py (`rms_forward`, `rms_backward`), so a layer loop written against that module reads
the same here. The kernels are hand-written sm_100a CUDA behind the C ABI (include/nf4ll.h); there is no Triton
and no CPU fallback.

Where the reference's forward writes the dropped-out copies xq / xv ([M, D] fp16) for the LoRA-A GEMMs that
follow (solution/fast_qwen.py:943-944), this one takes the lora_A shadows (`aq`, `av`) and writes the rank-16
products tq / tv ([M, 16] fp32) directly: hand them to linear.forward_multi as ready-made. Where the reference's
backward takes the [M, D] LoRA input gradients lq / lv (solution/fast_qwen.py:1376-1380), this one takes the
rank-16 factors uq / uv ([M, 16] fp32 = scale * d(out) . lora_B) with `aq`, `av` and expands them per element.
"""

import torch

from . import _lib


def rms_forward(x, w, y, rstd, eps, *, delta=None, xout=None, aq=None, av=None, tq=None, tv=None, mq=None, mv=None,
                keep_scale=1.0):
    """x fp32 [n, d] (+ delta fp16) -> xout fp32 (optional), y fp16 (optional, may be a column slice), rstd fp32 [n],
    tq / tv fp32 [n, 16] = fp16(dropout_{q,v}(norm output)) . {aq, av}^T. Reference: solution/k_norm.py:99-115."""
    _lib.host().rms_forward(x, w, y, rstd, eps, delta, xout, aq, av, tq, tv, mq, mv, keep_scale)


def rms_backward(dy16, gscale, x, w, rstd, out, *, dres=None, uq=None, uv=None, aq=None, av=None, mq=None, mv=None,
                 keep_scale=1.0, out16=None, delta=None):
    """out (fp32, may alias dres) = dres + d(norm input); out16 = its fp16 copy. dy16 is the fp16 gradient of the
    norm output from the projections' backward-dX (run WITHOUT their LoRA branch); uq / uv with aq / av and the
    keep-masks add the LoRA branches' input gradients. Reference: solution/k_norm.py:118-131."""
    g = float(gscale.item()) if isinstance(gscale, torch.Tensor) else float(gscale)
    _lib.host().rms_backward(dy16, g, x, w, rstd, out, dres, uq, uv, aq, av, mq, mv, keep_scale, out16, delta)
