"""The calls that users of this library make, over the range of sizes they make them at, as timed cases.

`listed()` names a fixed set, `draw(rng)` gives further ones of the same ranges. `prepare(case, seed)` builds what a
program holds before the call (weights, LoRA factors, activations, a captured graph), `run(state)` is one pass through
the public entry points, `work(case)` the bytes and operations that pass cannot do without, `tolerance(case)` how far
two correct implementations at the same precision may lie apart.

Kinds:
  linear       one projection's forward (linear.forward): a layer server or a test bench calling one matrix
  decode       the four linear launches of one decoder layer at a decode-sized batch (Q|K|V, O, gate|up, down),
               issued call by call or replayed from a captured graph, as a serving loop does
  prefill      one decoder layer's forward over packed prompts, norms and attention included (stack.NormedStack)
  autograd     one projection as a differentiable op: forward, d(input), LoRA gradients (linear.nf4_lora_linear)
  mlp          forward and backward of an MLP block with LoRA + dropout on all three projections (blocks.MlpBlock)
  stack        training step of whole decoder layers over packed sequences as one autograd node (stack.NormedStack)
  projections  training step of one layer's seven projections (stack.ProjectionStack)
  dequant      a layer's weights to fp16 (k_nf4.dequant_layer): weight export, the reference's workspace fill
"""

import math

import torch

from decentrik_prime_b200 import blocks, k_nf4, linear, quantize, stack

RANK = 16
P_DROP = 0.05
KEEP_SCALE = 1.0 / float(torch.tensor(1.0 - P_DROP, dtype=torch.float32))
BYTES_PER_WEIGHT = 0.5 + 1 / 64 + 8 / 16384          # codes, absmax codes, second-level scale and offset
HEAD = 128                                           # head dimension of the attention layers


def listed():
    return [
        # decoding one sequence: a single square projection, the smallest call there is
        dict(name="linear_m1_5120x5120", kind="linear", N=5120, K=5120, M=1, lora=True, bias=False),
        # decoding a few sequences against the widest projection
        dict(name="linear_m8_27648x5120", kind="linear", N=27648, K=5120, M=8, lora=True, bias=False),
        # a full decode batch against the longest contraction
        dict(name="linear_m64_5120x27648", kind="linear", N=5120, K=27648, M=64, lora=True, bias=False),
        # one token through a 7B-sized layer, launches replayed from a graph
        dict(name="decode_m1_7b_graph", kind="decode", hidden=3584, kv=512, inter=18944, M=1, graph=True),
        # a mid-sized decode batch through a 32B-sized layer, issued call by call
        dict(name="decode_m24_32b", kind="decode", hidden=5120, kv=1024, inter=27648, M=24, graph=False),
        # one prompt of odd length through a 7B-sized layer
        dict(name="prefill_333_7b", kind="prefill", hidden=3584, kv=512, inter=18944, lengths="333"),
        # fine-tuning: one attention projection as a module in somebody's model
        dict(name="autograd_m2048_1536x1536", kind="autograd", N=1536, K=1536, M=2048),
        # fine-tuning: the MLP of a 1.5B layer at the benchmark's batch
        dict(name="mlp_m2048_1.5b", kind="mlp", hidden=1536, inter=8960, M=2048),
        # the same block on a short ragged batch
        dict(name="mlp_m187_1.5b", kind="mlp", hidden=1536, inter=8960, M=187),
        # fine-tuning: two 1.5B decoder layers over four packed sequences of a data loader's batch (951 rows)
        dict(name="stack_951_1.5b", kind="stack", hidden=1536, kv=256, inter=8960, layers=2, lengths="227,277,365,82"),
        # fine-tuning: the projections of one 7B layer at the largest packed batch
        dict(name="projections_m16384_7b", kind="projections", hidden=3584, kv=512, inter=18944, M=16384),
        # all weights of a 1.5B layer to fp16
        dict(name="dequant_1.5b", kind="dequant", hidden=1536, kv=256, inter=8960),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, lo, hi, step):
    return max(lo, min(hi, _log_int(rng, lo, hi) // step * step))


def _lengths(rng, most_rows, most_sequences=4):
    n = rng.randint(1, most_sequences)
    each = max(16, most_rows // n)
    return ",".join(str(_log_int(rng, 16, each)) for _ in range(n))


def draw(rng):
    kind = rng.choice(("linear", "linear", "decode", "decode", "prefill", "autograd", "mlp", "stack", "projections", "dequant"))
    if kind == "linear":
        N, K = _multiple(rng, 1024, 27648, 128), _multiple(rng, 1024, 27648, 128)
        while N * K > 27648 * 5120:
            N, K = _multiple(rng, 1024, 27648, 128), _multiple(rng, 1024, 27648, 128)
        return dict(kind=kind, N=N, K=K, M=_log_int(rng, 1, 512), lora=rng.random() < 0.7, bias=rng.random() < 0.4)
    if kind == "autograd":
        return dict(kind=kind, N=_multiple(rng, 512, 5120, 128), K=_multiple(rng, 512, 5120, 128), M=_log_int(rng, 64, 8192))
    widest = {"decode": 5120, "prefill": 3584, "mlp": 2048, "stack": 2048, "projections": 3584, "dequant": 3584}[kind]
    hidden = _multiple(rng, 1024, widest, 256)
    inter = _multiple(rng, int(2.6 * hidden), int(5.8 * hidden), 128) // 128 * 128
    if kind == "mlp":
        return dict(kind=kind, hidden=hidden, inter=inter, M=_log_int(rng, 48, 4096))
    kv_heads = rng.choice([n for n in (1, 2, 4, 8) if hidden // HEAD % n == 0])
    case = dict(kind=kind, hidden=hidden, kv=kv_heads * HEAD, inter=inter)
    if kind == "decode":
        case.update(M=_log_int(rng, 1, 64), graph=rng.random() < 0.5)
    elif kind == "prefill":
        case.update(lengths=_lengths(rng, 2048))
    elif kind == "stack":
        case.update(layers=rng.randint(1, 3), lengths=_lengths(rng, 2048))
    elif kind == "projections":
        case.update(M=_log_int(rng, 256, 16384))
    return case


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
class _Draws:
    """Seeded draws on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=torch.float32):
        return (torch.randn(*shape, device=self.dev, generator=self.gen) * std).to(dtype)

    def uniform(self, *shape, bound):
        return (torch.rand(*shape, device=self.dev, generator=self.gen) * 2 - 1) * bound

    def mask(self, M, K):
        return (torch.rand(M, K, device=self.dev, generator=self.gen) >= P_DROP).to(torch.uint8)

    def nf4(self, N, K):
        """A 4-bit linear with weights ~ N(0, 0.02), as a checkpoint would hold it."""
        return quantize.FakeLinear4bit(quantize.quantize_nf4(self.normal(N, K, std=0.02, dtype=torch.float16)))

    def lora_masters(self, N, K):
        """fp32 A (kaiming uniform) and B of a partly trained adapter."""
        return self.uniform(RANK, K, bound=1.0 / math.sqrt(K)), self.normal(N, RANK, std=0.01)

    def lora(self, N, K, scale=2.0):
        A, B = self.lora_masters(N, K)
        return (A.half(), B.half(), scale, B.half().t().contiguous())

    def layer_parts(self, hidden, kv, inter):
        shapes = _layer_shapes(hidden, kv, inter)
        layer, code2 = k_nf4.repack_layer({n: self.nf4(*s) for n, s in shapes.items()}, self.dev)
        return {"layer": layer, "code2": code2,
                "bias": {n: self.normal(shapes[n][0], std=0.1, dtype=torch.float16) for n in ("q_proj", "k_proj", "v_proj")},
                "lora": {n: (*self.lora_masters(*shapes[n]), 2.0) for n in ("q_proj", "v_proj")},
                "norm": (self.uniform(hidden, bound=0.5) + 1.0, self.uniform(hidden, bound=0.5) + 1.0, 1e-6)}

    def layer_masks(self, M, hidden):
        return {n: self.mask(M, hidden) for n in ("q_proj", "v_proj")}


def _layer_shapes(hidden, kv, inter):
    return {"q_proj": (hidden, hidden), "k_proj": (kv, hidden), "v_proj": (kv, hidden), "o_proj": (hidden, hidden),
            "gate_proj": (inter, hidden), "up_proj": (inter, hidden), "down_proj": (hidden, inter)}


def _seq(case):
    return [int(n) for n in case["lengths"].split(",")]


def prepare(case, seed):
    d, kind = _Draws(seed), case["kind"]
    s = {"kind": kind}
    if kind in ("linear", "autograd"):
        N, K, M = case["N"], case["K"], case["M"]
        layer, code2 = k_nf4.repack_layer({"w": d.nf4(N, K)}, d.dev, names=("w",))
        s["w"] = linear.Nf4Weight.from_layer(layer, "w", code2)
        s["x"] = d.normal(M, K, dtype=torch.float16)
        if kind == "linear":
            s["lora"] = d.lora(N, K) if case["lora"] else None
            s["bias"] = d.normal(N, std=0.1, dtype=torch.float16) if case["bias"] else None
        else:
            s["x"].requires_grad_(True)
            A, B = d.lora_masters(N, K)
            s["A"], s["B"] = A.requires_grad_(True), B.requires_grad_(True)
            s["mask"], s["dy"] = d.mask(M, K), d.normal(M, N, dtype=torch.float16)
    elif kind == "decode":
        hidden, kv, inter, M = case["hidden"], case["kv"], case["inter"], case["M"]
        p = d.layer_parts(hidden, kv, inter)
        group = lambda *names: linear.Nf4Weight.from_layer_group(p["layer"], names, p["code2"])  # noqa: E731
        s["w_qkv"], s["w_gu"] = group("q_proj", "k_proj", "v_proj"), group("gate_proj", "up_proj")
        s["w_o"], s["w_down"] = (linear.Nf4Weight.from_layer(p["layer"], n, p["code2"]) for n in ("o_proj", "down_proj"))
        s["bias"] = torch.cat([p["bias"][n] for n in ("q_proj", "k_proj", "v_proj")])
        s["segments"] = [(hidden, d.lora(hidden, hidden), None, 1.0), (kv, None, None, 1.0), (kv, d.lora(kv, hidden), None, 1.0)]
        # what the norms and the attention between the projections hand over
        s["x"], s["attn"], s["x2"] = (d.normal(M, hidden, dtype=torch.float16) for _ in range(3))
        if case["graph"]:
            side = torch.cuda.Stream(d.dev)
            side.wait_stream(torch.cuda.current_stream(d.dev))
            with torch.cuda.stream(side):
                _decode_layer(s)
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=side):
                    s["outputs"] = _decode_layer(s)
            torch.cuda.current_stream(d.dev).wait_stream(side)
            s["graph"] = graph
    elif kind == "mlp":
        hidden, inter, M = case["hidden"], case["inter"], case["M"]
        s["bucket"] = blocks.GradBucket(blocks.MlpBlock.grad_numel(hidden, inter), d.dev)
        s["block"] = blocks.MlpBlock(hidden, inter, seed=int(seed), device=d.dev, lora=True, bucket=s["bucket"])
        s["x"], s["dy"] = d.normal(M, hidden, dtype=torch.float16), d.normal(M, hidden, dtype=torch.float16)
        s["masks"] = [d.mask(M, k) for k in (hidden, hidden, inter)]
    elif kind in ("prefill", "stack"):
        hidden, kv, inter = case["hidden"], case["kv"], case["inter"]
        s["seq"] = _seq(case)
        M = sum(s["seq"])
        parts = [d.layer_parts(hidden, kv, inter) for _ in range(case.get("layers", 1))]
        s["stack"] = stack.NormedStack(hidden, inter, kv, len(parts), d.dev, layer_parts=parts, n_heads=hidden // HEAD)
        s["x"] = d.normal(M, hidden)
        if kind == "prefill":
            s["masks"] = [{} for _ in parts]
        else:
            s["masks"] = [d.layer_masks(M, hidden) for _ in parts]
            s["dres"] = d.normal(M, hidden, std=0.1)
            s["leaves"] = [t.requires_grad_(True) for t in s["stack"].lora_masters()] + [s["x"].requires_grad_(True)]
    elif kind == "projections":
        hidden, kv, inter, M = case["hidden"], case["kv"], case["inter"], case["M"]
        s["stack"] = stack.ProjectionStack(hidden, inter, kv, 1, d.dev, layer_parts=[d.layer_parts(hidden, kv, inter)])
        s["x"], s["dy"] = d.normal(M, hidden, dtype=torch.float16), d.normal(M, hidden, std=0.1, dtype=torch.float16)
        s["masks"] = [d.layer_masks(M, hidden)]
    elif kind == "dequant":
        p = d.layer_parts(case["hidden"], case["kv"], case["inter"])
        s["layer"], s["code2"] = p["layer"], p["code2"]
        s["nf4"] = torch.tensor(k_nf4.NF4_CODE, dtype=torch.float32, device=d.dev)
        s["out"] = torch.empty(p["layer"].numel, dtype=torch.float16, device=d.dev)
    else:
        raise ValueError(f"unknown kind {kind}")
    return s


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def _decode_layer(s):
    qkv, t = linear.forward_multi(s["w_qkv"], s["x"], s["segments"], bias=s["bias"])
    o, _ = linear.forward(s["w_o"], s["attn"])
    g, u, h, _, _ = linear.forward_gate_up(s["w_gu"], s["x2"])
    y, _ = linear.forward(s["w_down"], h)
    return [qkv, t[0], t[2], o, g, u, h, y]


def run(s):
    kind = s["kind"]
    if kind == "linear":
        return linear.forward(s["w"], s["x"], bias=s["bias"], lora=s["lora"])[0]
    if kind == "decode":
        if "graph" in s:
            s["graph"].replay()
            return s["outputs"]
        return _decode_layer(s)
    if kind == "autograd":
        y = linear.nf4_lora_linear(s["x"], s["w"], lora=(s["A"], s["B"], 2.0), mask=s["mask"], keep_scale=KEEP_SCALE)
        return [y, *torch.autograd.grad(y, (s["x"], s["A"], s["B"]), s["dy"])]
    if kind == "mlp":
        y = s["block"].forward(s["x"], s["masks"], KEEP_SCALE)
        return [y, s["block"].backward(s["dy"]), s["bucket"].flat]
    if kind == "prefill":
        with torch.no_grad():
            return s["stack"].forward(s["x"], s["masks"], 1.0, s["seq"])
    if kind == "stack":
        out = s["stack"].apply(s["x"], s["masks"], KEEP_SCALE, s["seq"])
        return [out, *torch.autograd.grad(out, s["leaves"], s["dres"])]
    if kind == "projections":
        out, dx = s["stack"].step(s["x"], s["dy"], s["masks"], KEEP_SCALE, need_input_grad=True)
        return [out, dx, s["stack"].bucket.flat]
    return k_nf4.dequant_layer(s["layer"], s["code2"], s["nf4"], s["out"])


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _attention_flops(lengths, hidden, backward):
    """Causal attention: two products of n (n + 1) / 2 x hidden each, five more halves of them in the backward."""
    pairs = sum(n * (n + 1) // 2 for n in lengths)
    return pairs * hidden * (4 + (10 if backward else 0))


def work(case):
    kind = case["kind"]
    if kind in ("linear", "autograd"):
        N, K, M = case["N"], case["K"], case["M"]
        lora = kind == "autograd" or case["lora"]
        factors = RANK * (N + K)
        nbytes = N * K * BYTES_PER_WEIGHT + 2 * M * (N + K) + (2 * factors if lora else 0) + (2 * N if case.get("bias") else 0)
        flops = 2 * M * (N * K + (factors if lora else 0))
        if kind == "autograd":       # x, mask and dy in, y and dx out, fp32 factors in and gradients out; weights once
            nbytes = N * K * BYTES_PER_WEIGHT + 4 * M * (N + K) + M * K + 8 * factors
            flops = 4 * M * N * K + 6 * M * factors
        return {"bytes": nbytes, "flops": flops}
    hidden, inter = case["hidden"], case["inter"]
    if kind == "mlp":
        M = case["M"]
        factors = 3 * RANK * (hidden + inter)
        weights = 3 * hidden * inter
        return {"bytes": weights * BYTES_PER_WEIGHT + M * (8 * hidden + 2 * hidden + inter) + 6 * factors,
                "flops": 4 * M * weights + 6 * M * factors}
    kv = case["kv"]
    weights = sum(n * k for n, k in _layer_shapes(hidden, kv, inter).values())
    factors = RANK * (2 * hidden + hidden + kv)
    if kind == "dequant":
        return {"bytes": weights * (BYTES_PER_WEIGHT + 2), "flops": 2 * weights}
    if kind == "decode":
        M = case["M"]
        return {"bytes": weights * BYTES_PER_WEIGHT + 2 * factors + 2 * M * (3 * hidden + hidden + 2 * kv + hidden + 3 * inter + hidden),
                "flops": 2 * M * (weights + factors)}
    if kind == "prefill":
        M = sum(_seq(case))
        return {"bytes": weights * BYTES_PER_WEIGHT + 2 * factors + 8 * M * hidden,
                "flops": 2 * M * (weights + factors) + _attention_flops(_seq(case), hidden, False)}
    if kind == "projections":
        M = case["M"]
        return {"bytes": weights * BYTES_PER_WEIGHT + M * hidden * (8 + 2) + 6 * factors,
                "flops": 4 * M * weights + 6 * M * factors}
    layers, M = case["layers"], sum(_seq(case))
    return {"bytes": layers * (weights * BYTES_PER_WEIGHT + 2 * M * hidden + 8 * factors) + 16 * M * hidden,
            "flops": layers * (4 * M * weights + 6 * M * factors + _attention_flops(_seq(case), hidden, True))}


def tolerance(case):
    """Activations are fp16 (unit roundoff 4.9e-4). One product: its output's rounding and the rounding of a scaled
    4-bit level, each a few 1e-4 in the 2-norm. Chains add one such term per stored activation on the way to a result."""
    kind = case["kind"]
    if kind == "dequant":
        return "exact"
    if kind in ("linear", "autograd"):
        return {"rel": 1.5e-3}
    if kind == "decode":
        return {"rel": 2e-3}
    if kind in ("mlp", "prefill", "projections"):
        return {"rel": 3e-3}
    return {"rel": 6e-3}
