"""The work that a user of this framework has it do, as cases to be timed.

Four kinds, each through the public entry points that a user's program calls:

  linear  one Linear on torch CUDA tensors (vai_b200.torch_linear.TorchLinear): a layer of a model whose other
          operators stay in PyTorch.
  block   the Linears of one transformer block on torch CUDA tensors, each fed with what such a program has at that
          point (q / k / v, the attention output + residual, gate|value with the gate, down + residual; the GPT-2
          block has its fused qkv and an ungated MLP).
  net     one step of a whole model's Linear nodes as a recorded net (vai_b200.NeuralNet, presets.build_linear_chain):
          host input in, host output back.
  head    the end of a sampling decoder as a recorded net: RmsNorm -> lm_head -> TopKSampling, which gives back the
          token and the logits.

Shapes are those of the presets (vai_b200/presets.py), of the tests, or generic.  Weights are N(0, 0.02) and activations
N(0, 1), made on the GPU from the seed; a net's input is host data, as in a user's program.
"""
import math

import numpy as np
import torch

import vai_b200
from vai_b200 import Dtype, Epilogue, Tensor, nodes, presets
from vai_b200.torch_linear import TorchLinear

TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
DT = {"f32": Dtype.F32, "f16": Dtype.F16, "bf16": Dtype.BF16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # The smallest call: the attention output projection of a GPT-2-small decode step (one row).
        {"name": "linear-decode-small", "kind": "linear", "M": 1, "K": 768, "N": 768, "io": "f32", "w": "f16", "bias": True,
         "residual": True, "act": "NONE", "gate": False},
        # fp32 end to end: the single GPT-2-small MLP Linear that the fp32 parity tests and the benchmark use.
        {"name": "linear-fp32-mlp", "kind": "linear", "M": 128, "K": 768, "N": 3072, "io": "f32", "w": "f32", "bias": True,
         "residual": False, "act": "GELU_TANH", "gate": False},
        # Ragged: 17 rows (a few prompts scored together) against GPT-2's vocabulary of 50257, an odd number of columns.
        {"name": "linear-ragged-head", "kind": "linear", "M": 17, "K": 768, "N": 50257, "io": "f32", "w": "f16", "bias": False,
         "residual": False, "act": "NONE", "gate": False},
        # The lm_head of a 64-stream decode step with Gemma's 262144-entry vocabulary.
        {"name": "linear-batch-head", "kind": "linear", "M": 64, "K": 2560, "N": 262144, "io": "bf16", "w": "bf16", "bias": False,
         "residual": False, "act": "NONE", "gate": False},
        # A short prompt (or one chunk of a long one) of a 1B model: one block, a row count that fits no tile.
        {"name": "block-chunk", "kind": "block", "preset": "llama-3.2-1b", "M": 333, "io": "bf16", "w": "bf16"},
        # Prefill of 4 x 2048 tokens of a 3B model: one block, the largest GEMMs.
        {"name": "block-prefill", "kind": "block", "preset": "llama-3.2-3b", "M": 8192, "io": "bf16", "w": "bf16"},
        # Greedy decode of a small model, one stream: fp16 weights and fp32 activations, the engine's defaults.
        {"name": "net-gpt2-decode", "kind": "net", "preset": "gpt2-small", "layers": 12, "M": 1, "io": "f32", "w": "f16", "head": True},
        # Prefill of a whole 1024-token context of the same model (the lm_head takes one row and is not part of it).
        {"name": "net-gpt2-prefill", "kind": "net", "preset": "gpt2-small", "layers": 12, "M": 1024, "io": "f32", "w": "f16", "head": False},
        # Decode of a 1B model, one stream: the benchmark's headline step.
        {"name": "net-llama1b-decode", "kind": "net", "preset": "llama-3.2-1b", "layers": 16, "M": 1, "io": "f32", "w": "bf16", "head": True},
        # The same model with eight streams decoded together (logits to the host are left to the head cases).
        {"name": "net-llama1b-batch8", "kind": "net", "preset": "llama-3.2-1b", "layers": 16, "M": 8, "io": "f32", "w": "bf16", "head": False},
        # Decode of a 4B model, 64 streams: all blocks.
        {"name": "net-gemma4b-batch64", "kind": "net", "preset": "gemma-3-4b", "layers": 34, "M": 64, "io": "bf16", "w": "bf16", "head": False},
        # The end of a sampling decoder: final norm, a 128256-entry vocabulary, top-40 sampling.
        {"name": "head-sample", "kind": "head", "M": 1, "K": 2048, "N": 128256, "w": "bf16", "k": 40},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "block", "block", "net", "net", "head"])
    if kind == "linear":
        io, w = rng.choice([("bf16", "bf16"), ("bf16", "bf16"), ("f32", "bf16"), ("f16", "f16"), ("f32", "f16"), ("f32", "f32")])
        if rng.random() < 0.5:         # a layer of one of the presets
            p = presets.PRESETS[rng.choice(sorted(presets.PRESETS))]
            _, K, N, ex = rng.choice(presets.block_linears(p) + [("lm_head", p["d"], p["vocab"], {})])
            gate, residual, bias = bool(ex.get("gate")), bool(ex.get("residual")), bool(ex.get("bias"))
            act = p["act"] if gate or ex.get("act") else "NONE"
        else:                          # a generic one; one in four has an inner size that no 16-byte vector divides
            K, N = _log(rng, 200, 12288), _log(rng, 10, 32768)
            if rng.random() < 0.75:
                K = (K + 7) // 8 * 8
            gate = rng.random() < 0.2
            N += N % 2 if gate else 0
            residual, bias = not gate and rng.random() < 0.3, rng.random() < 0.4
            act = rng.choice(["SILU", "GELU_TANH"]) if gate else rng.choice(["NONE", "NONE", "RELU", "GELU", "GELU_TANH", "SILU"])
        # 50 GFLOP where the tensor cores do not apply, 1 TFLOP elsewhere
        most = int((25e9 if w == "f32" or K % 8 else 5e11) / (K * N))
        M = _log(rng, 1, max(1, min(8192, most)))
        return {"kind": "linear", "M": M, "K": K, "N": N, "io": io, "w": w, "bias": bias, "residual": residual, "act": act, "gate": gate}
    if kind == "block":
        io, w = rng.choice([("bf16", "bf16"), ("bf16", "bf16"), ("f16", "f16"), ("f32", "f16")])
        return {"kind": "block", "preset": rng.choice(["gpt2-small", "llama-3.2-1b", "llama-3.2-3b", "gemma-3-4b"]), "M": _log(rng, 1, 6000),
                "io": io, "w": w}
    if kind == "net":
        preset, layers = rng.choice([("gpt2-small", 12), ("llama-3.2-1b", 16), ("llama-3.2-3b", 28), ("gemma-3-4b", 34)])
        M = _log(rng, 1, 1024 if preset == "gpt2-small" else 128)
        io, w = rng.choice([("f32", "f16"), ("f32", "bf16"), ("bf16", "bf16")])
        return {"kind": "net", "preset": preset, "layers": layers, "M": M, "io": io, "w": w, "head": M <= 2 and rng.random() < 0.5}
    return {"kind": "head", "M": rng.randint(1, 4), "K": rng.choice([768, 2048, 2560, 3072]), "N": rng.choice([50257, 128256, 262144, _log(rng, 10000, 262144)]),
            "w": rng.choice(["f16", "bf16"]), "k": rng.choice([1, 8, 40, 64])}


# ---- preparation -----------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _normal(g, shape, dtype, std=1.0):
    return torch.empty(shape, dtype=TORCH[dtype], device="cuda").normal_(0.0, std, generator=g)


class _Held:
    """Device memory of a torch tensor in the place of an engine buffer."""

    def __init__(self, t):
        self.t, self.ptr, self.nbytes, self.device = t, t.data_ptr(), t.numel() * t.element_size(), vai_b200.Device.default()


def _parameter(g, shape, dtype, std=0.02):
    t = Tensor(shape, DT[dtype])
    t.buffer = _Held(_normal(g, shape, dtype, std))
    return t


class _Given(dict):
    """The parameters of one Linear node of a chain, made before the chain."""

    def has_bias(self):
        return "bias" in self


def _host_input(g, shape, dtype):
    x = _normal(g, shape, dtype).cpu()
    return Tensor.from_numpy(x.numpy() if dtype == "f32" else x.view(torch.int16).numpy().view(np.uint16), dtype=DT[dtype])


def _prepare_linear(c, g):
    M, K, N = c["M"], c["K"], c["N"]
    out_n = N // 2 if c["gate"] else N
    lin = TorchLinear(_normal(g, (N, K), c["w"], 0.02), _normal(g, (N,), c["w"]) if c["bias"] else None,
                      epilogue=getattr(Epilogue, c["act"]), gate_fuse=c["gate"], device=vai_b200.Device.default())
    s = {"lin": lin, "x": _normal(g, (M, K), c["io"]), "res": _normal(g, (M, out_n), c["io"]) if c["residual"] else None}
    lin(s["x"], s["res"])                  # the plan and its workspace, which a program keeps
    return s


def _prepare_block(c, g):
    p, M = presets.PRESETS[c["preset"]], c["M"]
    calls = []
    for name, K, N, ex in presets.block_linears(p):
        gate = bool(ex.get("gate"))
        act = getattr(Epilogue, p["act"]) if gate or ex.get("act") else Epilogue.NONE
        lin = TorchLinear(_normal(g, (N, K), c["w"], 0.02), _normal(g, (N,), c["w"], 0.02) if ex.get("bias") else None, epilogue=act,
                          gate_fuse=gate, device=vai_b200.Device.default())
        calls.append((name, lin))
    s = {"calls": calls, "hidden": _normal(g, (M, p["d"]), c["io"]), "attention": _normal(g, (M, p["q"]), c["io"]),
         "normed": _normal(g, (M, p["d"]), c["io"])}
    _run_block(s)
    return s


def _prepare_net(c, g):
    p = presets.PRESETS[c["preset"]]
    given = []
    for _ in range(c["layers"]):
        for _, K, N, ex in presets.block_linears(p):
            one = _Given(weight=_parameter(g, (N, K), c["w"]))
            if ex.get("bias"):
                one["bias"] = _parameter(g, (N,), c["w"])
            given.append(one)
    if c["head"]:
        given.append(_Given(weight=_parameter(g, (p["vocab"], p["d"]), c["w"])))
    net = vai_b200.NeuralNet(w_default_dtype=DT[c["w"]], o_default_dtype=DT[c["io"]])
    presets.build_linear_chain(net, c["preset"], w_dtype=DT[c["w"]], layers=c["layers"], lm_head=c["head"], share_weights=given)
    s = {"net": net, "x": _host_input(g, (c["M"], p["d"]), c["io"]), "given": given}
    torch.cuda.synchronize()               # the parameters are in place before the net's own stream reads them
    net(s["x"])                            # the recording, which a program keeps
    return s


def _prepare_head(c, g):
    net = vai_b200.NeuralNet(w_default_dtype=DT[c["w"]])
    norm, head, pick = nodes.RmsNormNode(), nodes.LinearNode(in_dim=c["K"], out_dim=c["N"]), nodes.TopKSamplingNode(k=c["k"], temperature=0.8)
    norm["scale"] = _parameter(g, (c["K"],), "f32", 1.0)
    head["weight"] = _parameter(g, (c["N"], c["K"]), c["w"])
    net.input("x") - norm - head - pick - net.output("token")
    presets.Flow_of(head) - net.output("logits")
    u = float(torch.rand(1, generator=g, device="cuda"))
    s = {"net": net, "pick": pick, "u": u, "x": _host_input(g, (c["M"], c["K"]), "f32")}
    torch.cuda.synchronize()
    pick.set_uniform(u)
    net(s["x"])
    return s


def prepare(case, seed):
    g = _gen(seed)
    s = {"linear": _prepare_linear, "block": _prepare_block, "net": _prepare_net, "head": _prepare_head}[case["kind"]](case, g)
    s["kind"] = case["kind"]
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------

def _run_block(s):
    out, hidden = {}, s["hidden"]
    for name, lin in s["calls"]:
        if name == "o":
            out[name] = hidden = lin(s["attention"], residual=hidden)
        elif name in ("down", "fc2"):
            out[name] = lin(mid, residual=hidden)
        elif name in ("gate_up", "fc1"):
            out[name] = mid = lin(s["normed"])
        else:
            out[name] = lin(s["normed"])
    return out


def _floats(t):
    """A host output as floating-point values, without a copy."""
    if t.dtype == Dtype.F32:
        return t.host
    return torch.from_numpy(t.host.view(np.int16)).view(torch.float16 if t.dtype == Dtype.F16 else torch.bfloat16)


def run(s):
    if s["kind"] == "linear":
        return s["lin"](s["x"], s["res"])
    if s["kind"] == "block":
        return _run_block(s)
    if s["kind"] == "net":
        return _floats(s["net"](s["x"]))
    s["pick"].set_uniform(s["u"])
    out = s["net"](s["x"])
    return {"token": out["token"].to_u32(), "logits": _floats(out["logits"])}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------

def _act64(name, x):
    if name == "GELU_TANH":
        return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))
    return {"NONE": lambda t: t, "RELU": torch.relu, "SILU": torch.nn.functional.silu, "GELU": torch.nn.functional.gelu}[name](x)


def _linear64(x, w, bias=None, residual=None, act="NONE", gate=False, scale=1.0):
    y = x.double() @ w.double().t()
    if bias is not None:
        y = y + bias.double()
    if gate:
        h = y.shape[-1] // 2
        y = _act64(act, y[..., :h]) * y[..., h:]
    else:
        y = _act64(act, y)
    y = y * scale
    return y if residual is None else y + residual.double()


def exact(case, seed):
    """What run returns, in float64 from the stored operands (nothing between the layers is rounded); the operands are drawn
    in the order in which the preparations above draw them."""
    c, g = case, _gen(seed)
    if c["kind"] == "linear":
        M, K, N = c["M"], c["K"], c["N"]
        w, b = _normal(g, (N, K), c["w"], 0.02), _normal(g, (N,), c["w"]) if c["bias"] else None
        x, r = _normal(g, (M, K), c["io"]), _normal(g, (M, N // 2 if c["gate"] else N), c["io"]) if c["residual"] else None
        return _linear64(x, w, b, r, c["act"], c["gate"])
    if c["kind"] == "head":
        scale, w = _normal(g, (c["K"],), "f32", 1.0), _normal(g, (c["N"], c["K"]), c["w"], 0.02)
        torch.rand(1, generator=g, device="cuda")
        x = _normal(g, (c["M"], c["K"]), "f32").double()
        x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * scale.double()
        return {"token": None, "logits": _linear64(x, w).cpu()}
    p, M = presets.PRESETS[c["preset"]], c["M"]
    specs = presets.block_linears(p)

    def act_of(ex):
        return p["act"] if ex.get("gate") or ex.get("act") else "NONE"

    if c["kind"] == "block":
        given = {name: (_normal(g, (N, K), c["w"], 0.02), _normal(g, (N,), c["w"], 0.02) if ex.get("bias") else None) for name, K, N, ex in specs}
        hidden, attention, normed = (_normal(g, (M, n), c["io"]) for n in (p["d"], p["q"], p["d"]))
        out = {}
        for name, _, _, ex in specs:
            w, b = given[name]
            if name == "o":
                out[name] = hidden = _linear64(attention, w, b, hidden)
            elif name in ("down", "fc2"):
                out[name] = _linear64(mid, w, b, hidden)
            else:
                out[name] = _linear64(normed, w, b, None, act_of(ex), bool(ex.get("gate")))
                if name in ("gate_up", "fc1"):
                    mid = out[name]
        return out
    given = [[(_normal(g, (N, K), c["w"], 0.02), _normal(g, (N,), c["w"], 0.02) if ex.get("bias") else None) for _, K, N, ex in specs]
             for _ in range(c["layers"])]
    head = _normal(g, (p["vocab"], p["d"]), c["w"], 0.02) if c["head"] else None
    x = x0 = _normal(g, (M, p["d"]), c["io"]).double()
    for layer in given:
        made = {name: (w, b, act_of(ex), bool(ex.get("gate"))) for (name, _, _, ex), (w, b) in zip(specs, layer)}
        attention = _linear64(x, *made["q"][:2]) if p["gated"] else x
        h = _linear64(attention, *made["o"][:2], x0, scale=0.5)
        w, b, act, gate = made["gate_up" if p["gated"] else "fc1"]
        mid = _linear64(h, w, b, None, act, gate)
        x = _linear64(mid, *made["down" if p["gated"] else "fc2"][:2], x0, scale=0.25)
    return (x if head is None else _linear64(x, head)).cpu()


# ---- what a pass cannot do without, and how far two correct ones may differ --------------------------------------------

def _linear_work(M, K, N, io, w, bias, residual, gate):
    out = M * (N // 2 if gate else N) * SIZE[io]
    return N * K * SIZE[w] + M * K * SIZE[io] + out + (N * SIZE[w] if bias else 0) + (out if residual else 0), 2.0 * M * N * K


def work(case):
    c = case
    if c["kind"] == "linear":
        b, f = _linear_work(c["M"], c["K"], c["N"], c["io"], c["w"], c["bias"], c["residual"], c["gate"])
        return {"bytes": b, "flops": f}
    if c["kind"] == "head":
        b, f = _linear_work(c["M"], c["K"], c["N"], "f32", c["w"], False, False, False)
        return {"bytes": b, "flops": f}
    p = presets.PRESETS[c["preset"]]
    b = f = 0
    for _, K, N, ex in presets.block_linears(p):
        lb, lf = _linear_work(c["M"], K, N, c["io"], c["w"], ex.get("bias"), ex.get("residual"), ex.get("gate"))
        b, f = b + lb, f + lf
    if c["kind"] == "net":
        b, f = b * c["layers"], f * c["layers"]
        if c["head"]:
            lb, lf = _linear_work(c["M"], p["d"], p["vocab"], c["io"], c["w"], False, False, False)
            b, f = b + lb, f + lf
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times what the path differs by from itself with its sums in another order (other K splits, other row
    groups), measured over the listed cases and two dozen drawn ones; for fp32 sums, from float64."""
    c = case
    io, w = c.get("io", "f32"), c["w"]
    if c["kind"] == "linear":
        if io == "f32":
            # fp32 sums of exact products: 1.5e-7 at K = 768, growing with sqrt(K); up to 2e-6 where tensor cores add them up
            return {"rel": 8e-6, "max": 4e-5} if w != "f32" and c["M"] > 4 else {"rel": 2.5e-6, "max": 2.5e-5}
        # one rounding of the output differs now and then: 5e-5 (max one ulp, 9.7e-4) in fp16, 1.1e-4 (7.8e-3) in bf16
        return {"rel": 2e-4, "max": 4e-3} if io == "f16" else {"rel": 5e-4, "max": 3.2e-2}
    if c["M"] <= 4 and io == "f32":
        return {"rel": 1e-6, "max": 5e-6}          # fp32 activations all the way: 1.9e-7, 8e-7
    if c["kind"] == "block":
        # the gated activations are rounded, then summed: 6e-4 (1.6e-2) in bf16, an eighth of that in fp16
        return {"rel": 2.5e-3, "max": 6e-2} if "bf16" in (io, w) else {"rel": 3e-4, "max": 8e-3}
    # every layer's activations are rounded: 3e-3 (1.4e-2) with bf16 between the layers, 9e-4 (4.7e-3) with bf16 in the
    # multiplications alone, 2e-5 (1.2e-4) with fp16 there through 12 layers and about five times that in the wider models
    if io == "bf16":
        return {"rel": 1.2e-2, "max": 6e-2}
    return {"rel": 4e-3, "max": 2e-2} if w == "bf16" else {"rel": 5e-4, "max": 4e-3}
