"""Performance cases of the library: the operator calls of an AlphaFold2-style Evoformer, from one small call to the
1024-residue triangle attention.

A case is a dict of plain values; ``prepare`` makes its inputs on the GPU (or in pinned host memory for ``host``
cases), ``run`` is one pass through the public entry points of ``kutacc_b200.api`` and returns the outputs.

ops
  attention   pair-bias projection (where the layer has one) followed by the gated attention
              pair "own": the bias comes from the activations themselves (triangle attention, batch == seq);
              pair "z": from a pair tensor of its own [seq, seq, c_z] (MSA row attention); pair "none": no bias
              ln: the LayerNorm-fused entry points (activations arrive un-normalised)
              host: activations, mask and result live in host memory, as a caller of the CPU library holds them
  global      extra-MSA global column attention, 64 channels, 8 heads of 8
  transition  two-layer MLP with ReLU
  triangle    triangle multiplication: both projections, the per-channel product, the caller's channel-last copy with
              LayerNorm, gate and output linear, final gate
"""
import math

import torch

from kutacc_b200 import api

DEV = "cuda:0"
EPS = 1e-5


def _attention(name, batch, seq, heads, head_dim, dtype="bf16", pair="none", c_z=0, ln=False, host=False):
    case = {"op": "attention", "batch": batch, "seq": seq, "heads": heads, "head_dim": head_dim, "dtype": dtype, "pair": pair,
            "c_z": c_z, "ln": ln, "host": host}
    return dict(case, name=name) if name else case


def _named(name, **case):
    return dict(case, name=name) if name else case


def listed():
    return [
        # one short call of a small crop, all fixed costs: launches, descriptors, synchronisation-free queueing
        _attention("row_small", 4, 192, 4, 32, pair="z", c_z=128),
        # MSA row attention with pair bias of a caller that keeps fp32 activations
        _attention("msa_row_fp32", 128, 256, 8, 32, dtype="fp32", pair="z", c_z=128),
        # triangle attention of a long protein, and of a short one of any length: an odd residue count (rows that no
        # 16-byte load fits), LayerNorm in the same calls
        _attention("triangle_end_1024", 1024, 1024, 4, 32, pair="own", c_z=128),
        _attention("triangle_ln_301", 301, 301, 4, 32, pair="own", c_z=128, ln=True),
        # MSA column attention, no pair bias, and the same layer called with host buffers
        _attention("msa_col_512", 384, 512, 8, 32),
        _attention("msa_col_512_host", 384, 512, 8, 32, host=True),
        # narrow heads: pair stack with 64 channels (4 heads of 16), extra-MSA row attention (8 heads of 8)
        _attention("pair_c64_256", 256, 256, 4, 16, pair="own", c_z=64),
        _attention("extra_row_256", 256, 384, 8, 8, pair="z", c_z=128),
        # extra-MSA global column attention
        _named("extra_msa_global", op="global", batch=384, seq=5120),
        # pair transition; triangle multiplication of a 384-residue crop (incoming edges) and of an odd length (outgoing)
        _named("transition_384", op="transition", rows=384 * 384, channels=128, hidden=512),
        _named("triangle_mul_384", op="triangle", n=384, channels=128, incoming=True),
        _named("triangle_mul_301", op="triangle", n=301, channels=128, incoming=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["row", "row_fp32", "triangle", "triangle", "col", "col_host", "pair_c64", "extra_row", "global",
                       "transition", "triangle_mul"])
    if kind == "row":
        return _attention(None, _log_int(rng, 4, 512), _log_int(rng, 48, 512), rng.choice([4, 8]), 32, pair="z", c_z=128)
    if kind == "row_fp32":
        return _attention(None, _log_int(rng, 8, 128), _log_int(rng, 48, 384), 8, 32, dtype="fp32", pair="z", c_z=128)
    if kind == "triangle":
        n = _log_int(rng, 64, 1024)
        return _attention(None, n, n, 4, 32, pair="own", c_z=128, ln=rng.random() < 0.5)
    if kind == "col":
        return _attention(None, _log_int(rng, 48, 384), _log_int(rng, 32, 512), 8, 32)
    if kind == "col_host":
        return _attention(None, _log_int(rng, 48, 384), _log_int(rng, 64, 512), 8, 32, host=True)
    if kind == "pair_c64":
        n = _log_int(rng, 64, 384)
        return _attention(None, n, n, 4, 16, pair="own", c_z=64)
    if kind == "extra_row":
        return _attention(None, _log_int(rng, 16, 256), _log_int(rng, 48, 384), 8, 8, pair="z", c_z=128)
    if kind == "global":
        return {"op": "global", "batch": _log_int(rng, 16, 384), "seq": _log_int(rng, 128, 5120)}
    if kind == "transition":
        channels = rng.choice([128, 256])
        return {"op": "transition", "rows": _log_int(rng, 2048, 400 * 400), "channels": channels, "hidden": 4 * channels}
    return {"op": "triangle", "n": _log_int(rng, 64, 301), "channels": 128, "incoming": rng.random() < 0.5}


# ---- inputs ------------------------------------------------------------------------------------------
class _Random:
    """Seeded N(0, 1) activations, N(0, 1 / fan_in) weights."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed)

    def normal(self, *shape, dtype=torch.bfloat16, scale=1.0):
        return (torch.randn(*shape, generator=self.g, device=DEV) * scale).to(dtype)

    def weight(self, out, inp, dtype=torch.bfloat16):
        return self.normal(out, inp, dtype=dtype, scale=1.0 / math.sqrt(inp))

    def vector(self, n, mean=0.0, scale=0.1):
        return self.normal(n, dtype=torch.float32, scale=scale) + mean

    def keep(self, *shape, masked=0.05):
        return (torch.rand(*shape, generator=self.g, device=DEV) >= masked).to(torch.float32)


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _prepare_attention(case, r):
    b, s, h, d = case["batch"], case["seq"], case["heads"], case["head_dim"]
    c, dt = h * d, torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    place = _pinned if case["host"] else (lambda t: t)
    x = r.normal(b, s, c, dtype=dt)
    if case["ln"]:
        x = (x * (0.5 + 2 * torch.rand(b, s, 1, generator=r.g, device=DEV)) + r.normal(b, s, 1, dtype=dt)).to(dt)
    if case["pair"] == "own":                    # residue mask: 5 % of the residues absent, their rows fully masked
        keep = r.keep(s)
        mask = keep[:, None] * keep[None, :]
    elif case["pair"] == "z":
        mask = r.keep(b, s)
    else:                                        # column attention: 10 % of the sequences are padding
        mask = r.keep(s, masked=0.10)[None, :].expand(b, s)
    st = {"case": case, "x": place(x), "bias": place((1e9 * (mask - 1.0)).to(dt).contiguous())}
    for k in ("wq", "wk", "wv", "wg", "wo"):
        st[k] = place(r.weight(c, c, dt))
    st["bg"], st["bo"] = place(r.vector(c, mean=1.0)), place(r.vector(c))
    st["out"] = place(torch.zeros(b, s, c, dtype=dt, device=DEV))
    st["t_x"] = api.tensor(st["x"], sizes=[b * s, c], strides=[c, 1])
    st["t_bias"], st["t_out"] = api.tensor(st["bias"]), api.tensor(st["out"])
    st["inputs"] = api.make_inputs(b, s)
    st["weights"] = api.make_weights(c, h, d, *(st[k] for k in ("wq", "wk", "wv", "wg", "bg", "wo", "bo")))
    code = api.DTYPE_FP32 if case["dtype"] == "fp32" else api.DTYPE_BF16
    st["t_nb"] = api.empty_tensor(code)
    if case["pair"] != "none":
        st["z"] = st["x"] if case["pair"] == "own" else r.normal(s, s, case["c_z"], dtype=dt)
        st["wb"] = r.weight(h, case["c_z"], dt)
        st["nb"] = torch.zeros(h, s, s, dtype=dt, device=DEV)
        st["t_z"], st["t_wb"], st["t_nb"] = api.tensor(st["z"]), api.tensor(st["wb"]), api.tensor(st["nb"])
    if case["ln"]:
        st["gamma"], st["beta"] = r.vector(c, mean=1.0), r.vector(c)
    return st


def _prepare_global(case, r):
    b, s, c, d = case["batch"], case["seq"], 64, 8
    keep = torch.ones(b, s, device=DEV)
    keep[:, int(s * 0.8):] = 0.0                 # trailing 20 % of the rows are padding
    st = {"case": case, "x": r.normal(b, s, c), "mask": keep.to(torch.bfloat16)}
    ws = [r.weight(c, c), r.weight(d, c), r.weight(d, c), r.weight(c, c), r.vector(c, mean=1.0), r.weight(c, c), r.vector(c)]
    st["out"] = torch.zeros(b, s, c, dtype=torch.bfloat16, device=DEV)
    st["weights"], st["inputs"] = api.make_weights(c, 8, d, *ws), api.make_inputs(b, s)
    st["t_x"], st["t_mask"] = api.tensor(st["x"]), api.tensor(st["mask"], sizes=[b, s, 1], strides=[s, 1, 1])
    st["t_out"] = api.tensor(st["out"])
    return st


def _prepare_transition(case, r):
    m, c, hidden = case["rows"], case["channels"], case["hidden"]
    st = {"case": case, "out": torch.zeros(1, m, c, dtype=torch.bfloat16, device=DEV)}
    ts = [r.normal(1, m, c), r.weight(hidden, c), r.vector(hidden), r.weight(c, hidden), r.vector(c)]
    st["args"] = [api.tensor(t) for t in ts] + [api.tensor(st["out"])]
    return st


def _prepare_triangle(case, r):
    n, c = case["n"], case["channels"]
    keep = r.keep(n)
    st = {"case": case, "x": r.normal(n, n, c), "mask": (keep[:, None] * keep[None, :]).to(torch.bfloat16)}
    st["t_mask"] = api.tensor(st["mask"])
    for side in ("left", "right"):
        st[side], gate = (torch.zeros(c, n, n, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        st["acts_" + side] = api.make_tm_acts(n, n, st[side], st["x"], gate)
        st["w_" + side] = api.make_tm_proj_weights(c, c, r.weight(c, c), r.vector(c), r.weight(c, c), r.vector(c, mean=1.0))
        st["t_" + side] = api.tensor(st[side])
    st["center"] = torch.zeros(c, n, n, dtype=torch.bfloat16, device=DEV)
    for k in ("rows", "normed", "gate", "out"):
        st[k] = torch.zeros(n, n, c, dtype=torch.bfloat16, device=DEV)
        st["t_" + k] = api.tensor(st[k])
    st["t_center"] = api.tensor(st["center"])
    st["gamma"], st["beta"] = r.vector(c, mean=1.0), r.vector(c)
    st["acts"] = api.make_tm_acts(n, n, None, st["x"], None)
    st["w_out"] = api.make_tm_linear_weights(c, c, r.weight(c, c), r.vector(c, mean=1.0), r.weight(c, c), r.vector(c))
    return st


def prepare(case, seed):
    make = {"attention": _prepare_attention, "global": _prepare_global, "transition": _prepare_transition,
            "triangle": _prepare_triangle}[case["op"]]
    return make(case, _Random(seed))


# ---- one pass --------------------------------------------------------------------------------------------
def run(st):
    case = st["case"]
    # device-resident layers are queued one after another; a call with host buffers returns with its result
    api.set_async(not case.get("host", False))
    if case["op"] == "attention":
        if case["ln"]:
            gamma, beta = st["gamma"].data_ptr(), st["beta"].data_ptr()
            api.pair_bias_ln(st["t_z"], gamma, beta, EPS, st["t_wb"], st["t_nb"])
            api.gating_attention_ln(st["t_x"], st["inputs"], st["t_bias"], st["t_nb"], st["weights"], gamma, beta, EPS, st["t_out"])
        else:
            if case["pair"] != "none":
                api.pair_bias(st["t_z"], st["t_wb"], st["t_nb"])
            api.gating_attention(st["t_x"], st["inputs"], st["t_bias"], st["t_nb"], st["weights"], st["t_out"])
        return {"out": st["out"]} if case["pair"] == "none" else {"out": st["out"], "pair_bias": st["nb"]}
    if case["op"] == "global":
        api.global_attention(st["inputs"], st["t_x"], st["t_mask"], st["weights"], st["t_out"])
        return {"out": st["out"]}
    if case["op"] == "transition":
        api.transition(1, case["rows"], case["channels"], case["hidden"], *st["args"])
        return {"out": st["out"]}
    n, c = case["n"], case["channels"]
    for side in ("left", "right"):
        api.tm_calc_proj(st["acts_" + side], st["t_mask"], st["w_" + side])
    api.tm_equation(st["t_center"], st["t_left"], st["t_right"], n, case["incoming"])
    st["rows"].copy_(st["center"].permute(1, 2, 0))
    api.layernorm_rows(st["rows"].data_ptr(), st["gamma"].data_ptr(), st["beta"].data_ptr(), n * n, c, EPS, st["normed"].data_ptr())
    api.tm_gate_and_out_linear(st["t_gate"], st["t_out"], st["acts"], st["t_normed"], st["w_out"])
    api.tm_last(st["t_out"], st["t_gate"], n, n, c)
    return {"out": st["out"], "center": st["center"], "left": st["left"], "right": st["right"]}


# ---- what a pass cannot do without -------------------------------------------------------------------------
def work(case):
    """Compulsory bytes (inputs once, outputs once, weights) and flops (2 per multiply-add; exp and sigmoid not counted)."""
    if case["op"] == "attention":
        b, s, h, d = case["batch"], case["seq"], case["heads"], case["head_dim"]
        c, e = h * d, 4 if case["dtype"] == "fp32" else 2
        nbytes = e * (2.0 * b * s * c + 5.0 * c * c + b * s) + 8.0 * c
        flops = 10.0 * b * s * c * c + 4.0 * b * s * s * c
        if case["pair"] != "none":
            nbytes += e * (h * s * s + h * case["c_z"] + (s * s * case["c_z"] if case["pair"] == "z" else 0))
            flops += 2.0 * s * s * case["c_z"] * h
        return {"bytes": nbytes, "flops": flops}
    if case["op"] == "global":
        b, s, c, h, d = case["batch"], case["seq"], 64, 8, 8
        flops = 2.0 * b * s * c + 2.0 * b * c * c + 4.0 * b * s * c * d + 4.0 * b * s * h * d + 4.0 * b * s * c * c
        return {"bytes": 2.0 * (2 * b * s * c + b * s + 3 * c * c + 2 * c * d), "flops": flops}
    if case["op"] == "transition":
        m, c, hidden = case["rows"], case["channels"], case["hidden"]
        return {"bytes": 2.0 * (2 * m * c + 2 * c * hidden), "flops": 4.0 * m * c * hidden}
    n, c = case["n"], case["channels"]
    # left, right and center are results of entry points of their own; the product reads both projections
    return {"bytes": 2.0 * (n * n * c * 5 + n * n + 6 * c * c), "flops": 2.0 * n * n * c * c * 6 + 2.0 * c * float(n) ** 3}


def tolerance(case):
    # bf16 tensors: a handful of roundings to 8 bits on the way, softmax weights included. fp32: every product is
    # carried to fp32 accuracy; sums over up to 512 terms in another order, and the hardware exponential.
    if case.get("dtype") == "fp32":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 1e-2, "max": 0.25}
