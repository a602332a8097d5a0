"""Performance cases of the Mega EMA layer path, through the package's public entry points.

A case is a dict of plain values.  ``listed()`` names the representative ones, ``draw(rng)`` gives one more of the same
ranges; ``prepare`` builds what a user's program has in hand (modules, inputs, running state), ``run`` is one pass,
``work`` the bytes and operations a pass cannot do without, ``tolerance`` what another correct implementation at the same
precision may differ by.

Kinds
  step      one decoding step of TimestepNorm -> EMA on a running state (one token per sequence)
  ema       the EMA layer alone, causal, on time-major activations with right padding
  layer     TimestepNorm -> causal EMA forward over whole sequences; with ``state`` it is the prefill of a generation
            (running state exported), with ``normed`` the normalised activations come back too, as the Mega block asks
  encoder   SequenceNorm -> bidirectional EMA forward, right padding
  train     forward and backward of TimestepNorm -> EMA
  block     a causal Mega block (EMA, gates, chunked attention), inference over whole sequences
  generate  a causal Mega block serving one batch of requests: ragged prompt, then tokens one at a time
  btrain    a training pass (forward and backward) of a causal Mega block
  etrain    a training pass of a bidirectional Mega block on padded batches
"""
import math

import torch

import fairseq_apollo_b200 as M

NDIM = 16
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}


def listed():
    return [
        # interactive decoding: one sequence, one token; nothing but latency
        {"name": "step_single", "kind": "step", "dtype": "bf16", "batch": 1, "dim": 512, "complex": False},
        # batched decoding at the serving width of the long-context configuration
        {"name": "step_batched", "kind": "step", "dtype": "bf16", "batch": 64, "dim": 2048, "complex": False},
        # the EMA layer by itself in fp32, time-major, batch padded to its longest sequence
        {"name": "ema_padded_fp32", "kind": "ema", "dtype": "fp32", "batch": 8, "length": 1024, "dim": 512, "pad": 0.25},
        # the causal layer at an ordinary language-model shape
        {"name": "layer_lm", "kind": "layer", "dtype": "bf16", "batch": 16, "length": 4096, "dim": 1024, "complex": False,
         "pad": 0.0, "state": False, "normed": False},
        # long context: the largest forward pass of the path
        {"name": "layer_long", "kind": "layer", "dtype": "bf16", "batch": 64, "length": 32768, "dim": 2048,
         "complex": False, "pad": 0.0, "state": False, "normed": False},
        # prefill of ragged prompts with the complex-pole layer, as the Mega block calls it
        {"name": "prefill_complex", "kind": "layer", "dtype": "bf16", "batch": 6, "length": 4999, "dim": 2048,
         "complex": True, "pad": 0.0, "state": True, "normed": True},
        # bidirectional encoder layer on long padded fp32 sequences
        {"name": "encoder_long_fp32", "kind": "encoder", "dtype": "fp32", "batch": 32, "length": 16384, "dim": 256,
         "pad": 0.5},
        # training step of the causal layer
        {"name": "layer_train", "kind": "train", "dtype": "bf16", "batch": 16, "length": 4096, "dim": 1024,
         "complex": False, "pad": 0.0},
        # a language-model block, inference
        {"name": "block_lm", "kind": "block", "dtype": "bf16", "batch": 8, "length": 8192, "dim": 1024, "zdim": 256,
         "hdim": 2048, "chunk": 1024, "complex": False},
        # the same block answering requests: prompts shorter than a chunk, then token by token
        {"name": "block_generate", "kind": "generate", "dtype": "bf16", "batch": 4, "length": 700, "tokens": 32,
         "dim": 1024, "zdim": 256, "hdim": 2048, "chunk": 1024, "complex": False},
        # training of a causal block with complex poles and grouped statistics
        {"name": "block_train", "kind": "btrain", "dtype": "bf16", "batch": 4, "length": 4096, "dim": 1024, "zdim": 256,
         "hdim": 2048, "chunk": 1024, "complex": True, "groups": 32},
        # training of a bidirectional classifier block on padded batches
        {"name": "encoder_train", "kind": "etrain", "dtype": "bf16", "batch": 16, "length": 1024, "dim": 256, "zdim": 64,
         "hdim": 512, "chunk": -1, "complex": False, "pad": 0.25},
    ]


def _spread(rng, low, high, step=1):
    """Log-uniform multiple of ``step`` in [low, high]."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return min(high, max(low, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["step", "ema", "layer", "layer", "encoder", "train", "block", "generate", "btrain", "etrain"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp32", "fp16"])
    half = rng.choice(["bf16", "bf16", "fp16"])
    cplx = rng.random() < 0.4
    pad = round(rng.uniform(0.05, 0.5), 3) if rng.random() < 0.4 else 0.0
    if kind == "step":
        return {"kind": kind, "dtype": dtype, "batch": _spread(rng, 1, 96), "dim": _spread(rng, 128, 2048, 8),
                "complex": cplx}
    if kind == "ema":
        return {"kind": kind, "dtype": dtype, "batch": _spread(rng, 1, 32), "length": _spread(rng, 64, 4096),
                "dim": _spread(rng, 64, 1024, 8), "pad": pad}
    if kind == "layer":
        dim, length = _spread(rng, 128, 2048, 8), _spread(rng, 100, 32768)
        batch = _spread(rng, 1, max(1, min(64, (1 << 28) // (dim * length))))
        state = rng.random() < 0.4
        return {"kind": kind, "dtype": dtype, "batch": batch, "length": length, "dim": dim, "complex": cplx,
                "pad": 0.0 if state else pad, "state": state, "normed": rng.random() < 0.5}
    if kind == "encoder":
        dim, length = _spread(rng, 64, 512, 8), _spread(rng, 512, 16384)
        batch = _spread(rng, 1, max(1, min(32, (1 << 27) // (dim * length))))
        return {"kind": kind, "dtype": rng.choice(["fp32", "bf16"]), "batch": batch, "length": length, "dim": dim,
                "pad": pad}
    if kind == "train":
        dim, length = _spread(rng, 128, 2048, 8), _spread(rng, 200, 8192)
        batch = _spread(rng, 1, max(1, min(32, (1 << 26) // (dim * length))))
        return {"kind": kind, "dtype": dtype, "batch": batch, "length": length, "dim": dim, "complex": cplx, "pad": pad}
    dim = _spread(rng, 256, 1024, 64)
    zdim, hdim = rng.choice([64, 128, 256]), 2 * dim
    if kind in ("block", "btrain"):
        chunk = rng.choice([128, 256, 512, 1024])
        length = chunk * _spread(rng, 1, 8)
        batch = _spread(rng, 1, max(1, min(16, (1 << (25 if kind == "block" else 24)) // (dim * length))))
        case = {"kind": kind, "dtype": half, "batch": batch, "length": length, "dim": dim, "zdim": zdim, "hdim": hdim,
                "chunk": chunk, "complex": cplx}
        if kind == "btrain":
            case["groups"] = rng.choice([dim // 64, dim // 32])
        return case
    if kind == "generate":
        return {"kind": kind, "dtype": half, "batch": _spread(rng, 1, 16), "length": _spread(rng, 16, 900),
                "tokens": _spread(rng, 8, 64), "dim": dim, "zdim": zdim, "hdim": hdim, "chunk": 1024, "complex": cplx}
    dim = _spread(rng, 64, 512, 8)
    length = _spread(rng, 128, 2048)
    batch = _spread(rng, 1, max(1, min(32, (1 << 23) // (max(dim, length) * length))))
    return {"kind": "etrain", "dtype": "bf16", "batch": batch, "length": length, "dim": dim, "zdim": 64, "hdim": 2 * dim,
            "chunk": -1, "complex": cplx, "pad": pad}


# ------------------------------------------------------------------------------------------------ what a program has
def _activations(gen, dtype, *shape):
    """Activations of a trained model: near zero mean and unit scale, filled one leading slice at a time."""
    x = torch.empty(*shape, device="cuda", dtype=dtype)
    if x.numel() < 1 << 24:
        x.copy_(torch.randn(*shape, generator=gen, device="cuda") * 1.1 + 0.05)
    else:
        for row in x:
            row.normal_(0.05, 1.1, generator=gen)
    return x


def _padding(gen, batch, length, pad):
    """Right padding of up to ``pad`` of each sequence (the first one is full), or None."""
    if not pad:
        return None
    lost = (torch.rand(batch, generator=gen, device="cuda") * (pad * length)).long()
    lost[0] = 0
    return torch.arange(length, device="cuda").unsqueeze(0) >= (length - lost).unsqueeze(1)


def _trained(module):
    """Affine parameters and priors away from their initial constants, as after training."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            leaf = name.split(".")[-1]
            if leaf == "prior_mean" or (leaf in ("weight", "bias") and p.dim() == 1):
                p.normal_(0.0, 0.1)
            elif leaf == "prior_logv":
                p.normal_(0.0, 0.2)
            elif name in ("gamma", "beta") and hasattr(module, "mx_proj"):
                p.normal_(0.0, 0.5)
    return module


def _moving(case, bidirectional=False):
    layer = M.MultiHeadComplexEMA if case.get("complex") else M.MultiHeadEMA
    return layer(case["dim"], ndim=NDIM, bidirectional=bidirectional)


def _block(case):
    c = case
    common = dict(chunk_size=c["chunk"], moving_layer="cema" if c["complex"] else "ema", moving_act="silu")
    if c["kind"] == "etrain":
        blk = M.MovingAverageGatedAttention(c["dim"], c["zdim"], c["hdim"], NDIM, bidirectional=True,
                                            rel_pos_bias="simple", max_positions=c["length"], **common)
    else:
        blk = M.MovingAverageGatedAttention(c["dim"], c["zdim"], c["hdim"], NDIM, efficient_attn=True,
                                            rel_pos_bias="rotary", norm_num_groups=c.get("groups"), **common)
    return _trained(blk).to(DTYPES[c["dtype"]])


def prepare(case, seed):
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    batch, dim, length = case["batch"], case["dim"], case.get("length")
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    s = {"case": case, "mask": None}
    with torch.device("cuda"):
        if kind in ("block", "generate", "btrain", "etrain"):
            s["block"] = _block(case)
        elif kind == "encoder":
            s["norm"], s["move"] = _trained(M.SequenceNorm(dim)), _moving(case, bidirectional=True)
        else:
            s["norm"], s["move"] = _trained(M.TimestepNorm(dim, prior_count=2)), _moving(case)
    for name in ("norm", "move", "block"):
        if name in s:
            s[name].train(kind in ("train", "btrain", "etrain"))
    if kind == "step":
        s["inc"] = {}
        with torch.no_grad():   # the state that a prompt left
            M.timestep_norm_ema(s["norm"], s["move"], _activations(gen, dtype, batch, 64, dim), None, s["inc"])
        s["x"] = _activations(gen, dtype, batch, 1, dim)
    elif kind == "ema":
        s["x"] = _activations(gen, dtype, length, batch, dim)
        s["mask"] = _padding(gen, batch, length, case["pad"])
    elif kind == "encoder":
        s["x"] = _activations(gen, dtype, batch, dim, length)
        s["mask"] = _padding(gen, batch, length, case["pad"])
    elif kind == "generate":
        s["x"] = _activations(gen, dtype, batch, length, dim)
        s["next"] = list(_activations(gen, dtype, case["tokens"], batch, 1, dim))
    else:
        s["x"] = _activations(gen, dtype, batch, length, dim)
        s["mask"] = _padding(gen, batch, length, case.get("pad", 0.0))
    if kind in ("train", "btrain", "etrain"):
        s["x"].requires_grad_(True)
        s["dy"] = torch.randn(batch, length, dim, generator=gen, device="cuda").to(dtype)
    return s


# ----------------------------------------------------------------------------------------------------------- one pass
def _running_state(inc):
    """The tensors of an incremental state under their published names."""
    return {"%s.%s" % (key.split(".")[-1], name): v for key, buf in inc.items() for name, v in buf.items()
            if v is not None}


def _backward(s, modules, out):
    out.backward(s["dy"])
    grads = {"%d.%s" % (i, n): p.grad for i, m in enumerate(modules) for n, p in m.named_parameters()}
    return {"y": out.detach(), "dx": s["x"].grad, "grads": grads}


def _zero_grad(s, modules):
    s["x"].grad = None
    for m in modules:
        m.zero_grad(set_to_none=True)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        _zero_grad(s, (s["norm"], s["move"]))
        return _backward(s, (s["norm"], s["move"]), M.timestep_norm_ema(s["norm"], s["move"], s["x"], s["mask"]))
    if kind in ("btrain", "etrain"):
        _zero_grad(s, (s["block"],))
        return _backward(s, (s["block"],), s["block"](s["x"], s["mask"])[0])
    with torch.no_grad():
        if kind == "step":
            y = M.timestep_norm_ema(s["norm"], s["move"], s["x"], None, s["inc"])
            return {"y": y, "state": _running_state(s["inc"])}
        if kind == "ema":
            return s["move"].forward_time_major(s["x"], s["mask"])
        if kind == "layer":
            inc = {} if case["state"] else None
            act = "silu" if case["normed"] else None
            out = M.timestep_norm_ema(s["norm"], s["move"], s["x"], s["mask"], inc, act, case["normed"])
            return {"y": out, "state": _running_state(inc) if inc is not None else None}
        if kind == "encoder":
            return M.sequence_norm_ema(s["norm"], s["move"], s["x"], s["mask"])
        if kind == "block":
            return s["block"](s["x"])[0]
        inc = {}
        ys = [s["block"](s["x"], incremental_state=inc)[0]]
        for token in s["next"]:
            ys.append(s["block"](token, incremental_state=inc)[0])
        return {"y": torch.cat(ys, 1), "state": _running_state(inc)}


# ------------------------------------------------------------------------------------------------------ what it costs
def work(case):
    kind, es = case["kind"], SIZE[case["dtype"]]
    batch, dim = case["batch"], case["dim"]
    tokens = batch * case.get("length", 1)
    cplx = case.get("complex", False)
    sides = 2 if kind in ("encoder", "etrain") else 1
    pole = 14 if cplx else 4                          # state update and output sum, per pole and position
    coeffs = 4.0 * dim * NDIM * (5 if cplx else 3) * sides
    state = 4.0 * batch * dim * NDIM * (2 if cplx else 1)
    scan = float(tokens) * dim * NDIM * pole * sides
    if kind == "step":
        return {"bytes": 2.0 * state + 4 * 4.0 * batch * dim + coeffs + 2.0 * batch * dim * es, "flops": scan}
    if kind == "ema":
        return {"bytes": 2.0 * tokens * dim * es + coeffs, "flops": scan}
    if kind == "layer":
        moved = (3.0 if case["normed"] else 2.0) * tokens * dim * es
        return {"bytes": moved + coeffs + (state if case["state"] else 0.0), "flops": scan + 10.0 * tokens * dim}
    if kind == "encoder":
        return {"bytes": 2.0 * tokens * dim * es + coeffs, "flops": scan + 10.0 * tokens * dim}
    if kind == "train":
        return {"bytes": 4.0 * tokens * dim * es + 2 * coeffs, "flops": 4.0 * scan + 30.0 * tokens * dim}
    z, h = case["zdim"], case["hdim"]
    weights = dim * h + dim * (z + h + 2 * dim) + h * dim
    if kind == "generate":
        new, prompt = case["tokens"], case["length"]
        seen = prompt * (prompt + 1) / 2 + new * prompt + new * (new + 1) / 2
        flops = batch * (prompt + new) * (2.0 * weights + dim * NDIM * pole) + 2.0 * batch * seen * (z + h)
        cache = batch * (z + h) * es * (new * prompt + new * (new + 1) / 2.0)
        moved = 2.0 * batch * (prompt + new) * dim * es + (new + 1) * (weights * es + coeffs + 2.0 * state)
        return {"bytes": moved + cache, "flops": flops}
    span = case["length"] if case["chunk"] < 0 else min(case["chunk"], case["length"])
    pairs = tokens * span * (1.0 if kind == "etrain" else 0.5)
    flops = 2.0 * tokens * weights + 2.0 * pairs * (z + h) + scan
    if kind == "block":
        return {"bytes": 2.0 * tokens * dim * es + weights * es + coeffs, "flops": flops}
    return {"bytes": 4.0 * tokens * dim * es + 2.0 * weights * es + 2 * coeffs, "flops": 3.0 * flops}


def tolerance(case):
    """Relative 2-norm.  fp32: sums of 32-bit values (gradients add over batch and length).  16-bit: one rounding of
    the result is 2^-9 (bf16) or 2^-12 (fp16), and a layer rounds operands and intermediate activations a few times.
    Through a block's attention the gradients of the query / key affine and of the relative bias are sums of weight
    gradients that cancel: each bf16 implementation is 1e-2 to 2e-2 off the fp32 result there, fp16 an eighth of that."""
    kind, dtype = case["kind"], case["dtype"]
    if dtype == "fp32":
        return {"rel": 5e-5 if kind == "train" else 1e-5}
    if kind in ("btrain", "etrain"):
        return {"rel": 3e-2 if dtype == "bf16" else 5e-3}
    return {"rel": 1e-2 if dtype == "bf16" else 2e-3}
