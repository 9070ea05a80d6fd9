"""The work that users of this package have it do, as cases that can be timed and compared.

Two entry points are covered: the operator `ssd.bi.ssd_combined.bimamba_chunk_scan_combined` and the layer
`ssd.modules.BiMamba2`, each forward only (inference) and forward + backward (training).  A case is a dict of plain
values:

  kind      "scan" (the operator) or "layer" (BiMamba2)
  train     forward + backward, else forward under no_grad
  dtype     of the activations: "bf16", "fp16" or "fp32"
  batch, seqlen, nheads, headdim, ngroups, dstate, chunk    sizes; a layer has d_model = nheads * headdim / 2
  z, D, bias, dt    scan only: gate given or not; D per "head", per "channel" or "none"; dt_bias given or not; dt as
            fp32 "logits" (softplus inside the operator) or "steps" (already positive, used as given)
  mem_eff   layer only: the single-node path that recomputes instead of saving
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.abspath("bi-mamba2_b200")          # the package's folder is no importable name: its parent is put on the path
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_WIDTH = 7                                            # BiMamba2's default convolution


def _scan(name, train, dtype, batch, seqlen, nheads, headdim, ngroups, dstate, chunk, z=False, D="head", bias=True, dt="logits"):
    case = dict(kind="scan", train=train, dtype=dtype, batch=batch, seqlen=seqlen, nheads=nheads, headdim=headdim,
                ngroups=ngroups, dstate=dstate, chunk=chunk, z=z, D=D, bias=bias, dt=dt)
    return dict(case, name=name) if name else case


def _layer(name, train, batch, seqlen, nheads, dstate, chunk=256, mem_eff=False):
    case = dict(kind="layer", train=train, dtype="bf16", batch=batch, seqlen=seqlen, nheads=nheads, headdim=64, ngroups=1,
                dstate=dstate, chunk=chunk, mem_eff=mem_eff)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest call: fp32, four small heads, one short sequence; latency and launches are all there is
        _scan("fp32_tiny_train", True, "fp32", 1, 256, 4, 32, 1, 16, 64),
        # the small fp32 heads the operator's published plots use, at their longest sequence
        _scan("fp32_small_heads_train", True, "fp32", 2, 8192, 4, 16, 4, 16, 128, z=True, bias=False),
        # one short prompt scored in bf16
        _scan("bf16_short_infer", False, "bf16", 1, 384, 8, 64, 2, 64, 128, bias=False),
        # encoding a few medium sequences of a length that is no multiple of the chunk
        _scan("bf16_ragged_infer", False, "bf16", 3, 1777, 24, 64, 1, 128, 256, z=True),
        # training step on one sequence of odd length
        _scan("bf16_ragged_train", True, "bf16", 1, 1021, 24, 64, 1, 128, 256, z=True),
        # training step of a 24-head layer: the benchmark's default workload
        _scan("bf16_24_heads_train", True, "bf16", 8, 2048, 24, 64, 1, 128, 256, z=True),
        # training on long sequences with eight groups and D per channel, the share of one of eight devices
        _scan("bf16_long_groups_train", True, "bf16", 2, 8192, 32, 64, 8, 128, 256, D="channel", bias=False),
        # wide heads and a large state in fp16, dt used as given
        _scan("fp16_large_state_train", True, "fp16", 8, 1024, 16, 128, 2, 256, 128, z=True, D="channel", bias=False, dt="steps"),
        # the layer scoring one prompt of odd length
        _layer("layer_prompt_infer", False, 1, 733, 24, 128),
        # the layer's training step at a middling size, recomputing instead of saving
        _layer("layer_mem_eff_train", True, 2, 1536, 24, 128, mem_eff=True),
        # the layer's training step at full size: d_model 1024, 65 536 tokens
        _layer("layer_large_train", True, 16, 4096, 32, 64),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _cost(case):
    """Scan work in multiply-adds, roughly: keeps a drawn case no dearer than the largest listed one of its kind."""
    d = case
    per_token = d["nheads"] * d["headdim"] * (4 * d["dstate"] + d["chunk"]) + d["ngroups"] * d["chunk"] * d["dstate"]
    return d["batch"] * d["seqlen"] * per_token * (3 if d["train"] else 1)


def draw(rng):
    kind = rng.choice(["train16", "train16", "train16", "infer16", "infer16", "fp32", "fp32", "layer", "layer"])
    while True:
        if kind == "layer":
            case = _layer(None, rng.random() < 0.6, _log_int(rng, 1, 16), _log_int(rng, 200, 4096), rng.choice([8, 16, 24, 32]),
                          rng.choice([64, 128]), rng.choice([128, 256]), rng.random() < 0.3)
            most = 3 * 16 * 4096 * 32 * 64 * 512
        elif kind == "fp32":
            groups = rng.choice([1, 2, 4])
            heads = groups * rng.choice([1, 2, 4, 8])
            case = _scan(None, rng.random() < 0.7, "fp32", _log_int(rng, 1, 4), _log_int(rng, 100, 8192), heads,
                         rng.choice([16, 32, 64]), groups, rng.choice([16, 32, 64]), rng.choice([64, 128]),
                         z=rng.random() < 0.5, D=rng.choice(["head", "channel", "none"]), bias=rng.random() < 0.5,
                         dt=rng.choice(["logits", "logits", "steps"]))
            most = 3 * 2 * 8192 * 16 * 32 * 256
        else:
            groups = rng.choice([1, 1, 2, 4, 8])
            heads = max(8, groups * rng.choice([1, 2, 4, 8, 12, 16, 24]))
            headdim = rng.choice([64, 64, 64, 128])
            dstate = rng.choice([64, 128, 128, 256]) if headdim == 128 else rng.choice([64, 128, 128])
            case = _scan(None, kind == "train16", rng.choice(["bf16", "bf16", "fp16"]), _log_int(rng, 1, 8),
                         _log_int(rng, 100, 8192), heads, headdim, groups, dstate, 128 if dstate == 256 else rng.choice([128, 256]),
                         z=rng.random() < 0.5, D=rng.choice(["head", "channel"]), bias=rng.random() < 0.5,
                         dt=rng.choice(["logits", "logits", "steps"]))
            most = 3 * 2 * 8192 * 32 * 64 * 1024
        if case["nheads"] <= 64 and _cost(case) <= most:
            return case


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _DTYPES[case["dtype"]]
    b, L, H, P, G, N = (case[k] for k in ("batch", "seqlen", "nheads", "headdim", "ngroups", "dstate"))
    normal = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    uniform = lambda *shape: torch.rand(*shape, generator=gen, device="cuda")
    if case["kind"] == "layer":
        from ssd.modules import BiMamba2
        d_model = H * P // 2
        with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
            torch.manual_seed(seed)
            layer = BiMamba2(d_model, d_state=N, d_conv=_WIDTH, expand=2, headdim=P, ngroups=G, chunk_size=case["chunk"],
                             use_mem_eff_path=case["mem_eff"], device="cuda").to(dtype)
        u = normal(b, L, d_model).to(dtype)
        if not case["train"]:
            return dict(case=case, layer=layer.requires_grad_(False), u=u)
        params = [p for name, p in layer.named_parameters() if not name.startswith("fc_D")]      # fc_D takes no part in the layer
        return dict(case=case, layer=layer, leaves=[u.requires_grad_(True), *params], u=u, dout=normal(b, L, d_model).to(dtype))
    scale = 0.5 if dtype == torch.float16 else 1.0
    logits = case["dt"] == "logits"
    args = dict(x=(normal(b, L, H, P) * scale).to(dtype),
                dt=normal(b, L, H) - 4.0 if logits else uniform(b, L, H) * 0.099 + 0.001,
                A=-torch.exp(uniform(H) * math.log(16.0)),
                B=(normal(b, L, G, N) * scale).to(dtype), C=(normal(b, L, G, N) * scale).to(dtype))
    if case["D"] != "none":
        args["D"] = normal(H) if case["D"] == "head" else normal(H, P)
    if case["z"]:
        args["z"] = (normal(b, L, H, P) * scale).to(dtype)
    if case["bias"]:
        args["dt_bias"] = -uniform(H) if logits else 0.01 * uniform(H)
    state = dict(case=case, args=args, options=dict(chunk_size=case["chunk"], dt_softplus=logits))
    if case["train"]:
        state["leaves"] = [t.requires_grad_(True) for t in args.values()]
        state["dout"] = (normal(b, L, H, P) * scale).to(dtype)
    return state


def _call(state):
    if state["case"]["kind"] == "layer":
        return state["layer"](state["u"])
    from ssd.bi.ssd_combined import bimamba_chunk_scan_combined
    return bimamba_chunk_scan_combined(**state["args"], **state["options"])


def run(state):
    if not state["case"]["train"]:
        with torch.no_grad():
            return _call(state)
    out = _call(state)
    return [out, *torch.autograd.grad(out, state["leaves"], state["dout"])]


def work(case):
    """Bytes: every input read once, every output written once.  Flops: the products of the chunked form (states in and
    out of a chunk in both directions, the two products inside a chunk, C.B^T once a group; twice that again for the
    backward pass), and for a layer its two projections and its convolution."""
    b, L, H, P, G, N = (case[k] for k in ("batch", "seqlen", "nheads", "headdim", "ngroups", "dstate"))
    Q, tokens, train = min(case["chunk"], L), b * L, case["train"]
    size = _DTYPES[case["dtype"]].itemsize
    flops = tokens * (H * (8 * P * N + 2 * Q * P) + 2 * G * Q * N)
    if case["kind"] == "layer":
        inner, d_model = H * P, H * P // 2
        channels = inner + 2 * G * N
        weights = d_model * (inner + channels + H) + inner * d_model + channels * (_WIDTH + 1) + inner + 3 * H
        flops += 2 * tokens * (d_model * (inner + channels + H) + inner * d_model + channels * _WIDTH)
        nbytes = size * ((4 if train else 2) * tokens * d_model + (2 if train else 1) * weights)
    else:
        X, BC, DT = tokens * H * P, tokens * G * N, tokens * H
        z = 1 if case["z"] else 0
        nbytes = size * (X * ((4 + 2 * z) if train else (2 + z)) + 2 * BC * (2 if train else 1)) + 4 * DT * (2 if train else 1)
    return {"bytes": nbytes, "flops": flops * (3 if train else 1)}


def tolerance(case):
    """fp32: exponents are sums over a chunk and gradients are sums over all tokens.  16-bit: one rounding of an operand
    gives 4e-3 in bf16; in training the gradients of A, D and dt_bias are sums of mixed sign over all tokens, which no
    16-bit computation gets closer than about 2e-2 where heads are few."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-4}
    return {"rel": 2e-2 if case["train"] else 1e-2}
