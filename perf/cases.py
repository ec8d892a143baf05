"""The work a user of this library has it do, as cases that can be prepared, run once and compared.

Three families, each through the entry points a user's program calls:
  stack : tokens through a run of MoE feed-forward layers at the Gemma-4-26B-A4B geometry (MoeEngine), in the decode
          arithmetic (one token, draft-verify and batched decode) or the prefill arithmetic (prompts);
  gemm  : the quantised GEMM with per-row and per-column scales (int_gemm_scaled), int8 or packed int4;
  hook  : the plugin hook of a host program with its own router (MoeExt), once per layer of its model.
"""
import math

import numpy as np
import torch

from kairos_engine_b200 import FLAVOUR_DECODE, FLAVOUR_PREFILL, GEMMA4_26B_A4B, MoeEngine, MoeExt, q4b_quantize, synth
from kairos_engine_b200.engine import int_gemm_scaled

MODEL_LAYERS = 30
DISTINCT_LAYERS = 3      # the stack cycles this many seeded layers; every layer has its own copy in device memory


def _stack(name, flavour, tokens, entry, layers=MODEL_LAYERS, zipf=False):
    return {"name": name, "kind": "stack", "flavour": flavour, "tokens": tokens, "layers": layers, "entry": entry, "zipf": zipf}


def listed():
    return [
        # one decode step of the whole stack, inputs and results in device memory: the benchmark's headline
        _stack("decode 1", "decode", 1, "device"),
        # the same step as an engine does it that has attention between the layers: one call per layer
        _stack("decode 1 by layer", "decode", 1, "layers"),
        # a draft of five tokens verified by a host program that wants the routing too
        _stack("verify 5 from host", "decode", 5, "host"),
        # batched decode: a few sequences, and the largest batch that is served as one step
        _stack("decode 16", "decode", 16, "device"),
        _stack("decode 64", "decode", 64, "device"),
        # prompts: a short question, an ordinary one of no round length, the benchmark's 4096 tokens
        _stack("prefill 37", "prefill", 37, "device"),
        _stack("prefill 717", "prefill", 717, "device"),
        _stack("prefill 4096", "prefill", 4096, "device"),
        # the load-imbalance stress: a Zipf(1.2) bias on the router sends nearly all tokens to the same few experts
        _stack("prefill 512 zipf", "prefill", 512, "device", zipf=True),
        # the quantised GEMM at the size its acceptance gate names, and a small ragged one of packed int4 operands
        {"name": "gemm int8", "kind": "gemm", "bits": 8, "m": 3072, "k": 8192, "n": 3072},
        {"name": "gemm int4 ragged", "kind": "gemm", "bits": 4, "m": 513, "k": 1040, "n": 1000},
        # the smallest calls: one token through the hook, host vectors in and out, at the expert shape of its tests
        {"name": "hook", "kind": "hook", "layers": 8, "experts": 32, "used": 8, "e": 2048, "ff": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "prefill", "gemm", "hook"])
    if what == "decode":
        entry = rng.choice(["device", "device", "host", "layers"])
        c = _stack("", "decode", _log_int(rng, 1, 64), entry, layers=rng.randint(8, MODEL_LAYERS))
    elif what == "prefill":
        c = _stack("", "prefill", _log_int(rng, 24, 4096), rng.choice(["device", "device", "host", "layers"]),
                   layers=rng.randint(8, MODEL_LAYERS), zipf=rng.random() < 0.25)
    elif what == "gemm":
        c = {"kind": "gemm", "bits": rng.choice([8, 4]), "m": _log_int(rng, 16, 4096), "k": 16 * _log_int(rng, 16, 512),
             "n": _log_int(rng, 64, 4096)}
    else:
        c = {"kind": "hook", "layers": rng.randint(4, 12), "experts": rng.randint(16, 48), "used": rng.randint(2, 8),
             "e": 32 * rng.randint(16, 88), "ff": 32 * rng.randint(8, 24)}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- what the program has in hand before the call
def _prepare_stack(case, seed):
    cfg, M, n = GEMMA4_26B_A4B, case["tokens"], case["layers"]
    eng = MoeEngine(n_layers=n, max_tokens=M, **cfg)
    bias = synth.zipf_bias(cfg["NE"], 1.2, seed) if case["zipf"] else None
    for k in range(min(DISTINCT_LAYERS, n)):
        layer = synth.make_layer(cfg, seed + 1000 * k, rand_norms=True, bias=bias)
        for L in range(k, n, DISTINCT_LAYERS):
            eng.upload_layer(L, layer, on_device=True)
        del layer
    x = synth.make_inputs(cfg, M, seed + 7)
    torch.cuda.synchronize()
    state = {"case": case, "eng": eng, "flavour": FLAVOUR_DECODE if case["flavour"] == "decode" else FLAVOUR_PREFILL}
    if case["entry"] == "host":
        state["x"], state["y"] = x.cpu().pin_memory().numpy(), torch.empty(M, cfg["E"]).pin_memory().numpy()
    else:
        state["x"], state["bufs"] = x, [torch.empty_like(x), torch.empty_like(x)]
    return state


def _prepare_gemm(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    m, k, n = case["m"], case["k"], case["n"]
    if case["bits"] == 8:
        A, B = (torch.randint(-127, 128, (r, k), dtype=torch.int8, device="cuda", generator=g) for r in (m, n))
    else:
        A, B = (torch.randint(0, 256, (r, k // 2), dtype=torch.uint8, device="cuda", generator=g) for r in (m, n))
    sa, sb = (torch.rand(r, device="cuda", generator=g) * 1e-3 + 1e-4 for r in (m, n))
    return {"case": case, "A": A, "B": B, "sa": sa, "sb": sb}


def _prepare_hook(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    NE, FF, E = case["experts"], case["ff"], case["e"]
    rng = np.random.default_rng(seed)
    ext, calls = MoeExt(), []
    for L in range(case["layers"]):
        w = []
        for rows, cols in ((NE * FF, E), (NE * FF, E), (NE * E, FF)):
            codes, bs = q4b_quantize(torch.randn((rows, cols), generator=g, device="cuda") * 0.05)
            w += [codes.cpu().numpy(), bs.cpu().numpy().view(np.uint16)]
        tag = "blk.%d.ffn_gate_exps.weight" % L
        ext.upload_experts(tag, *w, NE, FF, E)
        wt = rng.random(case["used"]).astype(np.float32)
        calls.append((tag, rng.choice(NE, case["used"], replace=False).astype(np.int32), wt / wt.sum(),
                      rng.standard_normal(E).astype(np.float32), FF))
    return {"case": case, "ext": ext, "calls": calls}


def prepare(case, seed):
    return {"stack": _prepare_stack, "gemm": _prepare_gemm, "hook": _prepare_hook}[case["kind"]](case, seed)


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "gemm":
        return int_gemm_scaled(state["A"], state["B"], state["sa"], state["sb"], packed_int4=case["bits"] == 4)
    if case["kind"] == "hook":
        return [state["ext"].moe(*call) for call in state["calls"]]
    eng, x, flavour = state["eng"], state["x"], state["flavour"]
    if case["entry"] == "host":
        y, sel, wts = eng.forward(x, flavour=flavour, out=state["y"])
        return {"y": y, "sel": sel, "wts": wts}
    if case["entry"] == "device":
        eng.forward_dev(x, state["bufs"][0], flavour=flavour)
        return state["bufs"][0]
    cur = x
    for L in range(case["layers"]):
        out = state["bufs"][L & 1]
        eng.forward_dev(cur, out, layer_first=L, n_layers=1, flavour=flavour)
        cur = out
    return cur


# ---------------------------------------------------------------- what a pass cannot do without, and how exact it is
def work(case):
    if case["kind"] == "gemm":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": (m + n) * k * case["bits"] // 8 + 4 * (m + n) + 2 * m * n, "flops": 2 * m * k * n}
    if case["kind"] == "hook":
        w = 3 * case["e"] * case["ff"] * case["used"]
        return {"bytes": case["layers"] * (w * 9 // 16 + 8 * case["e"]), "flops": case["layers"] * 2 * w}
    cfg, M, n = GEMMA4_26B_A4B, case["tokens"], case["layers"]
    NE, NU = cfg["NE"], cfg["NU"]
    # distinct experts of a layer: what M tokens of an even router reach; the Zipf bias leaves about NU of them
    U = NU if case["zipf"] else NE * (1.0 - (1.0 - NU / NE) ** M)
    per_layer = synth.algorithmic_bytes_per_layer(cfg, 0, U)
    out = 8 * M * NU * n if case["entry"] == "host" else 0
    return {"bytes": int(n * per_layer + 2 * M * cfg["E"] * 4 + out), "flops": n * M * synth.flops_per_token_layer(cfg)}


def tolerance(case):
    if case["kind"] == "gemm":
        return "exact"                    # integer sums, then a fixed sequence of roundings
    if case["kind"] == "hook" or case["flavour"] == "decode":
        # int8 activations: a sum in another order moves a code here and there; the expert ids do not change
        return {"rel": 1e-3, "max": 0.04}
    # fp32-grade GEMMs. Another order of summation moves a router logit by about 1e-7 of its spread, and where a token's
    # 8th and 9th expert lie closer than that it takes the other one: about two of the 4096 * 30 choices, each a
    # visible change of that one token's row
    return {"rel": 1e-2, "max": 0.9, "differ": 1e-3}
