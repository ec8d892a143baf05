"""The branches that the kernels take by value or by size inside one path, against the CPU checker: logits that tie or nearly do
in the single-token selection, units of tokens in the batched row kernel, tiles drawn from a counter in the prefill GEMM."""
import numpy as np
import pytest

import orc
from gpu_common import assert_close, assert_same_experts, make_stack, oracle_stack

pytestmark = pytest.mark.gpu
A, B = 0, 1


def _cfg(E, NE, NU, FFE, FFS):
    return dict(E=E, NE=NE, NU=NU, FFE=FFE, FFS=FFS, eps=1e-6)


def _logits(kind, NE, NU, rng):
    if kind == "equal":                     # the lowest ids win
        return np.zeros(NE, np.float32)
    if kind == "repeated":                  # equal logits in several warps, positive, negative and zeros of both signs
        return rng.choice(np.float32([-1.5, -0.0, 0.0, 0.25, 0.25, 2.0]), NE)
    if kind == "one ulp":                   # different logits whose probabilities round to the same float
        return (np.float32(1.0) + rng.permutation(NE).astype(np.float32) * np.float32(2.0 ** -23)).astype(np.float32)
    if kind == "narrow":                    # neighbours on both sides of 1e-6
        gaps = np.tile([9e-7, 1.1e-6, 2e-6, 0.0], NE // 4 + 1)[:NE]
        return np.cumsum(gaps)[rng.permutation(NE)].astype(np.float32)
    if kind == "underflow":                 # probabilities that are subnormal or zero
        v = -np.linspace(0.0, 800.0, NE)
        return v[rng.permutation(NE)].astype(np.float32)
    assert kind == "edge of 80"
    v = np.full(NE, -200.0)
    v[:NU] = -np.linspace(0.0, 80.5, NU)
    return v[rng.permutation(NE)].astype(np.float32)


@pytest.mark.parametrize("kind", ["equal", "repeated", "one ulp", "narrow", "underflow", "edge of 80"])
@pytest.mark.parametrize("cfg", [orc.GEMMA, _cfg(256, 128, 1, 64, 128), _cfg(96, 37, 5, 96, 32), _cfg(64, 3, 3, 32, 64), _cfg(128, 160, 8, 32, 64)])
def test_single_token_selection(cfg, kind):
    """A router of zeros leaves the bias as the logits: up to 128 experts they decide unless they are too close, then (and with
    more experts) the probabilities do; expert counts off multiples of 32, rows of a few pairs and chunks."""
    import torch
    from kairos_engine_b200 import MoeEngine, synth
    bias = _logits(kind, cfg["NE"], cfg["NU"], np.random.default_rng(cfg["NE"] + cfg["NU"]))
    layer = synth.make_layer(cfg, 75, rand_norms=True, bias=torch.from_numpy(bias).cuda())
    layer["router_w"] = torch.zeros_like(layer["router_w"])
    eng = MoeEngine(n_layers=1, max_tokens=1, **cfg)
    eng.upload_layer(0, layer, on_device=True)
    x = np.random.default_rng(5).standard_normal((1, cfg["E"])).astype(np.float32)
    y, sel, wts = eng.forward(x, flavour=A)
    ry, rsel, rwts, _ = oracle_stack(cfg, [orc.LayerWeights(**synth.layer_to_host(layer))], x, A)
    assert np.array_equal(sel, rsel)
    assert np.array_equal(wts.view(np.uint32), rwts.view(np.uint32)) and np.array_equal(y.view(np.uint32), ry.view(np.uint32))
    eng.close()


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("cfg,M", [(orc.SMALL, 95), (orc.SMALL, 96), (orc.SMALL, 97), (_cfg(96, 8, 2, 32, 96), 7), (_cfg(1088, 8, 3, 96, 64), 64), (_cfg(1088, 8, 3, 96, 64), 65)])
def test_decode_units(cfg, M, bias):
    """24 items per expert on average, where units of four tokens become units of sixteen: both sides of the line, evenly filled
    experts and a few that take nearly all tokens, last units of one to three. A token's bits do not depend on its batch."""
    import torch
    b = torch.linspace(3, -3, cfg["NE"]).cuda() if bias else None
    eng, host = make_stack(cfg, 1, seed=76, rand_norms=True, max_tokens=M, bias=b)
    x = np.random.default_rng(M).standard_normal((M, cfg["E"])).astype(np.float32)
    y, sel, wts = eng.forward(x, flavour=A)
    ry, rsel, _, margin = oracle_stack(cfg, host, x, A)
    assert np.array_equal(sel, rsel), f"expert ids differ (min margin {margin:.3e})"
    assert_close(y, ry, "decode batch")
    for t in (0, M // 2, M - 1):
        assert np.array_equal(eng.forward(x[t:t + 1], flavour=A)[0][0].view(np.uint32), y[t].view(np.uint32))
    eng.close()


@pytest.mark.parametrize("cfg,M", [(_cfg(2112, 160, 8, 64, 1024), 400), (_cfg(2112, 160, 8, 64, 1024), 20), (_cfg(64, 4, 2, 704, 64), 700), (_cfg(2112, 8, 2, 64, 64), 130)])
def test_prefill_drawn_tiles(cfg, M):
    """More tiles than the ring announces, tiles of one 64-k step beside tiles of sixteen, last tiles of one block, fewer tiles
    than CTAs: the same bits at every pass, whichever CTA drew a tile."""
    eng, host = make_stack(cfg, 1, seed=77, rand_norms=True, max_tokens=M)
    x = np.random.default_rng(M).standard_normal((M, cfg["E"])).astype(np.float32)
    y, sel, wts = eng.forward(x, flavour=B)
    ry, rsel, rwts, margin = oracle_stack(cfg, host, x, B)
    assert_same_experts(sel, rsel, wts, rwts, margin)
    assert_close(y, ry, "prefill")
    for _ in range(8):
        assert np.array_equal(eng.forward(x, flavour=B)[0].view(np.uint32), y.view(np.uint32))
    eng.status(); eng.close()


def _tie_then_one_ulp(NE, NU, same_warp):
    """NU - 1 larger logits, two equal ones of which one is the last chosen, and one a float below with a lower id whose
    probability rounds to theirs: the oracle takes that one."""
    near, tied = (3, (9, 11)) if same_warp else (3, (NE - 5, NE - 2))
    rest = [i for i in range(NE) if i not in (near, *tied)]
    for k in range(1, 200):
        v = -1.0 - np.arange(NE, dtype=np.float32) / NE
        v[rest[-(NU - 1):] if NU > 1 else []] = np.float32(2.0) + np.arange(NU - 1, dtype=np.float32)
        v[list(tied)] = np.float32(0.001 * k)
        v[near] = np.nextafter(np.float32(0.001 * k), np.float32(0.0))
        _, idx, _ = orc.topk(v, NU)
        if idx[NU - 1] == near:
            return v
    raise AssertionError("no such logits")


@pytest.mark.parametrize("same_warp", [True, False])
@pytest.mark.parametrize("cfg", [orc.GEMMA, _cfg(256, 128, 1, 64, 128), _cfg(96, 37, 5, 96, 32)])
def test_single_token_tie_at_the_last_place(cfg, same_warp):
    """The last chosen logit equals the first one left out and a third is one float below: probabilities decide, in the
    single-token kernels as in a batch of two."""
    import torch
    from kairos_engine_b200 import MoeEngine, synth
    bias = _tie_then_one_ulp(cfg["NE"], cfg["NU"], same_warp)
    layer = synth.make_layer(cfg, 78, rand_norms=True, bias=torch.from_numpy(bias).cuda())
    layer["router_w"] = torch.zeros_like(layer["router_w"])
    eng = MoeEngine(n_layers=1, max_tokens=2, **cfg)
    eng.upload_layer(0, layer, on_device=True)
    x = np.random.default_rng(6).standard_normal((2, cfg["E"])).astype(np.float32)
    ry, rsel, rwts, _ = oracle_stack(cfg, [orc.LayerWeights(**synth.layer_to_host(layer))], x, A)
    y, sel, wts = eng.forward(x, flavour=A)
    assert np.array_equal(sel, rsel) and np.array_equal(wts.view(np.uint32), rwts.view(np.uint32))
    for t in range(2):
        y1, sel1, wts1 = eng.forward(x[t:t + 1], flavour=A)
        assert np.array_equal(sel1[:, 0], rsel[:, t])
        assert np.array_equal(wts1[:, 0].view(np.uint32), rwts[:, t].view(np.uint32)) and np.array_equal(y1[0].view(np.uint32), ry[t].view(np.uint32))
        assert np.array_equal(y1[0].view(np.uint32), y[t].view(np.uint32))
    eng.close()
