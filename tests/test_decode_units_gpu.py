"""Units of four and of sixteen tokens of the batched row kernel: chosen by each group's own count beside the average, with down rows
long enough for the two-tile form, whose stages and sums pass from one batch of a unit to the next."""
import numpy as np
import pytest

import orc
from gpu_common import assert_close, make_stack, oracle_stack

pytestmark = pytest.mark.gpu
A = 0


def _cfg(E, NE, NU, FFE, FFS):
    return dict(E=E, NE=NE, NU=NU, FFE=FFE, FFS=FFS, eps=1e-6)


LONG = _cfg(96, 4, 2, 1056, 2112)       # above 24 items per expert from 49 tokens on: units of sixteen for all
SKEW = _cfg(96, 32, 2, 1056, 2112)      # below it up to 384 tokens


@pytest.mark.parametrize("cfg,M,skew", [(LONG, 48, False), (LONG, 49, False), (LONG, 50, False), (LONG, 65, False), (SKEW, 48, True), (SKEW, 49, True), (SKEW, 50, True),
                                        (SKEW, 65, True), (SKEW, 131, True), (orc.SMALL, 49, True), (_cfg(1088, 16, 2, 96, 64), 67, True)])
def test_units_by_the_groups_own_count(cfg, M, skew):
    """skew: one expert takes every token (up to 48 in units of four, above that of sixteen) and the others share the rest: both
    sizes in one launch. A token's bits do not depend on its batch, and no pass differs from the first."""
    import torch
    bias = None
    if skew:
        bias = torch.zeros(cfg["NE"], device="cuda")
        bias[1] = 30.0
    eng, host = make_stack(cfg, 1, seed=81, rand_norms=True, max_tokens=M, bias=bias)
    x = np.random.default_rng(M).standard_normal((M, cfg["E"])).astype(np.float32)
    y, sel, wts = eng.forward(x, flavour=A)
    ry, rsel, _, margin = oracle_stack(cfg, host, x, A)
    assert np.array_equal(sel, rsel), f"expert ids differ (min margin {margin:.3e})"
    assert not skew or (sel[0] == 1).any(axis=-1).all()
    assert_close(y, ry, "decode batch")
    for _ in range(10):
        assert np.array_equal(eng.forward(x, flavour=A)[0].view(np.uint32), y.view(np.uint32))
    for t in {0, 1, M // 2, M - 2, M - 1}:
        assert np.array_equal(eng.forward(x[t:t + 1], flavour=A)[0][0].view(np.uint32), y[t].view(np.uint32))
    eng.close()


@pytest.mark.parametrize("M,owned", [(23, 2), (24, 2), (25, 2), (49, 2), (70, 4)])
def test_expert_parallel_units(M, owned):
    """The rows of one rank's experts: `owned` of 32 experts have them, more than 24 each or not; the shared expert of more than 24
    tokens. The stages give the bits of the same rows alone, and of the layer."""
    import torch
    from kairos_engine_b200 import ep
    cfg = SKEW
    eng, _ = make_stack(cfg, 1, seed=82, rand_norms=True, max_tokens=M, max_expert_rows=2 * M + 8)
    g = torch.Generator(device="cuda").manual_seed(M)
    R = 2 * M
    rows = torch.randn(R, cfg["E"], device="cuda", generator=g)
    ids = (8 + torch.arange(R, device="cuda") * owned // R).to(torch.int32)
    out = eng.ep_experts(0, rows, ep.expert_offsets(ids, cfg["NE"]), A)
    for r in (0, 1, R // owned - 1, R // owned, R - 1):
        one = eng.ep_experts(0, rows[r:r + 1].contiguous(), ep.expert_offsets(ids[r:r + 1], cfg["NE"]), A)
        assert torch.equal(out[r].view(torch.int32), one[0].view(torch.int32))
    x = torch.randn(M, cfg["E"], device="cuda", generator=g)
    y = torch.empty_like(x)
    eng.forward_dev(x, y, 0, 1, A)
    sel_asc, cw, send, counts, pair_index = eng.ep_route(0, x, A, defer_shared=True)
    eng.ep_shared(0, M, A)
    off = torch.zeros(cfg["NE"] + 1, dtype=torch.int32, device="cuda")
    off[1:] = torch.cumsum(counts, 0).to(torch.int32)
    y2 = eng.ep_finish(0, x, eng.ep_experts(0, send, off, A), pair_index=pair_index)
    eng.status()
    assert torch.equal(y.view(torch.int32), y2.view(torch.int32))
    eng.close()


@pytest.mark.parametrize("cfg,M", [(_cfg(64, 160, 8, 2048, 64), 120), (_cfg(2080, 160, 8, 1056, 64), 200)])
def test_more_units_than_the_table_holds(cfg, M):
    """Some 200 units a CTA of gate|up, and of down: those beyond the first 128 are found later, 32 at a time."""
    import torch
    from kairos_engine_b200 import MoeEngine, synth
    eng = MoeEngine(n_layers=1, max_tokens=M, **cfg)
    eng.upload_layer(0, synth.make_layer(cfg, 83, rand_norms=True), on_device=True)
    x = synth.make_inputs(cfg, M, 84)
    y, y1 = torch.empty_like(x), torch.empty_like(x[:1])
    eng.forward_dev(x, y, flavour=A)
    for t in range(0, M, 7):
        eng.forward_dev(x[t:t + 1].contiguous(), y1, flavour=A)
        assert torch.equal(y1[0].view(torch.int32), y[t].view(torch.int32)), t
    again = torch.empty_like(x)
    for _ in range(10):
        eng.forward_dev(x, again, flavour=A)
        assert torch.equal(again.view(torch.int32), y.view(torch.int32))
    eng.status(); eng.close()
