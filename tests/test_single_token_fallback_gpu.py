"""Phase stamps of a single-token step whose selection falls back on the probabilities."""
import numpy as np
import pytest

import orc
from gpu_common import make_stack

pytestmark = pytest.mark.gpu


def test_stamps_of_a_fallback_are_its_own(monkeypatch):
    """Layer 0 selects from its logits, layer 1 (equal logits) from the probabilities: every stamp the second kernel reports lies
    between its entry and its end."""
    import torch
    from kairos_engine_b200 import MoeEngine, synth
    cfg = orc.SMALL
    monkeypatch.setenv("SP_MOE_TIMING", "1")
    eng = MoeEngine(n_layers=2, **cfg)
    monkeypatch.delenv("SP_MOE_TIMING")
    for L in range(2):
        layer = synth.make_layer(cfg, 40 + L, bias=torch.zeros(cfg["NE"], device="cuda") if L else None)
        if L:
            layer["router_w"] = torch.zeros_like(layer["router_w"])
        eng.upload_layer(L, layer, on_device=True)
    x = np.random.default_rng(3).standard_normal((1, cfg["E"])).astype(np.float32)
    for L in (0, 1, 0, 1, 1):
        eng.forward(x, layer_first=L, n_layers=1)
        raw = eng.decode_timing()["raw_us"][1]
        taken = [raw[i] for i in (0, 1, 5, 6, 7, 2, 3, 12, 4)]
        assert all(v > 0.0 for v in taken) and taken == sorted(taken), (L, raw)
    eng.close()
