"""The sizes at which the batched kernels change their tile, variant or path, against the CPU checker: edges of tiles,
remainders, the smallest and the largest of each range."""
import numpy as np
import pytest

import orc
from gpu_common import MAX_ABS, REL_L2, assert_close, assert_same_experts, make_stack, oracle_stack

pytestmark = pytest.mark.gpu
A, B = 0, 1


def _cfg(E, NE, NU, FFE, FFS):
    return dict(E=E, NE=NE, NU=NU, FFE=FFE, FFS=FFS, eps=1e-6)


SMALL, GEMMA = orc.SMALL, orc.GEMMA
ODD = _cfg(96, 8, 2, 32, 96)            # rows of three chunks and of one: no whole groups of two
LONG = _cfg(1088, 16, 4, 1056, 64)      # rows just over 32 chunks, even and odd; down rows as two 16-row tiles
WIDEST = _cfg(4096, 4, 2, 64, 4096)     # the longest rows: fewest stages, the wide token kernel
MANY = _cfg(128, 160, 8, 32, 64)        # more than 128 experts: the block-wide selection


@pytest.mark.parametrize("cfg,M", [(ODD, 2), (ODD, 17), (ODD, 150), (SMALL, 4), (SMALL, 5), (SMALL, 64), (SMALL, 65), (GEMMA, 16), (GEMMA, 17),
                                   (LONG, 3), (LONG, 16), (WIDEST, 2), (WIDEST, 3), (MANY, 9), (MANY, 20), (MANY, 21)])
def test_decode_batch_edges(cfg, M, monkeypatch):
    """Tokens per expert around the two- and four-token forms of the row kernel and its 16-token units; the first pass of a
    fresh handle, whose weights are in no cache, and later ones."""
    monkeypatch.setenv("SP_MOE_SEQ_TOKENS", "1")
    eng, host = make_stack(cfg, 1, seed=71, rand_norms=True, max_tokens=M)
    x = np.random.default_rng(M).standard_normal((M, cfg["E"])).astype(np.float32)
    y, sel, wts = eng.forward(x, flavour=A)
    ry, rsel, rwts, margin = oracle_stack(cfg, host, x, A)
    assert np.array_equal(sel, rsel), f"expert ids differ (min margin {margin:.3e})"
    assert_close(y, ry, "decode batch")
    for _ in range(20):
        assert np.array_equal(eng.forward(x, flavour=A)[0].view(np.uint32), y.view(np.uint32))
    for t in {0, 1, M - 1}:                 # the single-token kernels' bits
        y1, sel1, wts1 = eng.forward(x[t:t + 1], flavour=A)
        assert np.array_equal(sel1[:, 0], sel[:, t])
        assert np.array_equal(y1[0].view(np.uint32), y[t].view(np.uint32)) and np.array_equal(wts1[:, 0].view(np.uint32), wts[:, t].view(np.uint32))
    eng.close()


@pytest.mark.parametrize("n", [1, 4, 5])
def test_single_token_runs_direct_and_replayed(n):
    """Runs of up to four layers are launched directly, longer ones replayed from a graph: the same bits, also when repeated."""
    cfg = orc.TINY
    eng, host = make_stack(cfg, 6, seed=72, rand_norms=True)
    x = np.random.default_rng(n).standard_normal((1, cfg["E"])).astype(np.float32)
    ry, rsel, _, _ = oracle_stack(cfg, host, x, A, first=1, n=n)
    for _ in range(3):
        y, sel, _ = eng.forward(x, flavour=A, layer_first=1, n_layers=n)
        assert np.array_equal(sel, rsel)
        assert np.array_equal(y.view(np.uint32), ry.view(np.uint32))
    eng.close()


PRE = _cfg(512, 8, 2, 160, 96)          # FFE and FFS off multiples of 64: the CUDA-core kernels
TC = _cfg(512, 8, 2, 192, 320)          # the tensor-core kernels with a last weight tile of one block, in both GEMMs
TC_MIN = _cfg(64, 4, 2, 64, 64)         # one k-step of 64, less than one block of down rows
TC_MANY = _cfg(576, 160, 8, 64, 192)    # more experts than the warp-wide selection takes, K off multiples of 256


@pytest.mark.parametrize("cfg,M", [(PRE, 2), (PRE, 32), (PRE, 33), (PRE, 64), (PRE, 129), (PRE, 257), (_cfg(544, 160, 8, 96, 608), 50), (_cfg(4096, 4, 2, 64, 128), 40),
                                   (TC, 2), (TC, 15), (TC, 32), (TC, 33), (TC, 64), (TC, 65), (TC, 129), (TC, 257), (TC_MIN, 2), (TC_MIN, 17), (TC_MIN, 33), (TC_MIN, 130),
                                   (TC_MANY, 3), (TC_MANY, 50), (TC_MANY, 170), (TC_MANY, 400)])
def test_prefill_tile_edges(cfg, M):
    """Rows per expert on both sides of the sixteen at which the GEMMs go from 32 to 64 rows a tile, and of tiles of 16, 32 and
    64 rows."""
    eng, host = make_stack(cfg, 1, seed=73, rand_norms=True, max_tokens=M)
    x = np.random.default_rng(M).standard_normal((M, cfg["E"])).astype(np.float32)
    y, sel, wts = eng.forward(x, flavour=B)
    ry, rsel, rwts, margin = oracle_stack(cfg, host, x, B)
    assert_same_experts(sel, rsel, wts, rwts, margin)
    assert_close(y, ry, "prefill")
    eng.close()


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("M,N,K", [(2305, 2305, 272), (1025, 2049, 272), (1025, 1030, 288), (17, 72, 32)])
def test_int_gemm_each_tile(M, N, K, packed):
    """One size for each of the four output tiles, with ragged rows, columns and depth."""
    import torch
    from kairos_engine_b200.engine import int_gemm_scaled
    r = np.random.default_rng(M + K)
    lo, hi = (-8, 8) if packed else (-128, 128)
    a, b = r.integers(lo, hi, (M, K), dtype=np.int8), r.integers(lo, hi, (N, K), dtype=np.int8)
    sa, sb = (r.random(M).astype(np.float32) + 0.5) * 1e-3, (r.random(N).astype(np.float32) + 0.5) * 1e-3
    ref = orc.int_gemm_scaled(a, b, sa, sb)
    if packed:
        a, b = (((q[:, 1::2].astype(np.uint8) << 4) | (q[:, 0::2].astype(np.uint8) & 15)) for q in (a, b))
    t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    got = int_gemm_scaled(t(a), t(b), t(sa), t(sb), packed_int4=packed)
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy().view(np.uint16), ref)


@pytest.mark.parametrize("E,FF,NE,NU", [(32, 32, 2, 1), (1056, 2080, 3, 3), (64, 96, 24, 20), (4096, 32, 2, 2)])
def test_hook_edges(E, FF, NE, NU):
    """The smallest shapes, rows just over 32 and 64 chunks, more experts than one round takes, the longest rows."""
    from kairos_engine_b200 import MoeExt
    from test_ext_hook_gpu import _q4b, _reference
    rng = np.random.default_rng(E + NU)
    w = [[_q4b(rng, rows, cols) for _ in range(NE)] for rows, cols in ((FF, E), (FF, E), (E, FF))]
    (g, gs), (u, us), (d, ds) = ([np.stack(c) for c in zip(*t)] for t in w)
    ext = MoeExt()
    ext.upload_experts("blk.0.ffn_gate_exps.weight", g, gs, u, us, d, ds, NE, FF, E)
    x = rng.standard_normal(E).astype(np.float32)
    idx = rng.choice(NE, NU, replace=False).astype(np.int32)
    wt = rng.random(NU).astype(np.float32)
    y = ext.moe("blk.0.ffn_gate_exps.weight", idx, wt / wt.sum(), x, FF)
    ref = _reference(x, idx, wt / wt.sum(), g, gs, u, us, d, ds, E, FF)
    diff = y.astype(np.float64) - ref
    assert np.abs(diff).max() <= MAX_ABS and np.linalg.norm(diff) / np.linalg.norm(ref) <= REL_L2
    ext.close()


def _at(t, off):
    """The values of t in a buffer that starts `off` floats past a 16-byte boundary."""
    import torch
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    out = buf[off:off + t.numel()].view(t.shape)
    assert out.data_ptr() % 16 == 4 * off
    return out.copy_(t)


@pytest.mark.parametrize("flavour", [A, B])
@pytest.mark.parametrize("cfg,M", [(SMALL, 66), (SMALL, 200), (_cfg(3200, 8, 2, 64, 64), 65)])
def test_vectors_on_any_float_boundary(cfg, M, flavour):
    """x, y and pair rows where only floats are aligned: the bits of the aligned call, through the layer and through its
    expert-parallel stages."""
    import torch
    eng, _ = make_stack(cfg, 2, seed=74, rand_norms=True, max_tokens=M)
    x = torch.randn(M, cfg["E"], generator=torch.Generator().manual_seed(M)).cuda()
    for n in (1, 2):
        want = torch.empty_like(x)
        eng.forward_dev(x, want, n_layers=n, flavour=flavour)
        for xo, yo in ((1, 0), (0, 2), (3, 3)):
            xm, y = _at(x, xo), _at(torch.zeros_like(x), yo)
            eng.forward_dev(xm, y, n_layers=n, flavour=flavour)
            assert torch.equal(y, want) and torch.equal(xm, x)
            eng.forward_dev(xm, xm, n_layers=n, flavour=flavour)          # in place
            assert torch.equal(xm, want)
    eng.forward_dev(x, want, n_layers=1, flavour=flavour)
    _, _, rows, counts, pair_index = eng.ep_route(0, _at(x, 1), flavour)
    off = torch.cat([torch.zeros(1, dtype=torch.int32, device="cuda"), counts.cumsum(0).int()])
    out = eng.ep_experts(0, _at(rows, 1) if flavour == A else rows, off, flavour)
    assert torch.equal(eng.ep_finish(0, _at(x, 2), _at(out, 3), pair_index=pair_index), want)
    eng.status(); eng.close()
