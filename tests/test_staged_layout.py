"""Geometries whose weight rows fill the shared memory of the single-token kernels: they keep the staged path, where the sums of
the routed pairs take the place of rows that are done."""
import numpy as np
import pytest

import fake_cuda
import orc

FULL = [(768, 8, 8, 3968, 4096), (1280, 8, 8, 2432, 4096), (2560, 16, 5, 2240, 512), (2560, 16, 6, 1600, 2816), (4096, 8, 5, 1184, 2112)]


def _cfg(E, NE, NU, FFE, FFS):
    return dict(E=E, NE=NE, NU=NU, FFE=FFE, FFS=FFS, eps=1e-6)


@pytest.mark.parametrize("geo", FULL)
def test_full_geometries_keep_the_staged_path(tmp_path_factory, geo):
    fake = fake_cuda.load(tmp_path_factory.mktemp("fake"))
    cfg = _cfg(*geo)
    h = fake.engine(cfg)
    x = np.zeros(cfg["E"] + 16, np.float32)
    x = x[(-x.ctypes.data) % 64 // 4:]
    assert fake.L.sp_moe_forward_dev(h, 0, 1, 0, 1, x.ctypes.data, x.ctypes.data, None, None, None) == 0
    assert len(fake.launches("k_ds_experts_up")) == 1
    fake.L.sp_moe_close(h)


@pytest.mark.gpu
@pytest.mark.parametrize("geo", FULL)
def test_full_geometries_give_the_oracles_bits(geo):
    from gpu_common import make_stack, oracle_stack
    cfg = _cfg(*geo)
    eng, host = make_stack(cfg, 2, seed=91, rand_norms=True, max_tokens=2)
    x = np.random.default_rng(9).standard_normal((2, cfg["E"])).astype(np.float32)
    batch = eng.forward(x, flavour=0)[0]
    for t in range(2):
        y, sel, wts = eng.forward(x[t:t + 1], flavour=0)
        assert np.array_equal(y[0].view(np.uint32), batch[t].view(np.uint32))
        if t == 0:
            ry, rsel, rwts, _ = oracle_stack(cfg, host, x[:1], 0)
            assert np.array_equal(sel, rsel) and np.array_equal(wts.view(np.uint32), rwts.view(np.uint32))
            assert np.array_equal(y.view(np.uint32), ry.view(np.uint32))
    eng.close()
