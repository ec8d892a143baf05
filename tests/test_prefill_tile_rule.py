"""Rows per activation tile of the prefill GEMMs: by the rows of an expert, and by how many tiles there are for the SMs."""
import re

import numpy as np
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.load(tmp_path_factory.mktemp("fake"))


def _aligned(n):
    raw = np.zeros(n + 64, np.float32)
    return raw[(-raw.ctypes.data) % 64 // 4:]


def _heights(fake):
    return [int(re.search(r"k_tc_gemmILb[01]ELi\dELi(\d+)E", k.name).group(1)) for k in fake.launches("k_tc_gemm")]


# FFE 640: five weight tiles of gate|up an expert, 160 with 32 experts; FFE 64: one, 32 in all
@pytest.mark.parametrize("ffe,rows_per_expert,tile", [(640, 8, 32), (640, 12, 32), (640, 13, 64), (640, 16, 64), (64, 13, 32), (64, 16, 32), (64, 17, 64)])
def test_tile_heights(fake, ffe, rows_per_expert, tile):
    """Above twelve rows an expert on average a skewed router has experts of many tiles (a line of 16 took 24% from a Zipf one at 256
    tokens); where tiles of 64 would not reach every SM the line is at 16."""
    cfg = dict(E=64, NE=32, NU=2, FFE=ffe, FFS=64, eps=1e-6)
    M = rows_per_expert * cfg["NE"] // cfg["NU"]
    h = fake.engine(cfg, max_tokens=M)
    x = _aligned(M * cfg["E"])
    assert fake.L.sp_moe_forward_dev(h, 0, 1, 1, M, x.ctypes.data, x.ctypes.data, None, None, None) == 0
    assert _heights(fake) == [tile, tile]
    fake.L.sp_moe_close(h)


@pytest.mark.parametrize("rows_per_expert,tile", [(8, 32), (9, 64), (16, 64), (17, 64)])
def test_experts_stage(fake, rows_per_expert, tile):
    """The stage call is not told how many of the experts are its rank's: averaged over all, nine rows an expert are already 18 to 72
    where there are rows, and belong on tiles of 64."""
    cfg = dict(E=64, NE=32, NU=2, FFE=640, FFS=64, eps=1e-6)
    R = rows_per_expert * cfg["NE"]
    h = fake.engine(cfg, max_tokens=4, max_expert_rows=R)
    rows, offsets = _aligned(R * cfg["E"]), np.zeros(cfg["NE"] + 1, np.int32)
    assert fake.L.sp_moe_ep_experts_dev(h, 0, 1, R, rows.ctypes.data, None, offsets.ctypes.data, rows.ctypes.data, None) == 0
    assert _heights(fake) == [tile, tile]
    fake.L.sp_moe_close(h)
