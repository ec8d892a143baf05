"""Rows per activation tile of the prefill GEMMs in the expert-parallel experts stage, whose rows belong to some of the experts."""
import re

import numpy as np
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.load(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("rows_per_expert,tile", [(8, 32), (9, 64), (16, 64), (17, 64)])
def test_experts_stage_does_not_count_experts_of_other_ranks(fake, rows_per_expert, tile):
    """The stage is not told how many of the experts are its rank's: averaged over all, sixteen rows an expert are already
    32 to 128 where there are rows, and belong on tiles of 64."""
    cfg = dict(E=64, NE=32, NU=2, FFE=64, FFS=64, eps=1e-6)
    R = rows_per_expert * cfg["NE"]
    h = fake.engine(cfg, max_tokens=4, max_expert_rows=R)
    raw = np.zeros(R * cfg["E"] + 64, np.float32)
    rows = raw.ctypes.data + (-raw.ctypes.data) % 64
    offsets = np.zeros(cfg["NE"] + 1, np.int32).ctypes.data
    fake.log.clear()
    assert fake.L.sp_moe_ep_experts_dev(h, 0, 1, R, rows, None, offsets, rows, None) == 0
    seen = [int(re.search(r"k_tc_gemmILb[01]ELi\dELi(\d+)E", k.name).group(1)) for k in fake.launches("k_tc_gemm")]
    assert seen == [tile, tile]
    fake.L.sp_moe_close(h)
