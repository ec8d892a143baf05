"""Host side of the entry points without a GPU: which kernels a call launches with which pointers, and what it does when a
launch fails (the library's own objects over the runtime of fake_cudart.c)."""
import ctypes as C
import glob
import os
import re

import numpy as np
import pytest

import fake_cuda
import orc


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.load(tmp_path_factory.mktemp("fake"))


@pytest.fixture(autouse=True)
def _reset(fake):
    yield
    fake.log.clear(); fake.read = {}; fake.on_launch = None
    fake.L.fake_set_sms(148)


def _floats(n, off):
    """n floats that start `off` bytes past a 64-byte boundary."""
    raw = np.zeros(4 * n + 128, np.uint8)
    at = (-raw.ctypes.data) % 64 + off
    return raw[at:at + 4 * n].view(np.float32)


def _vectorised(name):
    """Does this instance of k_b_token / k_b_quant_rows use 16-byte accesses of the rows it is given?"""
    m = re.search(r"k_b_tokenILb[01]ELi\dELb[01]ELb[01]E(?:Lb([01])E)?|k_b_quant_rows(?:ILb([01])E)?", name)
    return "0" not in (m.group(1), m.group(2))


def _token_kernels_are_safe(fake):
    seen = fake.launches("k_b_token")
    for k in seen:
        fin = "k_b_tokenILb1" in k.name
        x, eo, y = k.words[0], k.words[2], k.words[8]
        misaligned = any(p & 15 for p in ((x, eo, y) if fin else (x,)))
        assert not (misaligned and _vectorised(k.name)), f"{k.name} is given {x:#x} {eo:#x} {y:#x}"
    return len(seen)


@pytest.mark.parametrize("flavour", [0, 1])
@pytest.mark.parametrize("n_layers", [1, 3])
@pytest.mark.parametrize("xo,yo", [(0, 0), (4, 0), (0, 8), (12, 4)])
def test_forward_takes_any_float_boundary(fake, flavour, n_layers, xo, yo):
    """Beyond 64 tokens the kernels run on the caller's x and y: no kernel with 16-byte accesses may meet another boundary."""
    cfg, M = orc.SMALL, 70
    h = fake.engine(cfg, n_layers=n_layers, max_tokens=M)
    fake.read = {"k_b_token": (1, 9)}
    x, y = _floats(M * cfg["E"], xo), _floats(M * cfg["E"], yo)
    assert fake.L.sp_moe_forward_dev(h, 0, n_layers, flavour, M, x.ctypes.data, y.ctypes.data, None, None, None) == 0
    assert _token_kernels_are_safe(fake) >= n_layers + 1
    fake.L.sp_moe_close(h)


@pytest.mark.parametrize("flavour", [0, 1])
@pytest.mark.parametrize("off", [0, 4, 8])
def test_expert_parallel_stages_take_any_float_boundary(fake, flavour, off):
    cfg, M = orc.SMALL, 6
    E, NE, NU = cfg["E"], cfg["NE"], cfg["NU"]
    h = fake.engine(cfg, max_tokens=M)
    fake.read = {"k_b_token": (1, 9), "k_b_quant_rows": (0, 1)}
    x, y, pairs = _floats(M * E, off), _floats(M * E, off), _floats(M * NU * E, off)
    rows, out, ints = _floats(M * NU * E, 0), _floats(M * NU * E, 0), np.zeros(M * NU + NE + 1, np.int32)
    p = lambda a: a.ctypes.data
    route = lambda r: fake.L.sp_moe_ep_route_dev(h, 0, flavour, M, p(x), p(ints), p(_floats(M * NU, 0)), p(r), p(ints), p(ints), None, None, 0, 0, 0, None)
    assert route(rows) == 0
    assert fake.L.sp_moe_ep_finish_dev(h, 0, M, p(x), p(pairs), None, p(y), None) == 0
    assert _token_kernels_are_safe(fake) == 2
    experts = lambda r: fake.L.sp_moe_ep_experts_dev(h, 0, flavour, M * NU, p(r), None, p(ints), p(out), None)
    if flavour == 0 or off == 0:
        assert experts(pairs) == 0
        for k in fake.launches("k_b_quant_rows"):
            assert not (k.words[0] & 15 and _vectorised(k.name))
    else:                                                    # what only ever ran on 16-byte boundaries is refused, not launched
        before = len(fake.launches())
        assert experts(pairs) == -3 and route(pairs) == -3 and len(fake.launches()) == before
    fake.L.sp_moe_close(h)


def _hook(fake, E=64, FF=32, NE=4):
    h = C.c_void_p()
    assert fake.L.sp_moe_ext_open(0, C.byref(h)) == 0
    blob = np.zeros(NE * FF * E, np.uint8).ctypes.data
    assert fake.L.sp_moe_ext_upload_experts(h, b"t", blob, blob, blob, blob, blob, blob, NE, FF, E) == 0
    idx, wt, x, y = np.zeros(20, np.int32), np.zeros(20, np.float32), np.zeros(E, np.float32), np.zeros(E, np.float32)
    return h, lambda n: fake.L.sp_moe_ext_moe(h, b"t", idx.ctypes.data, wt.ctypes.data, n, x.ctypes.data, E, FF, y.ctypes.data)


@pytest.mark.parametrize("n,failing", [(2, 0), (2, 1), (2, 2), (20, 3)])
def test_hook_leaves_nothing_running_when_a_launch_fails(fake, n, failing):
    """The call reads its x from a buffer of the handle that the next call overwrites: also a call that fails waits for
    what it had launched."""
    h, call = _hook(fake)
    count = [0]

    def fail_one(_):
        count[0] += 1
        return 700 if count[0] == failing + 1 else 0
    fake.log.clear(); fake.on_launch = fail_one
    assert call(n) != 0
    assert isinstance(fake.log[-1], tuple) and fake.log[-1][0] == "sync"
    fake.on_launch = None; fake.log.clear()
    assert call(n) == 0 and fake.log[-1][0] == "sync"
    fake.L.sp_moe_ext_close(h)


def test_kernels_launched_programmatically_wait():
    """launch.cuh's rule, over the sources: a kernel launched with sp_launch waits for its predecessor before it lets its
    successor start; any other that lets its successor start waits too."""
    checked = 0
    for path in glob.glob(os.path.join(os.path.dirname(fake_cuda.HERE), "kairos_engine_b200", "csrc", "*.cu")):
        src = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
        if '"launch.cuh"' not in src:
            continue
        named = set(re.findall(r"k_\w+", " ".join(re.findall(r"sp_launch\(.*?;", src, flags=re.S))))
        for part in re.split(r"__global__", src)[1:]:
            name, body = re.search(r"\b(k_\w+)\s*\(", part).group(1), part[part.index("{"):]
            body = body[:body.index("\n}\n")]
            if name in named or "sp_pdl_next()" in body:
                wait, nxt = body.find("sp_pdl_wait()"), body.find("sp_pdl_next()")
                assert wait >= 0 and (nxt < 0 or wait < nxt or name not in named), f"{name} ({os.path.basename(path)})"
                checked += 1
    assert checked >= 12


def _gemm(fake, entry, A=None, B=None, out=None, M=32, K=32, N=32):
    a = np.zeros(4 * M * max(K, N) + 256, np.uint8)
    base = a.ctypes.data + (-a.ctypes.data) % 64
    p = lambda given: base if given is None else given
    return getattr(fake.L, entry)(p(A), p(B), base, base, p(out), M, K, N, None)


def _fail_wait(launch):
    C.cast(launch.words[7], C.POINTER(C.c_int))[0] = 2      # what the kernel does when a bounded wait runs out


def test_int4_calls_in_flight_together_have_their_own_verdict(fake):
    fake.read = {"k_i8_gemm": (1, 8)}
    inner = []

    def first(launch):
        _fail_wait(launch)
        fake.on_launch = None
        inner.append(_gemm(fake, "sp_frob_matmul_q4_dev"))  # another thread's call, while this one has not returned
    fake.on_launch = first
    assert _gemm(fake, "sp_frob_matmul_q4_dev") == -40 and inner == [0]
    assert _gemm(fake, "sp_frob_matmul_q4_dev") == 0
    for _ in range(200):                                    # the words are given back, by failed calls too
        fake.on_launch = _fail_wait
        assert _gemm(fake, "sp_frob_matmul_q4_dev") == -40
        fake.on_launch = lambda launch: 700
        assert _gemm(fake, "sp_frob_matmul_q4_dev") == -40


def test_int8_verdict_reaches_the_next_int8_call_only(fake):
    fake.read = {"k_i8_gemm": (1, 8)}
    fake.on_launch = _fail_wait
    assert _gemm(fake, "sp_frob_matmul_q8_dev") == 0        # returns before its kernel runs
    fake.on_launch = None
    assert _gemm(fake, "sp_frob_matmul_q4_dev") == 0
    before = len(fake.launches())
    assert _gemm(fake, "sp_frob_matmul_q8_dev") == -40 and b"earlier" in fake.L.sp_last_error() and len(fake.launches()) == before
    assert _gemm(fake, "sp_frob_matmul_q8_dev") == 0 and len(fake.launches()) == before + 1


@pytest.mark.parametrize("off", [(1, 0), (0, 8), (7, 3)])
def test_packed_operands_start_on_any_byte(fake, off):
    """They are moved to where the kernel's copies can read them; int8 operands on another boundary stay refused."""
    fake.read = {"k_i8_gemm": (1, 8)}
    raw = np.arange(4096, dtype=np.uint8)
    base = raw.ctypes.data + (-raw.ctypes.data) % 64
    assert _gemm(fake, "sp_frob_matmul_q4_dev", A=base + off[0], B=base + 1024 + off[1]) == 0
    a, b = fake.launches()[-1].words[:2]
    assert a % 16 == 0 and b % 16 == 0
    copies = [(src, n) for what, dst, src, n in (x for x in fake.log if isinstance(x, tuple)) if what == "memcpy"]
    assert copies == [(base + off[0], 32 * 16), (base + 1024 + off[1], 32 * 16)]
    assert _gemm(fake, "sp_frob_matmul_q8_dev", A=base + off[0], B=base + 1024 + off[1]) == -3


@pytest.mark.parametrize("E,M", [(64, 2), (128, 70), (448, 33), (512, 70), (4096, 2)])
def test_prefill_takes_the_fused_preparation_at_every_width(fake, E, M):
    """Seven launches a layer and one more, whatever the width: no geometry has a path that only its tests take."""
    cfg = dict(E=E, NE=8, NU=2, FFE=64, FFS=128, eps=1e-6)
    h = fake.engine(cfg, n_layers=2, max_tokens=M)
    x = _floats(M * E, 0)
    assert fake.L.sp_moe_forward_dev(h, 0, 2, 1, M, x.ctypes.data, x.ctypes.data, None, None, None) == 0
    assert len(fake.launches()) == 15 and len(fake.launches("k_tc_sort")) == 2 and len(fake.launches("k_tc_permute")) == 2
    fake.L.sp_moe_close(h)


@pytest.mark.parametrize("sms,M", [(148, 148), (148, 149), (100, 100), (100, 101), (160, 160)])
def test_one_block_per_sm_form_follows_the_device(fake, sms, M):
    """The token kernel's form for at most one block per SM: the device says how many SMs there are."""
    cfg = orc.SMALL
    fake.L.fake_set_sms(sms)
    h = fake.engine(cfg, max_tokens=M)
    x = _floats(M * cfg["E"], 0)
    assert fake.L.sp_moe_forward_dev(h, 0, 1, 0, M, x.ctypes.data, x.ctypes.data, None, None, None) == 0
    few = [re.search(r"k_b_tokenILb[01]ELi\dELb[01]ELb([01])E", k.name).group(1) for k in fake.launches("k_b_token")]
    assert few == ["1" if M <= sms else "0"] * 2
    fake.L.sp_moe_close(h)


@pytest.mark.parametrize("M,n_layers", [(1, 1), (1, 5), (8, 1), (70, 2)])
@pytest.mark.parametrize("failing", [0, 2])
def test_failed_launch_is_reported_once(fake, M, n_layers, failing):
    """The call whose launch fails says so; the runtime's record of it does not reach a later call that is fine."""
    cfg = orc.SMALL
    h = fake.engine(cfg, n_layers=n_layers, max_tokens=M)
    x = _floats(M * cfg["E"], 0)
    forward = lambda: fake.L.sp_moe_forward_dev(h, 0, n_layers, 0, M, x.ctypes.data, x.ctypes.data, None, None, None)
    count = [0]

    def fail_one(_):
        count[0] += 1
        return 700 if count[0] == failing + 1 else 0
    fake.on_launch = fail_one
    assert forward() == -40
    fake.on_launch = None
    ints = np.zeros(4 * cfg["NE"] + M * cfg["NU"], np.int32).ctypes.data
    assert fake.L.sp_moe_ep_recv_layout_dev(h, ints, 1, 0, M * cfg["NU"], ints, ints, None) == 0
    assert forward() == 0
    fake.L.sp_moe_close(h)
