"""Rules of the kernels' waits that a run does not show, read from the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kairos_engine_b200", "csrc")


def _source(name):
    return re.sub(r"/\*.*?\*/|//[^\n]*", "", open(os.path.join(CSRC, name)).read(), flags=re.S)


def test_roles_wait_for_one_another_on_bounded_barriers_only():
    """A kernel whose warps have roles may lose one of them when a bounded wait runs out: the others must not wait for it on a
    barrier that cannot give up (bar.sync, a block-wide one while roles run, a poll without a limit)."""
    for name in ("rows_mma.cu", "prefill_tc.cu", "int_gemm_tc.cu"):
        src = _source(name)
        assert not re.search(r"\"[^\"]*\bbar(rier)?\.(cta\.)?(sync|arrive|red)", src), f"{name}: a named barrier"
        assert not re.search(r"\bmbar_try(_suspend)?\s*\(", src), f"{name}: a poll of its own"
    roles = _source("rows_mma.cu")
    roles = roles[roles.index("bool failed = false;"):]
    roles = roles[:roles.index("\n}\n")]
    assert "mbar_wait(" in roles and "__syncthreads" not in roles and "__syncwarp" in roles
