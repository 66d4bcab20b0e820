"""What the tcgen05 kernels do when a wait runs out, read from their sources (an accumulator that never comes cannot be staged on a
GPU without a kernel that loses a signal on purpose)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "llm_b200" / "csrc"


@pytest.mark.parametrize("name", ["gemm_tc.cu", "gated_recurrence.cu"])
def test_no_thread_leaves_its_warps_on_its_own_wait(name):
    """`mbar_wait` answers each thread by itself. Behind it these kernels have barriers of several warps (`bar.sync 1`) or loads of
    whole warps (tcgen05.ld): a thread that breaks, returns or skips on its own answer leaves the others there, with no
    bound. Waits that decide where control goes are `mbar_wait_warp`; the epilogues of the products go on either way."""
    source = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    own = [m.start() for m in re.finditer(r"\bmbar_wait\(", source)]
    for at in own:
        statement = source[max(source.rfind(c, 0, at) for c in ";{}") + 1:source.index(";", at)].strip()
        assert statement.startswith("mbar_wait("), f"{name}: the answer of `{statement}` is used"
    assert "mbar_wait_warp(" in source
