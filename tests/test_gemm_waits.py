"""The GEMM's waits that a whole warp makes: every lane of a warp must take the
same branch behind one, since warp-wide (.aligned) instructions follow.  Read
from the source: the other outcome shows only when a wait runs out."""

import re

from gpusim2grid_b200._build import CSRC


def _epilogue_role():
    src = re.sub(r"//[^\n]*", "", (CSRC / "mlp_gemm.cuh").read_text())
    body = src[src.index("gemm_bf16_kernel("):]
    start = body.index("} else if (warp >= 2) {")
    return body[start:body.index("tcgen05.ld.sync.aligned", start)]


def test_epilogue_warps_give_up_together():
    role = _epilogue_role()
    waits = [m.start() for m in re.finditer(r"\bmbar_wait\(", role)]
    assert waits, "the epilogue waits for its accumulator"
    for at in waits:
        assert re.search(r"__all_sync\(0xffffffffu,\s*$", role[:at]), "a lane decides on its own wait alone"
    # nor does a lane look at the flag by itself
    assert "*fail" not in role
