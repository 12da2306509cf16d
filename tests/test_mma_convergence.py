"""tcgen05.ld and the aligned barriers of csrc/scan_mma.cuh are instructions that
a warp's lanes execute together.  Read from the source (no run can show a lane
arriving alone): the loop that reads accumulators for single hits has one path to
its one __syncwarp, and the team barriers gather the warp first."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "cas-offinder-rust-old_b200", "csrc", "scan_mma.cuh")


def _body(name):
    text = open(SRC).read()
    at = text.index("{", text.index(")", re.search(r"\b%s\(" % name, text).start()))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return re.sub(r"//[^\n]*", "", text[at:i + 1])
    raise AssertionError(name)


def test_hit_loop_has_one_path_to_the_next_load():
    body = _body("mma_hits")
    inner = body[body.index("for (uint32_t c = 0"):]
    assert inner.count("tmem_ld16(") == 1 and inner.count("__syncwarp()") == 1
    assert "continue" not in inner and "break" not in inner and "return" not in inner
    # the sync is the last statement of the loop over columns
    assert re.search(r"__syncwarp\(\);\s*\}\s*\}\s*$", inner)


def test_team_barriers_gather_the_warp():
    for name in ("team_count", "team_sync"):
        body = _body(name)
        assert body.index("__syncwarp()") < body.index(".aligned")
