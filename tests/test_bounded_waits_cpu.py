"""Every wait inside a kernel has a limit.  A named barrier has none, so where warps meet at one, a warp whose bounded wait
ran out may not simply leave: it has to come to all the meetings that are ahead, or its partner, whose own wait may have
succeeded a moment later, hangs."""
import re
from pathlib import Path

import pytest

import superscaler_b200

CSRC = Path(superscaler_b200.__file__).parent / "csrc"
NAMED = r'"(?:bar|barrier)(?:\.cta)?\.(?:sync|red)\b'


def _blocks_of_failed_waits(code):
    """What stands between each bounded wait that ran out and the `break` that follows."""
    return [m.group(1) for m in re.finditer(r"if \(!(?:mbar_wait_warp|ring\.wait_full)\([^;{]*\)\s*\{?(.*?)\bbreak;", code, re.S)]


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_warps_that_give_up_still_meet_their_partners(path):
    code = re.sub(r"//[^\n]*", "", path.read_text())
    for body in re.split(r"\b__global__\b", code)[1:]:
        if re.search(NAMED, body):
            left = _blocks_of_failed_waits(body)
            assert left and all("meet_to_the_end(" in b for b in left)


def test_copies_of_the_layernorm_ring_land_before_the_block_ends():
    """The thread that issues the bulk copies waits, with a limit, for the last ones of every stage after its loop."""
    code = re.sub(r"//[^\n]*", "", (CSRC / "layernorm.cu").read_text())
    (kernel,) = [k for k in re.split(r"\b__global__\b", code)[1:] if "bulk_load(" in k]
    behind = kernel[kernel.rindex("bulk_load("):]
    assert "mbar_try_wait(&bars[" in behind[:behind.index("} else {")]
