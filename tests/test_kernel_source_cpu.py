"""Rules on the kernels' source that no run can show to be broken."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tnpy_gb300" / "csrc"
SOURCES = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])


def _code(path):
    text = path.read_text()
    text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_shuffles_stand_outside_conditional_expressions(path):
    """A shuffle with a full mask is one instruction for all its lanes: as an operand of ?: the lanes of a warp may take
    it at two places."""
    for statement in re.split(r"[;{}]", _code(path)):
        if "?" in statement:
            operands = statement.split("?", 1)[1]
            assert not re.search(r"\b(lanes_sum|warp_sum|wsum|rr_sum|dc_warp_sum|__shfl\w*|__ballot_sync|__any_sync)\s*\(", operands), statement
