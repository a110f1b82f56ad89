"""Grids follow the device's SM count: no launch code has a number of SMs written in."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "btorch_b200" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_no_sm_count_in_expressions(path):
    code = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
    assert not re.search(r"\b148\b\s*\*|\*\s*148\b", code)
