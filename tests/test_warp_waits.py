"""Waits of kernels that run out: a warp whose lanes take part in matrix instructions and shuffles must leave as a whole."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "csrc" / "kernels"


@pytest.mark.parametrize("name", sorted(f.name for f in KERNELS.glob("*.cu*") if "mbar_wait(" in f.read_text()))
def test_no_lane_returns_alone(name):
    """A kernel does not return on what a single lane's wait says (loops of one elected lane leave by `break`)."""
    source = re.sub(r"//[^\n]*", "", (KERNELS / name).read_text())
    alone = re.findall(r"if \(!mbar_wait(?:_cluster)?\([^;{}]*\)\)\s*\{?\s*return", source)
    assert not alone
