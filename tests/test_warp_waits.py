"""Waits in kernels: a warp whose lanes take part in matrix instructions and shuffles must leave as a whole when one runs out, and a
launch that others read ahead of must itself have waited."""
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


def test_the_convolution_of_a_step_waits_before_it_lets_the_step_begin():
    """The step reads gates and states ahead of its own wait: all kernels before the convolution must be done by then."""
    source = re.sub(r"//[^\n]*", "", (KERNELS / "head_recurrence.cu").read_text())
    body = source[source.index("conv_step_kernel("):source.index("head_rec_step_kernel(")]
    assert 0 < body.index("griddep_wait();") < body.index("griddep_launch();")
