"""Which products fetch weight tiles before the kernel ahead of them has finished (the launch's arguments, on the CPU)."""
import pytest
import torch

from nkipy_b200 import ops


class Launches:
    """Stands in for the kernel library."""

    def __init__(self):
        self.static = None

    def nkb_gemm_bf16_2cta(self, *args):
        assert self.static is None
        self.static = args[-3]
        return 0


@pytest.mark.parametrize("rows,splits,static,ahead", [(300, 1, True, 1), (300, 1, False, 0), (511, 1, True, 1), (512, 1, True, 0),
                                                      (4096, 1, True, 0), (4096, 1, False, 0), (414, 2, True, 1), (640, 2, True, 1),
                                                      (640, 2, False, 0)])
def test_large_whole_products_wait_for_their_weights(monkeypatch, rows, splits, static, ahead):
    """A w that the kernel before has written is safe there without weights_static=False."""
    lib = Launches()
    monkeypatch.setattr(ops, "_native", lambda t: True)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops._lib, "lib", lambda: lib)
    x, w = torch.empty((rows, 1024), dtype=torch.bfloat16), torch.empty((4096, 1024), dtype=torch.bfloat16)
    ops.linear(x, w, swap=False, splits=splits, weights_static=static)
    assert lib.static == ahead
