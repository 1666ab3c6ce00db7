"""32-bit products on the CUDA cores against float64, at the edges of tiles, slabs and splits."""
import pytest
import torch

from nkipy_b200 import ops

pytestmark = pytest.mark.gpu

# rows around the tiles of 16, 32 and 64; columns around 256 and without whole vectors; k of one slab, a ragged one, and long
# enough to be split over a cluster
CASES = [(1, 256, 4), (15, 255, 8), (16, 257, 12), (17, 1000, 260), (33, 4096, 4096), (64, 512, 20), (65, 770, 1028),
         (130, 2048, 2048), (301, 4096, 4096), (301, 300, 14336)]


@pytest.mark.parametrize("m,n,k", CASES)
@pytest.mark.parametrize("pitch", [0, 4, 1])
def test_gemm_f32(m, n, k, pitch):
    """pitch 4: rows of a wider matrix; 1: rows without 16-byte alignment (the general kernel)."""
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n + k)
    x = torch.randn((m, k + pitch), generator=g, device="cuda")[:, :k]
    w = torch.randn((n, k + pitch), generator=g, device="cuda")[:, :k]
    y = ops.linear(x, w)
    want = x.double() @ w.double().T
    # k roundings of partial sums that never exceed the sum of the absolute products
    bound = (k + 8) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert y.shape == (m, n) and y.dtype == torch.float32
    assert ((y.double() - want).abs() <= bound).all()
    ops.raise_on_device_error()


def test_rows_do_not_depend_on_the_others():
    """A row of infinities, and a NaN, stay in their own rows."""
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w = torch.randn((70, 1024), generator=g, device="cuda"), torch.randn((300, 1024), generator=g, device="cuda")
    clean = ops.linear(x, w)
    x[69] = float("inf")
    x[3, 5] = float("nan")
    y = ops.linear(x, w)
    keep = [i for i in range(70) if i not in (3, 69)]
    assert torch.equal(y[keep], clean[keep]) and y[3].isnan().all() and not y[69].isfinite().any()
