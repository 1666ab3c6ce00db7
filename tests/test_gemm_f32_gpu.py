"""32-bit products against float64 (CUDA cores, and tensor cores over exact bf16 parts), at the edges of tiles, slabs and splits."""
import pytest
import torch

from nkipy_b200 import ops

pytestmark = pytest.mark.gpu

# rows around tiles of 32 to 160 and pieces of 3200, columns around 128, k around 256, in ragged slabs of 64 and in several ranges; sizes
# and pitches that the CUDA cores keep
CASES = [(1, 256, 4), (15, 255, 8), (16, 257, 12), (17, 1000, 260), (33, 4096, 4096), (64, 512, 20), (65, 770, 1028),
         (130, 2048, 2048), (301, 4096, 4096), (301, 300, 14336), (32, 127, 256), (32, 128, 252), (1, 128, 256), (160, 129, 320),
         (161, 300, 1028), (97, 4096, 4100), (500, 640, 2048), (40, 16, 4096),
         (200, 1, 640), (3201, 130, 14336)]


@pytest.mark.parametrize("m,n,k", CASES)
@pytest.mark.parametrize("pitch", [0, 4, 1])
def test_gemm_f32(m, n, k, pitch):
    """pitch 4: rows of a wider matrix; 1: rows without 16-byte alignment (the general kernel)."""
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n + k)
    x = torch.randn((m, k + pitch), generator=g, device="cuda")[:, :k]
    w = torch.randn((n, k + pitch), generator=g, device="cuda")[:, :k]
    y = ops.linear(x, w)
    want = x.double() @ w.double().T
    # k roundings of partial sums that never exceed the sum of the absolute products; the product of parts that is left out is
    # below 2^-30 of a product
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


def test_error_is_that_of_ordinary_sums():
    g = torch.Generator(device="cuda").manual_seed(5)
    for m, n, k in ((301, 512, 4096), (17, 256, 14336)):
        x, w = torch.randn((m, k), generator=g, device="cuda"), torch.randn((n, k), generator=g, device="cuda")
        want = x.double() @ w.double().T
        # one running fp32 sum per result has about 0.3 sqrt(k) 2^-24 (1.1e-6 at 4096); slabs of 64 stay well below
        assert float((ops.linear(x, w).double() - want).norm() / want.norm()) < 0.3 * k ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("n,k", [(256, 512), (100, 64)])
def test_infinities_and_exact_parts(n, k):
    """One infinity gives infinities of the weights' signs although its lower parts are zero; values with short significands
    give exact products."""
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randint(-8, 9, (40, k), generator=g, device="cuda").float()
    w = torch.randint(1, 9, (n, k), generator=g, device="cuda").float()
    w[1::2] *= -1
    assert torch.equal(ops.linear(x, w), (x.double() @ w.double().T).float())
    x[2, 7] = float("inf")
    w[3, 9] = float("-inf")
    x[:, 9] = 1.0
    y = ops.linear(x, w)
    sign = torch.sign(w[:, 7])
    rows = [j for j in range(n) if j != 3]
    assert torch.equal(y[2, rows], sign[rows] * float("inf"))
    assert (y[[i for i in range(40) if i != 2], 3] == float("-inf")).all()
    ops.raise_on_device_error()


@pytest.mark.parametrize("terms", [1, 2])
def test_few_terms_keep_all_their_bits(terms):
    """Rows in which one or two products count: nothing averages out what is left out of a product."""
    g = torch.Generator(device="cuda").manual_seed(13)
    m, n, k = 160, 512, 4096
    x, w = torch.zeros((m, k), device="cuda"), torch.randn((n, k), generator=g, device="cuda")
    for i in range(terms):
        x[torch.arange(m), (torch.arange(m) * (17 + 14 * i) + 7 * i) % k] = torch.randn(m, generator=g, device="cuda")
    x, w = (t.view(torch.int32).bitwise_or(0xff).view(torch.float32) for t in (x, w))   # full significands
    x[x.abs() < 1e-30] = 0.0
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # the product left out and truncations of the accumulator while it holds lower parts, its truncation per whole product, and the
    # rounding of the sum of two slabs
    assert ((ops.linear(x, w).double() - want).abs() <= (2.0 ** -27 + terms * 2.0 ** -23 + (terms - 1) * 2.0 ** -24) * size).all()
    ops.raise_on_device_error()


def test_not_a_number_costs_no_more_than_numbers():
    """Results that are not numbers are found to be none without a multiply-add for every element of their rows."""
    g = torch.Generator(device="cuda").manual_seed(17)
    x, w = torch.randn((301, 4096), generator=g, device="cuda"), torch.randn((2048, 4096), generator=g, device="cuda")
    nans, column = torch.full_like(x, float("nan")), w.clone()
    column[:, 4090] = float("nan")

    def best_ms(x, w):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            y = ops.linear(x, w)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times), y

    plain, _ = best_ms(x, w)
    for slow, y in (best_ms(nans, w), best_ms(x, column)):
        assert y.isnan().all()
        # 80 results of a warp, each a few loads on top of the product (thousands without the early end)
        assert slow < 100 * plain
    ops.raise_on_device_error()


@pytest.mark.parametrize("splits", [1, 3])
def test_only_infinities_are_summed_again(splits):
    """Infinities against whole numbers (whose lower parts are zero) in rows and columns on both sides of tiles, beside NaNs."""
    from nkipy_b200.ops import mixers

    g = torch.Generator(device="cuda").manual_seed(19)
    m, n, k = 170, 140, 1100
    x = torch.randint(1, 9, (m, k), generator=g, device="cuda").float()
    w = torch.randint(1, 9, (n, k), generator=g, device="cuda").float()
    for i, j in ((0, 0), (159, 700), (160, 1099), (169, 64)):
        x[i, j] = float("inf")
    for i, j in ((31, 5), (127, 1098), (128, 900), (139, 64)):
        w[i, j] = float("-inf")
    x[100, 1099] = float("nan")
    w[130, 3] = float("nan")
    plan = mixers.f32_split_plan
    mixers.f32_split_plan = lambda *a: (160, splits)
    try:
        y = ops.linear(x, w)
    finally:
        mixers.f32_split_plan = plan
    want = (x.double() @ w.double().T).float()
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.nan_to_num(7.0), want.nan_to_num(7.0))
    ops.raise_on_device_error()


@pytest.mark.parametrize("ex,ew", [(-90, 0), (-100, 0), (-105, 0), (-110, 0), (-115, 0), (-120, 0), (-126, 0), (0, -110), (0, -120), (-60, -60), (-66, -66)])
def test_tiny_values_keep_their_bits(ex, ew):
    """Down to results at fp32's smallest normal numbers, where parts and their products would lie below what they can hold."""
    g = torch.Generator(device="cuda").manual_seed(-ex - 2 * ew)
    m, n, k = 170, 140, 516
    x, w = (torch.randn((r, k), generator=g, device="cuda", dtype=torch.float64) * 2.0 ** e for r, e in ((m, ex), (n, ew)))
    x, w = x.float(), w.float()
    x[3] = 0.0
    x[5] *= 2.0 ** 40                                       # a row of another size beside the small ones
    y = ops.linear(x, w)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # ordinary sums: a rounding per term, of a number that may be denormal
    assert ((y.double() - want).abs() <= (k + 8) * (2.0 ** -24 * size + 2.0 ** -150)).all()
    # and no worse in the norm than one running sum per result (0.3 sqrt(k) 2^-24), wherever most terms are normal numbers
    rows = [i for i in range(m) if i not in (3, 5)]
    if ex + ew >= -120:
        assert float((y[rows].double() - want[rows]).norm() / want[rows].norm()) < 0.3 * k ** 0.5 * 2.0 ** -24
    assert (y[3] == 0).all()
    ops.raise_on_device_error()
