"""Large FP32 products, whose operands are split for the tensor cores: their errors, what
has no finite parts, and column sums on either side of their dispatch."""
import ctypes
import os

import pytest
import torch

from conftest import PACKAGE
from oracle import vit_oracle as vo
from test_op_table_gpu import run

pytestmark = pytest.mark.gpu

FP32 = 1
INF, NAN = float("inf"), float("nan")


@pytest.fixture(scope="module")
def lib():
    return ctypes.CDLL(os.path.join(PACKAGE, "libvitb200.so"))


def ptr(tensor):
    return ctypes.c_void_p(tensor.data_ptr() if tensor is not None else None)


def sizes(m, k, n):
    return (*(ctypes.c_size_t(x) for x in (m, k, n)), FP32, None)


def error(got, want):
    torch.cuda.synchronize()
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("m,k,n,input_bound,weight_bound", [
    (512, 768, 768, 0.66e-7, 0.63e-7), (1600, 512, 512, 3.1e-7, 0.74e-7),
    (1600, 512, 2048, 0.72e-7, 0.90e-7), (2048, 512, 2048, 0.72e-7, 0.72e-7),
    (4096, 512, 2048, 6.1e-7, 0.82e-7), (10000, 128, 512, 3.1e-7, 1.05e-7),
    (10000, 100, 132, 1.7e-7, 1.15e-7), (20000, 512, 2048, 6.1e-7, 1.54e-7)])
def test_sums_of_positive_terms(lib, m, k, n, input_bound, weight_bound):
    """Gradients that are added to, over rows that FMAs take in slices: nothing cancels, so
    that what the tensor core cuts off adds up.  The bounds are the errors that the FMA
    kernels have at these sizes, plus 2 %."""
    generator = torch.Generator(device="cuda").manual_seed(m + k + n)
    x, w, dy = (torch.rand(*shape, generator=generator, device="cuda")
                for shape in ((m, k), (k, n), (m, n)))
    dx, dw = torch.zeros(m, k, device="cuda"), torch.zeros(k, n, device="cuda")
    assert lib.vitb200_k_gemm_backward(ptr(x), ptr(w), ptr(dy), ptr(dx), ptr(dw),
                                       *sizes(m, k, n)) == 0
    found = error(dx, dy.double() @ w.double().T), error(dw, x.double().T @ dy.double())
    assert found[0] <= input_bound and found[1] <= weight_bound, found


@pytest.mark.parametrize("exponents", [(0, 0), (108, 0), (0, 108), (60, 60), (108, -40)])
def test_small_operands_keep_their_bits(lib, exponents):
    """Down to 2^-108 (values of a normal distribution reach further down, with less
    weight).  Bound as for ordinary values: a rounding (6e-8 at most, 2.5e-8 rms) per 64
    terms and four truncated additions (6e-8 on average) between two of them."""
    m, k, n = 12800, 128, 384
    generator = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(m, k, generator=generator, device="cuda") * 2.0 ** -exponents[0]
    w = torch.randn(k, n, generator=generator, device="cuda") * 2.0 ** -exponents[1]
    y = torch.empty(m, n, device="cuda")
    assert lib.vitb200_k_gemm(ptr(x), ptr(w), ptr(y), *sizes(m, k, n)) == 0
    found = error(y, x.double() @ w.double())
    assert found <= 1.3e-7, found


def agree(got, want, tolerance):
    """Infinities and NaNs where the reference has them; the rest to `tolerance` of its
    largest entry."""
    torch.cuda.synchronize()
    got, finite = got.double(), want.isfinite()
    assert torch.equal(got.nan_to_num(0.0, 1.0, -1.0)[~finite],
                       want.nan_to_num(0.0, 1.0, -1.0)[~finite])
    assert torch.equal(got.isnan(), want.isnan())
    worst = (got - want)[finite].abs().max() / want[finite].abs().max()
    assert float(worst) <= tolerance, float(worst)


@pytest.mark.parametrize("m,k,n", [(12800, 128, 384), (12833, 100, 132), (13001, 260, 36)])
def test_infinities_in_every_form(lib, m, k, n):
    """Whole and ragged tiles.  Sums of up to 260 terms 1e-5, of m terms 2e-5."""
    generator = torch.Generator(device="cuda").manual_seed(m)
    def normal(*shape):
        return torch.randn(*shape, generator=generator, device="cuda")
    x, w, dy, bias = normal(m, k), normal(k, n), normal(m, n), normal(n)
    x[3, 7], x[m - 1, k - 1], x[200, 9], x[201, 5] = INF, -INF, NAN, INF
    x[201, 6] = -INF
    dy[0, 0], dy[m - 1, n - 1], dy[77, 3] = -INF, INF, NAN
    dx0, dw0 = normal(m, k), normal(k, n)
    y, gelu, dx, dw = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda"), \
        dx0.clone(), dw0.clone()
    assert lib.vitb200_k_gemm_fused(ptr(x), ptr(w), ptr(y), ptr(bias), ptr(gelu), None, None,
                                    *sizes(m, k, n)) == 0
    assert lib.vitb200_k_gemm_backward(ptr(x), ptr(w), ptr(dy), ptr(dx), ptr(dw),
                                       *sizes(m, k, n)) == 0
    want = x.double() @ w.double() + bias.double()
    agree(y, want, 1e-5)
    finite = want.isfinite().all(dim=1)
    expected = torch.from_numpy(vo.gelu(want[finite].cpu().numpy())).cuda()
    agree(gelu[finite], expected, 1e-5)
    agree(dx, dx0.double() + dy.double() @ w.double().T, 1e-5)
    agree(dw, dw0.double() + x.double().T @ dy.double(), 2e-5)
    assert lib.vitb200_tensor_core_status() == 0


def test_infinity_in_a_long_reduction(lib):
    """The values beside it are computed again over the whole of it, which takes longer
    than the kernel's roles wait for one another (a tile has no slices, a CTA two tiles):
    nobody may be waiting.  Bound: a chain of FMAs, 1.8e-8 times the root of its terms."""
    m, k, n = 2048, 300000, 2048
    generator = torch.Generator(device="cuda").manual_seed(1)
    x, w = (torch.randn(*shape, generator=generator, device="cuda")
            for shape in ((m, k), (k, n)))
    x[70, k - 5] = INF
    y = torch.empty(m, n, device="cuda")
    assert lib.vitb200_k_gemm(ptr(x), ptr(w), ptr(y), *sizes(m, k, n)) == 0
    torch.cuda.synchronize()
    assert lib.vitb200_tensor_core_status() == 0
    assert torch.equal(y[70], INF * w[k - 5].sign())
    rows = [0, 63, 64, 69, 71, 95, 96, 2047]   # of the same values, and of others
    for row in rows:
        want = x[row].double() @ w.double()
        assert error(y[row], want) <= 1.8e-8 * k ** 0.5, (row, error(y[row], want))


def test_infinities_early_and_late_in_a_walk_of_many_tiles(lib):
    """549 tiles per CTA on 148 SMs, more than what is put off fits its 512 places.  Sums
    of 64 terms: 1e-5 of the largest."""
    m, k, n = 1300000, 64, 1024
    generator = torch.Generator(device="cuda").manual_seed(2)
    x, w = (torch.randn(*shape, generator=generator, device="cuda")
            for shape in ((m, k), (k, n)))
    rows = [5, 100000, 1212415, 1212416, m - 1]
    for row in rows:
        x[row, 3] = INF
    y = torch.full((m, n), 7.0, device="cuda")
    assert lib.vitb200_k_gemm(ptr(x), ptr(w), ptr(y), *sizes(m, k, n)) == 0
    torch.cuda.synchronize()
    assert lib.vitb200_tensor_core_status() == 0
    for row in rows:
        assert torch.equal(y[row], INF * w[3].sign())
        beside = [row - 1 if row == m - 1 else row + 1, row // 32 * 32]
        for other in beside:
            if other not in rows:
                agree(y[other], x[other].double() @ w.double(), 1e-5)


def test_slope_products_on_both_sides_of_the_dispatch():
    """FMA tiles with more rows of column sums than there is room for (313 and 501 for
    296): rows of dY that are no multiple of 16 bytes; and split products with whole and
    ragged tiles.  Bounds as for the FMA tiles: 2e-5 of the largest entry."""
    cases = [dict(kind="slope_product", m=m, k=k, n=n) for m, k, n in (
        (20000, 128, 511), (32001, 64, 129), (20000, 128, 512), (12833, 100, 132),
        (13001, 516, 36))]
    found = run(cases)
    assert len(found) == len(cases)
    for case, errors in zip(cases, found):
        assert errors.pop("fused") == 1, (case, errors)
        assert all(error <= 2e-5 for error in errors.values()), (case, errors)
