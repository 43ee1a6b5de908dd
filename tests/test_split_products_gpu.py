"""Large FP32 products, whose operands are split for the tensor cores."""
import ctypes
import os

import pytest
import torch

from conftest import PACKAGE

pytestmark = pytest.mark.gpu

FP32 = 1


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
