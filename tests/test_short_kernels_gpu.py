"""The kernels of small batches where their split of the work has an edge: FP32
attention with one, two or four lanes per row (rows that do not fill a warp, one
token, the longest sequences, the group counts at which the lanes change),
and products on 32- and 64-column tiles (ragged extents, reductions shorter and
longer than the load ring, both GELU epilogues), and products with one thin extent
(every register form, ragged widths, the widths and rows at which the tiled kernel
takes over), and sums over matrices of many columns.

Bounds: FP32 attention 1e-5 / 2e-5 of the largest entry, TF32 products 2e-3, as
for the same kernels at other sizes."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import vit_oracle as vo
from test_kernels_gpu import FP32, TF32, close, dev, host, lib, ptr, size  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,seq,hd", [
    (3, 1, 64), (2, 128, 64), (5, 33, 64), (2, 128, 32), (2, 128, 8), (7, 65, 16),
    (9, 63, 8), (148, 7, 32), (149, 7, 32), (149, 128, 32), (600, 50, 16), (1184, 5, 8),
    (1185, 50, 8), (149, 128, 16), (3, 33, 32),
])
def test_short_attention_fp32(lib, groups, seq, hd):
    rng = np.random.RandomState(groups * seq + hd)
    rows, scale = groups * seq, 1.0 / np.sqrt(hd)
    q, k, v, dout, dq0, dk0, dv0 = (rng.randn(rows, hd) for _ in range(7))
    tq, tk, tv, tdo, tdq, tdk, tdv = map(dev, (q, k, v, dout, dq0, dk0, dv0))
    to = torch.empty(rows, hd, device="cuda")
    dots = torch.empty(rows, device="cuda")
    assert lib.vitb200_k_attention(
        ptr(tq), ptr(tk), ptr(tv), None, ptr(to), size(groups), size(seq), size(hd),
        ctypes.c_float(scale), FP32, None) == 0
    assert lib.vitb200_k_attention_backward(
        ptr(tq), ptr(tk), ptr(tv), None, ptr(to), ptr(tdo), ptr(tdq), ptr(tdk),
        ptr(tdv), ptr(dots), size(groups), size(seq), size(hd),
        ctypes.c_float(scale), FP32, None) == 0
    p, o = vo.multi_head_attention(q, k, v, groups, seq, scale)
    dq, dk, dv = vo.multi_head_attention_backward(q, k, v, p, dout, groups, seq, scale)
    close(host(to), o, 1e-5)
    close(host(tdq), dq0 + dq, 2e-5)
    close(host(tdk), dk0 + dk, 2e-5)
    close(host(tdv), dv0 + dv, 2e-5)


@pytest.mark.parametrize("m,k,n", [
    (16, 16, 64), (129, 40, 68), (1600, 512, 128), (1600, 128, 512), (4329, 96, 288),
    (2000, 1024, 96), (640, 512, 512), (12801, 128, 128),
])
def test_products_of_few_tiles(lib, m, k, n):
    rng = np.random.RandomState(m + k + n)
    x, w, bias = rng.randn(m, k), rng.randn(k, n) / np.sqrt(k), rng.randn(n)
    dy, hidden = rng.randn(m, n), rng.randn(m, k) * 1.5
    dx0, dw0 = rng.randn(m, k), rng.randn(k, n)
    tx, tw, tb, tdy, th, tdx, tdw = map(dev, (x, w, bias, dy, hidden, dx0, dw0))
    ty, tgelu = (torch.empty(m, n, device="cuda") for _ in range(2))
    tdh = torch.empty(m, k, device="cuda")
    tsums = torch.full((296, k), 3.0, device="cuda")
    extents = size(m), size(k), size(n), TF32, None
    assert lib.vitb200_k_gemm_fused(ptr(tx), ptr(tw), ptr(ty), ptr(tb), ptr(tgelu),
                                    None, None, *extents) == 0
    assert lib.vitb200_k_gemm_backward(ptr(tx), ptr(tw), ptr(tdy), ptr(tdx), ptr(tdw),
                                       *extents) == 0
    assert lib.vitb200_k_gemm_backward_gelu(ptr(tw), ptr(tdy), ptr(th), ptr(tdh),
                                            ptr(tsums), *extents) == 0
    y = x @ w + bias
    dh = vo.gelu_backward(hidden, dy @ w.T)
    close(host(ty), y, 2e-3)
    close(host(tgelu), vo.gelu(y), 2e-3)
    close(host(tdx), dx0 + dy @ w.T, 2e-3)
    close(host(tdw), dw0 + x.T @ dy, 2e-3)
    close(host(tdh), dh, 2e-3)
    stored = host(tdh).astype(np.float64).sum(axis=0)
    sums = host(tsums).astype(np.float64).sum(axis=0)
    assert np.abs(sums - stored).max() <= 1e-4 * max(np.abs(stored).max(), 1.0)
    assert lib.vitb200_tensor_core_status() == 0


@pytest.mark.parametrize("m,k,n", [
    (8192, 4, 256), (8193, 4, 384), (9001, 1, 4), (8200, 7, 512), (8200, 8, 256),
    (8197, 9, 128), (8197, 12, 96), (10007, 13, 60), (8192, 16, 128), (8192, 4, 1024),
    (8192, 4, 1028), (9000, 12, 132), (300000, 4, 64),
])
def test_thin_products(lib, m, k, n):
    """Features of a small patch: FP32 sums of at most 16 terms, of n terms and
    (the weights') of m terms, 6e-8 each."""
    rng = np.random.RandomState(m + k + n)
    x, w, bias, dy = rng.randn(m, k), rng.randn(k, n), rng.randn(n), rng.randn(m, n)
    dx0, dw0 = rng.randn(m, k), rng.randn(k, n)
    tx, tw, tb, tdy, tdx, tdw = map(dev, (x, w, bias, dy, dx0, dw0))
    ty = torch.empty(m, n, device="cuda")
    extents = size(m), size(k), size(n), FP32, None
    assert lib.vitb200_k_gemm_fused(ptr(tx), ptr(tw), ptr(ty), ptr(tb), None, None, None,
                                    *extents) == 0
    assert lib.vitb200_k_gemm_backward(ptr(tx), ptr(tw), ptr(tdy), ptr(tdx), ptr(tdw),
                                       *extents) == 0
    close(host(ty), x @ w + bias, 1e-5)
    close(host(tdx), dx0 + dy @ w.T, 1e-5)
    close(host(tdw), dw0 + x.T @ dy, 2e-5)


@pytest.mark.parametrize("rows,cols,offset", [
    (1, 16384, 0), (7, 16388, 0), (64, 24600, 1), (9, 400004, 0), (700, 16384, 0),
    (64, 16380, 0),
    (2048, 6400, 0), (2049, 4096, 1), (2048, 4092, 0),
])
def test_sums_of_many_columns(lib, rows, cols, offset):
    """Up to 2049 terms, 6e-8 each, in FP32; the sums may start at any float."""
    rng = np.random.RandomState(rows + cols)
    x, base = rng.randn(rows, cols), rng.randn(cols + offset)
    tx, tout = dev(x), dev(base)
    lib.vitb200_k_column_sums(ptr(tx), ctypes.c_void_p(tout.data_ptr() + 4 * offset),
                              size(rows), size(cols), None)
    expected = base.copy()
    expected[offset:] += x.sum(axis=0)
    close(host(tout), expected, 1e-5)


def test_gelu_slope_of_large_values(lib):
    """The slope in the product's epilogue far out: one to the right, zero to the
    left, for every value whose square is finite (the TF32 product's bound)."""
    m, k, n = 256, 128, 64
    rng = np.random.RandomState(3)
    w, dy = rng.randn(k, n) / np.sqrt(n), rng.randn(m, n)
    hidden = np.exp(rng.uniform(np.log(5.0), np.log(1.8e19), (m, k)))
    hidden *= rng.choice([-1.0, 1.0], (m, k))
    tw, tdy, th, tdh = map(dev, (w, dy, hidden, np.zeros((m, k))))
    assert lib.vitb200_k_gemm_backward_gelu(ptr(tw), ptr(tdy), ptr(th), ptr(tdh), None,
                                            size(m), size(k), size(n), TF32, None) == 0
    close(host(tdh), np.where(hidden > 0, dy @ w.T, 0.0), 2e-3)


@pytest.mark.parametrize("rows,cols", [(64, 24600), (128, 50432), (700, 16384),
                                       (2049, 4096), (2048, 6400), (10000, 4096)])
def test_error_of_sums_of_many_columns(lib, rows, cols):
    """No larger than what the narrow sums' kernel leaves: lanes of a 32nd of a slice's
    rows, a tree of five levels, an addition per slice.  Along a row of L additions
    the running sum's square is half the result's on average, in a tree every level's
    is the result's.  Rounding a value of significand s leaves 2^-24 / (sqrt(3) s) of
    it, over the significands of normal sums 0.44 x 2^-24; the bound takes 0.475."""
    rng = np.random.RandomState(rows)
    x = rng.randn(rows, cols).astype(np.float32)
    tx, tout = dev(x), torch.zeros(cols, device="cuda")
    lib.vitb200_k_column_sums(ptr(tx), ptr(tout), size(rows), size(cols), None)
    exact = x.astype(np.float64).sum(axis=0)
    error = np.linalg.norm(host(tout) - exact) / np.linalg.norm(exact)
    strips = (cols + 127) // 128
    slices = max(1, min((296 + strips - 1) // strips, (rows + 127) // 128))
    row = np.ceil(rows / slices / 32)
    bound = 2.0 ** -24 * 0.475 * np.sqrt(row / 2 + 5 + slices / 2)
    assert error <= bound, (error, bound)


def split_row_bound(m, n, k):
    """2-norm error of a gradient [m, n], sums of k terms, in slices of at least 128
    of them, as many as make two tiles of 64 x 64 per SM; per addition as in
    test_error_of_sums_of_many_columns."""
    tiles = -(-m // 64) * -(-n // 64)
    slices = max(1, min(-(-296 // tiles), -(-k // 128)))
    rows = -(-(-(-k // slices)) // 16) * 16
    return 2.0 ** -24 * 0.475 * np.sqrt((min(rows, k) + slices) / 2)


@pytest.mark.parametrize("m,k,n", [
    (8200, 9, 128), (8625, 1, 256), (10007, 16, 128), (20000, 4, 256), (12000, 12, 1024),
    (9000, 4, 4),
])
def test_error_of_thin_weight_gradients(lib, m, k, n):
    rng = np.random.RandomState(m + n)
    x, dy = (rng.randn(m, c).astype(np.float32) for c in (k, n))
    tx, tdy, tw = dev(x), dev(dy), dev(rng.randn(k, n))
    tdx, tdw = torch.zeros(m, k, device="cuda"), torch.zeros(k, n, device="cuda")
    assert lib.vitb200_k_gemm_backward(ptr(tx), ptr(tw), ptr(tdy), ptr(tdx), ptr(tdw),
                                       size(m), size(k), size(n), FP32, None) == 0
    exact = x.astype(np.float64).T @ dy.astype(np.float64)
    error = np.linalg.norm(host(tdw) - exact) / np.linalg.norm(exact)
    assert error <= split_row_bound(k, n, m), (error, split_row_bound(k, n, m))


@pytest.mark.parametrize("m,k,n", [
    (4329, 96, 288), (1972, 128, 1024), (18321, 32, 256), (2905, 32, 1536),
    (4423, 64, 1024), (700, 1000, 300), (65, 33, 4000),
])
def test_error_of_accumulated_gradients(lib, m, k, n):
    """Both gradients of an FP32 product where its slices decide the error."""
    rng = np.random.RandomState(m + n)
    x, w, dy = (rng.randn(*s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    tx, tw, tdy = map(dev, (x, w, dy))
    tdx, tdw = torch.zeros(m, k, device="cuda"), torch.zeros(k, n, device="cuda")
    assert lib.vitb200_k_gemm_backward(ptr(tx), ptr(tw), ptr(tdy), ptr(tdx), ptr(tdw),
                                       size(m), size(k), size(n), FP32, None) == 0
    x, w, dy = (a.astype(np.float64) for a in (x, w, dy))
    for found, exact, bound in ((tdx, dy @ w.T, split_row_bound(m, k, n)),
                                (tdw, x.T @ dy, split_row_bound(k, n, m))):
        error = np.linalg.norm(host(found) - exact) / np.linalg.norm(exact)
        assert error <= bound, (error, bound)
