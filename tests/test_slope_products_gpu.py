"""Products behind a GELU, backward, on either side of the lines between the variants of
their epilogue (320, 512 and 768 terms), with whole and ragged rows, and on 128 x 256 tiles
whose second half is outside the matrix."""
import pytest

import test_kernels_gpu as kernels

pytestmark = pytest.mark.gpu
lib = kernels.lib


@pytest.mark.parametrize("m,k,n", [
    (25216, 512, 288), (25217, 384, 320), (25216, 640, 324), (20001, 512, 384),
    (20000, 768, 448), (20033, 1024, 512), (20033, 1024, 572), (20001, 512, 576), (12800, 512, 640),
    (9001, 1152, 640), (9000, 1024, 700), (12801, 384, 1024), (5000, 640, 1028)])
def test_slopes_of_all_reductions(lib, m, k, n):
    kernels.test_gemm_backward_through_gelu(lib, m, k, n, True)
