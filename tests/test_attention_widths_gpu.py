"""FP32 attention of long sequences at head dimensions below, at and above those that its
kernels are built for (48, 80, 96 and 112 beside 8, 16, 32, 64 and 128)."""
import pytest

import test_kernels_gpu as kernels

pytestmark = pytest.mark.gpu
lib = kernels.lib


@pytest.mark.parametrize("groups,seq,hd", [
    (2, 130, 40), (1, 193, 48), (1, 129, 49), (3, 129, 72), (2, 192, 80), (1, 200, 81),
    (2, 191, 96), (1, 129, 97), (2, 200, 112), (1, 130, 113)])
def test_head_dimensions(lib, groups, seq, hd):
    kernels.test_attention_forward_and_backward(lib, groups, seq, hd, kernels.FP32)
