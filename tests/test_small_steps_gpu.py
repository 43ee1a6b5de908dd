"""Training steps at the sizes where small batches leave a launch of their own: the loss
of a row per warp (32), the token embedding's gradients (256 samples), the column sums out
of the FP32 attention kernels (296 groups, 148 of 32-wide heads, none of 64-wide ones).
Bounds as for all FP32 steps."""
import pytest

from test_op_table_gpu import model, run, train, within

pytestmark = pytest.mark.gpu


def check(cases):
    found = run(cases)
    assert len(found) == len(cases)
    for case, errors in zip(cases, found):
        assert within(errors, 2e-5, 2e-5), (case, errors)


@pytest.mark.parametrize("batch,classes", [(16, 1024), (17, 500), (32, 256), (32, 257), (33, 11)])
def test_losses(batch, classes):
    check([train(batch, model(1, 6, 3, 32, 4, 1, classes))])


@pytest.mark.parametrize("batch,size", [(256, 6), (257, 6), (31, 72)])
def test_token_embeddings(batch, size):
    """On either side of 256 samples, and of a million floats (31 x 577 tokens of 64)."""
    check([train(batch, model(1, size, 3, 32 if size == 6 else 64, 4, 1, 2),
                 precision="fp32")])


@pytest.mark.parametrize("batch,width,heads", [
    (148, 32, 2), (149, 32, 2), (37, 32, 4), (38, 32, 4), (74, 64, 2), (75, 64, 2), (20, 64, 1),
    (20, 128, 2)])
def test_attention_gradients(batch, width, heads):
    check([train(batch, model(1, 12, 4, width, heads, 1, 3), precision="fp32")])
