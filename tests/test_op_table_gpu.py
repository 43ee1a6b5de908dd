"""Whole training steps through the op table against the numpy oracle, at sizes
where a kernel or a fusion has an edge: every product of the small FMA tiles (one
row, ragged extents, K split over a cluster), the GELU's two fusions on the FMA
and the tensor-core path, accumulated micro-batches, the update of weights that
pending definitions still read.

Bounds, relative to a gradient's largest entry: FP32 products 2e-5 (sums of up
to a few thousand terms, 6e-8 each, through all layers); TF32 products 2e-3 as
for the single products.  The loss moves with the logits: 2e-5, and 1e-3 for
TF32 (2^-11 per operand through a handful of images).  The value's change is
bounded in units of the learning rate by the gradient's error (it is normalised
by the second moment, so by about ten times as much)."""
import json
import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


def model(channels, size, patch, width, heads, layers, classes):
    return dict(channels=channels, size=size, patch=patch, width=width, heads=heads,
                layers=layers, classes=classes)


def train(batch, shape, micro=1, precision="auto", deferred=False, feed="host",
          weights=False):
    return dict(kind="train", batch=batch, micro=micro, precision=precision,
                deferred=deferred, feed=feed, weights=weights, **shape)


def predict(batch, shape):
    return dict(kind="predict", batch=batch, precision="auto", deferred=False, **shape)


FP32 = [
    predict(1, model(1, 28, 4, 128, 8, 2, 11)),
    train(1, model(1, 12, 4, 32, 4, 1, 2)),
    train(8, model(1, 28, 4, 32, 4, 2, 11)),
    train(3, model(3, 15, 5, 72, 9, 2, 5), weights=True),      # ragged everywhere
    train(5, model(1, 28, 7, 40, 5, 1, 13), micro=2, deferred=True),
    train(40, model(1, 28, 4, 128, 8, 1, 11), precision="fp32"),
    train(300, model(1, 16, 4, 64, 4, 1, 10), precision="fp32", deferred=True),
    # More rows of column sums in the slope product than there is room for: shared.
    train(400, model(1, 28, 4, 64, 4, 1, 10), precision="fp32"),
    # More parameters (212) than the optimiser's kernels take as arguments.
    train(2, model(1, 8, 4, 32, 4, 17, 3)),
]
TF32 = [
    train(32, model(1, 28, 4, 128, 8, 2, 11)),
    train(67, model(3, 36, 6, 96, 6, 1, 7), weights=True, deferred=True),
    train(24, model(1, 28, 2, 256, 8, 1, 11), micro=2, feed="dataset"),
]


def run(cases):
    worker = os.path.join(os.path.dirname(os.path.abspath(__file__)), "op_table_worker.py")
    done = subprocess.run([sys.executable, worker, json.dumps(cases)], timeout=600,
                          stdout=subprocess.PIPE, cwd=REPO, check=True)
    return [json.loads(line) for line in done.stdout.decode().splitlines()]


@pytest.mark.parametrize("cases,bound,loss_bound", [(FP32, 2e-5, 2e-5), (TF32, 2e-3, 1e-3)],
                         ids=["fp32", "tf32"])
def test_training_steps_match_the_oracle(cases, bound, loss_bound):
    found = run(cases)
    assert len(found) == len(cases)
    for case, errors in zip(cases, found):
        assert within(errors, bound, loss_bound), (case, errors)


def within(errors, bound, loss_bound):
    """Not a number is within nothing."""
    return (errors.get("declined", 0) == 0 and
            errors.get("logits", 0.0) <= bound and
            errors.get("loss", 0.0) <= loss_bound and
            errors.get("gradient", 0.0) <= bound and
            errors.get("moment", 0.0) <= 2 * bound and
            errors.get("value", 0.0) <= 10 * bound)


def test_weights_at_the_front_of_a_larger_allocation():
    """Their update may go on in another buffer (see device_view_update), which must
    not lose what the host keeps behind them.  (One small step after another repeats
    bit for bit: its products have no slices that meet in memory.)"""
    case = dict(train(2, model(1, 8, 4, 32, 4, 1, 2), precision="fp32"),
                shared_allocations=True)
    assert run([case]) == [{"values": 0, "rest": 0}]


def test_update_of_a_parameter_with_a_pending_gradient():
    """Computing it gives a buffer back that another weight of the same update is still
    read from.  A first step moves every value by the learning rate, in its gradient's
    sign; values of about one are rounded to 6e-8, 6e-5 of that."""
    (found,) = run([dict(kind="gelu_parameter")])
    assert found.keys() == {"w1", "a1", "w2"}
    assert all(error <= 1e-3 for error in found.values()), found


def test_slope_products_on_the_fma_tiles():
    """One row, rows that no vector access fits, slices in a cluster, ragged tiles, and
    more rows of column sums than there is room for (313 and 704 for 296).  FP32 sums of
    n terms, of m for the weights and the bias: 2e-5 of the largest entry."""
    cases = [dict(kind="slope_product", m=m, k=k, n=n) for m, k, n in (
        (1, 5, 3), (50, 512, 128), (50, 33, 515), (300, 257, 66), (4329, 33, 7),
        (4329, 130, 72), (20000, 128, 512), (45000, 64, 30))]
    found = run(cases)
    assert len(found) == len(cases)
    for case, errors in zip(cases, found):
        assert errors.pop("fused") == 1, (case, errors)
        assert all(error <= 2e-5 for error in errors.values()), (case, errors)


def test_gradients_of_small_products_share_a_launch():
    """One row, ragged tiles, slices in a cluster beside more or fewer weight slices;
    tensor-core tiles of 32 and of 64 columns with ragged edges, and products that are
    too large to run side by side.  Bounds as for the products."""
    def cases(precision, *sizes):
        return [dict(kind="gradient_pair", precision=precision, m=m, k=k, n=n)
                for m, k, n in sizes]
    small = cases("fp32", (1, 5, 3), (50, 512, 128), (50, 33, 11), (8, 128, 11),
                  (257, 40, 129), (1000, 32, 96))
    narrow = cases("auto", (1600, 128, 512), (1600, 512, 128), (1601, 100, 388),
                   (4329, 96, 384), (4329, 384, 96), (25, 1024, 1024))
    large = cases("auto", (20000, 128, 512), (9000, 512, 64)) + \
        cases("fp32", (9000, 16, 128))
    found = run(small + narrow + large)
    assert len(found) == len(small + narrow + large)
    for case, errors in zip(small + narrow + large, found):
        assert errors.pop("kernels") == (2 if case in large else 1), (case, errors)
        bound = 2e-5 if case["precision"] == "fp32" else 2e-3
        assert all(error <= bound for error in errors.values()), (case, errors)


def test_skipped_gradients_are_those_of_the_weights_before_the_step():
    """Bounds as for the products (FP32 2e-5, TF32 2e-3 of the largest entry); a step
    moves the weights by about a hundredth of themselves.  Definitions of a block and
    step: the probabilities, four head views forward and four backward, four aliases
    and the skipped gradient; the read computes the latter alone."""
    shape = model(1, 28, 4, 64, 4, 2, 11)
    cases = [dict(train(4, shape, precision="fp32"), skipped_gradients=True),
             dict(train(32, shape), skipped_gradients=True)]
    found = run(cases)
    for errors, bound in zip(found, (2e-5, 2e-3)):
        assert errors["before"] <= bound < errors["after"] / 2, errors
        assert errors["defined"] == 14 and errors["computed"] == 1, errors
    assert len(found) == len(cases)


def test_gradients_computed_later_keep_the_precision_they_were_asked_in():
    """FP32 products that wait (skipped by the GELU's backward pass, or held back for it)
    while the host switches to TF32."""
    tf32 = 2
    shape = model(1, 28, 4, 64, 4, 1, 11)
    skipped, held = run([
        dict(train(4, shape, precision="fp32"), skipped_gradients=True, read_under=tf32),
        dict(kind="slope_product", m=300, k=256, n=64, read_under=tf32)])
    assert skipped["before"] <= 2e-5, skipped
    assert held["activated"] <= 2e-5, held


SETTINGS = dict(max_shift_pixels=2.0, max_rotation_degrees=10.0, max_scale_delta=0.1,
                max_brightness_delta=0.05, max_contrast_delta=0.1,
                noise_standard_deviation=0.01, erasing_probability=0.5,
                erasing_max_side_fraction=0.4, erasing_value=0.5, minimum_value=0.0,
                maximum_value=1.0)
WITHOUT_NOISE = dict(SETTINGS, noise_standard_deviation=0.0)
ONLY_NOISE = dict(SETTINGS, max_shift_pixels=0.0, max_rotation_degrees=0.0,
                  max_scale_delta=0.0, max_brightness_delta=0.0,
                  max_contrast_delta=0.0, erasing_probability=0.0)


def test_augmentation_in_one_kernel_and_in_three():
    """Planes in shared memory (odd and even sizes, several channels, the largest
    that fit and the smallest that do not) against the oracle.  Bound: numpy's cos
    and sin may differ from the host libm by an ulp in the rotation (2e-6 of a
    pixel), the device's log and cos in the noise by 4e-6 of its deviation."""
    cases = [dict(kind="augment", batch=b, channels=c, height=h, width=w, settings=s)
             for b, c, h, w, s in (
                 (37, 1, 28, 28, SETTINGS), (5, 3, 17, 9, SETTINGS),
                 (3, 2, 1, 1, SETTINGS), (9, 1, 33, 32, WITHOUT_NOISE),
                 (4, 3, 12, 31, ONLY_NOISE), (2, 1, 160, 160, SETTINGS),
                 (2, 1, 161, 160, SETTINGS))]
    found = run(cases)
    assert len(found) == len(cases)
    for case, errors in zip(cases, found):
        assert errors["status"] == 0 and errors["stream"] == 0, case
        assert errors["pixel"] <= 2.1e-6, (case, errors)
