"""The comparison of whole training steps with the oracle: not a number in any result is
an error, in whatever order it comes."""
import math

import numpy as np

import op_table_worker
from test_op_table_gpu import within


def test_not_a_number_is_an_error():
    change = np.zeros(8)
    change[3] = np.nan
    for first, second in ((0.0, change.max()), (change.max(), 0.0)):
        worst = op_table_worker.larger(first, second)
        assert math.isnan(worst)
        for key in ("loss", "logits", "gradient", "moment", "value"):
            assert not within({key: worst}, 1.0, 1.0)
    assert within({"loss": 0.5, "gradient": op_table_worker.larger(0.25, 0.5)}, 1.0, 1.0)
