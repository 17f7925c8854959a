"""Barycentric evaluation around the column counts from which the tensor cores take it (8, 9 or 12, by the rows).
Values equal the oracle's."""
import pytest

import test_gpu_bary_mma as bary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,n_cols", [(17, 7), (17, 8), (18, 11), (18, 12), (19, 8), (19, 9), (21, 8), (21, 9), (22, 7), (22, 8)])
def test_evaluation(log_n, n_cols):
    bary.test_evaluation(log_n, n_cols)
