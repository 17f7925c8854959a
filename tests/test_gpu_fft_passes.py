"""FFT passes at the edges of their kernels: every pass length in both tile shapes, column counts
around a block's warps, a strided pass at the lowest layer it can start at, and columns that are not
16-byte aligned. Words equal the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from proving_gb300.synthetic import m31_columns

pytestmark = pytest.mark.gpu

# (layers, plan): contiguous passes of 6-11 layers alone and before strided ones of 1-11
PLANS = [(6, (6,)), (7, (7,)), (8, (8,)), (9, (9,)), (10, (10,)), (11, (11,)), (9, (3, 6)), (11, (6, 5)), (13, (3, 10)),
         (14, (3, 11)), (15, (4, 11)), (13, (4, 9)), (13, (7, 6)), (15, (8, 7)), (17, (9, 8)), (14, (10, 4)),
         (14, (11, 3)), (12, (5, 4, 3))]


def _run(log_src, log_n, inverse, plan, n_cols, offset):
    from proving_gb300 import autotune
    from proving_gb300.backend import BaseColumn, CudaBackend as B, canonic_half_coset
    tree = B.precompute_twiddles(canonic_half_coset(log_n + 1))
    tw, itw = O.canonic_twiddles(log_n + 1)
    vals = m31_columns(7 * log_n + log_src, n_cols, log_src)

    def placed(words, log):
        # each column at `offset` words past a 256-byte boundary
        buf = torch.zeros(n_cols, (1 << log) + 64, dtype=torch.int32, device="cuda")
        cols = [BaseColumn(buf[i, offset:offset + (1 << log)]) for i in range(n_cols)]
        if words is not None:
            for c, w in zip(cols, words):
                c.data.copy_(torch.from_numpy(w.view(np.int32)))
        return buf, cols

    keep, cols = placed(vals, log_src)
    autotune.set_plan(inverse, log_n, log_src, plan)
    try:
        if inverse:
            B.interpolate_columns(cols, tree)
            got, want = cols, O.interpolate_batch(list(vals), itw)
        else:
            keep2, out = placed(None, log_n)
            got = B.evaluate_polynomials(cols, log_n, tree, out)
            want = O.evaluate_batch(list(vals), [log_n] * n_cols, tw)
            assert int(keep2[:, :offset].abs().sum()) == 0 and int(keep2[:, offset + (1 << log_n):].abs().sum()) == 0
    finally:
        autotune.set_plan(inverse, log_n, log_src, [])
    for c, w in zip(got, want):
        assert np.array_equal(c.to_cpu(), w)


@pytest.mark.parametrize("layers,plan", PLANS)
@pytest.mark.parametrize("n_cols", [1, 3, 5])
def test_interpolate_passes(layers, plan, n_cols):
    _run(layers, layers, True, plan, n_cols, 0)


@pytest.mark.parametrize("layers,plan", PLANS)
@pytest.mark.parametrize("blowup", [0, 1, 3])
def test_evaluate_passes(layers, plan, blowup):
    _run(layers, layers + blowup, False, plan, 2, 0)


@pytest.mark.parametrize("layers,plan", [(6, (6,)), (10, (10,)), (11, (11,)), (13, (7, 6)), (14, (3, 11))])
@pytest.mark.parametrize("inverse", [True, False])
def test_unaligned_columns(layers, plan, inverse):
    _run(layers, layers if inverse else layers + 1, inverse, plan, 3, 1)
