"""The Wide-Fibonacci constraint kernel's splits: every number of runs a row group's constraints are cut
into (by rows and by columns), runs that come out short or empty, and domains smaller than a row group.
Words equal the oracle's, added to an accumulator that holds values."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from proving_gb300.synthetic import m31_columns, seeded_qm31

P = (1 << 31) - 1
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols,trace_log,eval_log", [
    (3, 1, 2), (3, 4, 5), (9, 5, 6), (17, 3, 4), (18, 7, 8), (34, 6, 9), (35, 10, 11), (66, 12, 13), (67, 4, 5),
    (100, 14, 15), (131, 9, 10), (256, 5, 6), (20, 16, 17), (40, 18, 19)])
def test_composition(n_cols, trace_log, eval_log):
    from proving_gb300.backend import BaseColumn, CudaBackend as B, SecureColumnByCoords
    cols = m31_columns(n_cols + eval_log, n_cols, eval_log)
    base = m31_columns(9, 4, eval_log)
    rc = np.stack([seeded_qm31(k) for k in range(n_cols - 2)])
    acc = SecureColumnByCoords([BaseColumn.from_cpu(c) for c in base])
    B.wide_fib_composition([BaseColumn.from_cpu(c) for c in cols], trace_log, rc, acc)
    want = O.wide_fib_composition(list(cols), eval_log, trace_log, rc)
    for got, b, w in zip(acc.to_cpu(), base, want):
        assert np.array_equal(got, ((b.astype(np.uint64) + w) % P).astype(np.uint32))
