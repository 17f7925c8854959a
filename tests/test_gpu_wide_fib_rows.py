"""The Wide-Fibonacci constraints on both sides of the lines between the row kernel and the split one (8 and 16
constraints, 2^16 rows), added to an accumulator that holds values. Words equal the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from proving_gb300.synthetic import m31_columns, seeded_qm31

P = (1 << 31) - 1
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols", [3, 9, 10, 18, 19])
@pytest.mark.parametrize("trace_log,eval_log", [(1, 2), (8, 9), (14, 15), (15, 16), (15, 17)])
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
