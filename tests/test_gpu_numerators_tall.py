"""Partial numerators at the fewest rows that go to the tensor cores (2^18), and one size below: term counts around
the smallest batch, a step, an emptying and a launch, and words whose bytes are all at their largest, where the
sums between two emptyings reach their bound. Equal to the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from proving_gb300.synthetic import m31_columns, seeded_qm31

P = (1 << 31) - 1
pytestmark = pytest.mark.gpu


def _check(vals, coeffs, blowup):
    from proving_gb300.backend import BaseColumn, CudaBackend as B
    got, first = B.accumulate_numerators([BaseColumn.from_cpu(v) for v in vals], coeffs, blowup)
    want, want_first = O.accumulate_numerators(list(vals), blowup, coeffs)
    assert list(first) == list(want_first)
    for g, w in zip(got.to_cpu(), want):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("n_terms,log_n,blowup", [(24, 18, 0), (25, 18, 0), (26, 17, 0), (28, 18, 0), (29, 18, 0), (33, 19, 1),
                                                  (64, 18, 0), (65, 18, 0), (255, 18, 0), (257, 18, 0), (290, 18, 0)])
def test_rows_and_terms(n_terms, log_n, blowup):
    coeffs = np.stack([np.stack([seeded_qm31(3 * t + k) for k in range(3)]) for t in range(n_terms)])
    _check(m31_columns(n_terms, n_terms, log_n), coeffs, blowup)


@pytest.mark.parametrize("value", [P - 1, 0x00ffffff, 0x7effffff])
@pytest.mark.parametrize("factor", [P - 1, 0x00ffffff, 0x7f00ffff])
def test_largest_bytes(value, factor):
    _check(np.full((66, 1 << 18), value, np.uint32), np.full((66, 3, 4), factor, np.uint32), 0)
