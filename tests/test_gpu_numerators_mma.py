"""Partial numerators on the tensor cores at their edges: row counts around a warp's and a block's, term
counts around a step's, an emptying's and a launch's, unaligned columns (the other kernel), and words whose
bytes are all at their largest, where the sums between two emptyings reach their bound. Equal to the
oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from proving_gb300 import prover as pr
from proving_gb300.synthetic import m31_columns, seeded_qm31

pytestmark = pytest.mark.gpu

P = (1 << 31) - 1


def _columns(vals, offset=0):
    from proving_gb300.backend import BaseColumn
    out = []
    for v in vals:
        buf = torch.zeros(v.size + 16, dtype=torch.int32, device="cuda")
        buf[offset:offset + v.size] = torch.from_numpy(np.ascontiguousarray(v).view(np.int32)).cuda()
        out.append(BaseColumn(buf[offset:offset + v.size]))
    return out


def _check(vals, coeffs, blowup, offset=0):
    from proving_gb300.backend import CudaBackend as B
    got, first = B.accumulate_numerators(_columns(vals, offset), coeffs, blowup)
    want, want_first = O.accumulate_numerators(list(vals), blowup, coeffs)
    assert list(first) == list(want_first)
    for g, w in zip(got.to_cpu(), want):
        assert np.array_equal(g, w)


def _coeffs(n):
    _, y = pr.random_point(tuple(int(v) for v in seeded_qm31(n)))
    return np.stack([O.line_coeffs(y, seeded_qm31(t), seeded_qm31(1000 + t)) for t in range(n)])


@pytest.mark.parametrize("n_terms,log_n,blowup", [(24, 8, 1), (25, 8, 1), (26, 6, 0), (26, 6, 1), (32, 9, 0),
                                                  (33, 10, 2), (64, 13, 1), (65, 12, 1), (255, 8, 0), (257, 9, 1),
                                                  (290, 7, 1), (515, 7, 1), (33, 16, 0), (41, 18, 1), (27, 20, 0)])
def test_rows_and_terms(n_terms, log_n, blowup):
    _check(m31_columns(n_terms, n_terms, log_n), _coeffs(n_terms), blowup)


@pytest.mark.parametrize("value", [P - 1, 0x7f7f7f7f, 0x00ffffff, 0x7effffff, 0])
@pytest.mark.parametrize("factor", [P - 1, 0x00ffffff, 0x7effffff, 0x7f00ffff])
def test_largest_bytes(value, factor):
    _check(np.full((130, 256), value, np.uint32), np.full((130, 3, 4), factor, np.uint32), 0)


def test_unaligned():
    _check(m31_columns(3, 30, 10), _coeffs(30), 1, offset=1)
