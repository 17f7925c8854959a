"""Barycentric evaluation on the tensor cores at its edges: the sizes around its smallest, column counts
around its groups of 16, unaligned columns (the other kernel), and words whose bytes are all at their
largest, where the sums between two emptyings reach their bound. Values equal the oracle's."""
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


def _check(vals, weights, offset=0):
    from proving_gb300.backend import CudaBackend as B, SecureColumnByCoords
    got = B.barycentric_eval_at_point(_columns(vals, offset), SecureColumnByCoords(_columns(weights)))
    got = got.cpu().numpy().view(np.uint32)
    for g, v in zip(got, vals):
        assert np.array_equal(g, O.barycentric_eval(v, weights))


@pytest.mark.parametrize("log_n,n_cols", [(11, 3), (12, 1), (12, 7), (12, 8), (18, 9), (12, 16), (12, 17), (13, 15), (14, 33), (16, 257), (17, 40),
                                          (20, 5)])
def test_evaluation(log_n, n_cols):
    x, y = pr.random_point(tuple(int(v) for v in seeded_qm31(log_n)))
    _check(m31_columns(log_n, n_cols, log_n), O.barycentric_weights(log_n, x, y))


@pytest.mark.parametrize("log_n", [12, 18])
@pytest.mark.parametrize("value", [P - 1, 0x7f7f7f7f, 0x00ffffff, 0x7effffff, 0])
def test_largest_bytes(log_n, value):
    full = np.full((17, 1 << log_n), value, np.uint32)
    full[3] = P - 1
    full[5, ::3] = 0
    _check(full, [np.full(1 << log_n, w, np.uint32) for w in (P - 1, 0x00ffffff, 0x7effffff, 1)])


def test_unaligned():
    weights = m31_columns(4, 4, 13)
    _check(m31_columns(3, 18, 13), list(weights), offset=1)
