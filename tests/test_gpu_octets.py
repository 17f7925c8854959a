"""The eight-row kernels of the barycentric weights and DEEP quotients at their edges: the smallest
domains (below and at eight points), points of the base field on the domain and their antipodes, points
off the circle and unaligned columns (the row kernels), lifted accumulations of every ratio and several
sample points. Words equal the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from proving_gb300 import prover as pr
from proving_gb300.synthetic import qm31_column, seeded_qm31

pytestmark = pytest.mark.gpu


def _secure(coords, offset=0):
    from proving_gb300.backend import BaseColumn, SecureColumnByCoords
    cols = []
    for c in coords:
        buf = torch.zeros(c.size + 16, dtype=torch.int32, device="cuda")
        buf[offset:offset + c.size] = torch.from_numpy(c.view(np.int32)).cuda()
        cols.append(BaseColumn(buf[offset:offset + c.size]))
    return SecureColumnByCoords(cols)


def _weights(log_n, point, offset=0):
    from proving_gb300 import _lib
    from proving_gb300.backend import _ptr_table, _stream, _u32_table
    out = _secure([np.zeros(1 << log_n, np.uint32) for _ in range(4)], offset)
    _lib.call("cs_barycentric_weights", log_n, _u32_table(point[0]), _u32_table(point[1]),
              _ptr_table([c.data for c in out.columns]), _stream())
    return out.to_cpu()


def _same(got, want):
    return all(np.array_equal(g, w) for g, w in zip(got, want))


def _point(seed):
    return pr.random_point(tuple(int(v) for v in seeded_qm31(seed)))


@pytest.mark.parametrize("log_n", [1, 2, 3, 4, 5, 9, 13])
@pytest.mark.parametrize("offset", [0, 1])
def test_weights(log_n, offset):
    point = _point(50 + log_n)
    assert _same(_weights(log_n, point, offset), O.barycentric_weights(log_n, *point))


@pytest.mark.parametrize("log_n", [3, 6])
@pytest.mark.parametrize("j", [0, 1, 5])
@pytest.mark.parametrize("turn", [0, 1, 2, 3])
def test_weights_at_domain_points(log_n, j, turn):
    # a domain point, its conjugate, its antipode and the antipode's conjugate
    x, y = pr.canonic_domain_point(log_n, j)
    x, y = [(x, y), (x, (pr.P - y) % pr.P), (pr.P - x, pr.P - y), (pr.P - x, y)][turn]
    point = (pr.qm(x), pr.qm(y))
    assert _same(_weights(log_n, point), O.barycentric_weights(log_n, *point))


@pytest.mark.parametrize("log_n", [3, 8])
def test_weights_off_the_circle(log_n):
    point = (tuple(int(v) for v in seeded_qm31(3)), tuple(int(v) for v in seeded_qm31(4)))
    assert _same(_weights(log_n, point), O.barycentric_weights(log_n, *point))


@pytest.mark.parametrize("sub_log,blowup,acc_logs", [(1, 1, [1]), (2, 1, [2, 1]), (3, 1, [3]), (3, 2, [1, 2, 3]),
                                                     (5, 1, [5, 4, 3, 2, 1]), (10, 1, [10, 7]), (13, 3, [13, 12, 1])])
@pytest.mark.parametrize("offset", [0, 1])
def test_quotients(sub_log, blowup, acc_logs, offset):
    from proving_gb300.backend import CudaBackend as B
    accs = [qm31_column(60 + k, n) for k, n in enumerate(acc_logs)]
    points = [_point(70 + k) for k in range(len(acc_logs))]
    linear = [tuple(int(v) for v in seeded_qm31(80 + k)) for k in range(len(acc_logs))]
    got = B.quotients_on_subdomain([_secure(a, offset) for a in accs], points, linear, sub_log + blowup, blowup)
    assert _same(got.to_cpu(), O.quotients_on_subdomain(accs, points, linear, sub_log + blowup, blowup))
