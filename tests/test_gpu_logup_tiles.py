"""LogUp running sums at the sizes where their launches change: one block per column (2^0 to 2^9 rows),
one tile that is its own mirror (2^10), one pair of tiles (2^11), run offsets over less than one step and
over several (2^15, 2^18 rows), batches of both kinds of column, and values that z meets (their fraction
counts as 0, alone and beside others of the same inversion)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from proving_gb300.synthetic import m31_column, seeded_qm31  # noqa: E402

P = 2**31 - 1


@pytest.fixture(scope="module")
def B():
    from proving_gb300 import build
    build.build()
    from proving_gb300.backend import CudaBackend
    return CudaBackend


@pytest.mark.parametrize("logs", [[9, 10], [10, 9, 1], [11], [3, 4, 9], [12, 2, 15, 10, 18]])
@pytest.mark.parametrize("base_z", [False, True])
def test_running_sums(B, logs, base_z):
    from proving_gb300.backend import BaseColumn
    z = np.array([77, 0, 0, 0], np.uint32) if base_z else seeded_qm31(sum(logs))
    vals = [m31_column(300 + k, l) for k, l in enumerate(logs)]
    if base_z:
        for v in vals:
            v[0] = v[-1] = v[v.size // 2] = 77
            v[v.size // 3] = 76  # a norm of 1
    else:
        for v in vals:
            v[0], v[-1] = 0, P - 1
    outs, claimed = B.logup_running_sums([BaseColumn.from_cpu(v) for v in vals], z)
    claimed = claimed.cpu().numpy().view(np.uint32)
    for k, (v, out) in enumerate(zip(vals, outs)):
        want, want_claimed = O.logup_running_sum(v, z)
        assert list(claimed[k]) == list(want_claimed)
        assert all(np.array_equal(g, w) for g, w in zip(out.to_cpu(), want))


@pytest.mark.parametrize("log_n", [9, 10, 11, 15])
def test_all_values_equal_z(B, log_n):
    from proving_gb300.backend import BaseColumn
    v = np.full(1 << log_n, 5, np.uint32)
    z = np.array([5, 0, 0, 0], np.uint32)
    got, claimed = B.logup_running_sum(BaseColumn.from_cpu(v), z)
    want, want_claimed = O.logup_running_sum(v, z)
    assert list(claimed) == list(want_claimed)
    assert all(np.array_equal(g, w) for g, w in zip(got.to_cpu(), want))
