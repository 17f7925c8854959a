"""LogUp running sums at the run counts where the offsets' steps change: segments of 1, 32, 64 (32 runs a step), 128
and 256 runs (128 a step), alone and beside each other. Words equal the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from proving_gb300.synthetic import m31_column, seeded_qm31

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logs", [[10], [15], [16], [17], [18], [14, 17, 16, 11]])
def test_running_sums(logs):
    from proving_gb300.backend import BaseColumn, CudaBackend as B
    z = seeded_qm31(sum(logs))
    vals = [m31_column(300 + k, l) for k, l in enumerate(logs)]
    outs, claimed = B.logup_running_sums([BaseColumn.from_cpu(v) for v in vals], z)
    claimed = claimed.cpu().numpy().view(np.uint32)
    for k, (v, out) in enumerate(zip(vals, outs)):
        want, want_claimed = O.logup_running_sum(v, z)
        assert list(claimed[k]) == list(want_claimed)
        assert all(np.array_equal(g, w) for g, w in zip(out.to_cpu(), want))
