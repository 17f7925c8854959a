"""Partial numerators of columns that are only word-aligned: batches of up to 512 terms are one launch, each of
which reads and writes the accumulators once, and batches around 256 and 512 terms equal the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from proving_gb300 import _lib
from proving_gb300.synthetic import m31_columns, seeded_qm31

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_terms,launches", [(24, 1), (256, 1), (257, 1), (512, 1), (513, 2), (600, 2)])
@pytest.mark.parametrize("log_n", [7, 12])
def test_unaligned(n_terms, launches, log_n):
    from proving_gb300.backend import BaseColumn, CudaBackend as B
    vals = m31_columns(n_terms, n_terms, log_n)
    buf = torch.zeros((n_terms, (1 << log_n) + 4), dtype=torch.int32, device="cuda")
    buf[:, 1:1 + (1 << log_n)] = torch.from_numpy(np.ascontiguousarray(vals).view(np.int32)).cuda()
    cols = [BaseColumn(buf[i, 1:1 + (1 << log_n)]) for i in range(n_terms)]
    coeffs = np.stack([np.stack([seeded_qm31(3 * t + k) for k in range(3)]) for t in range(n_terms)])
    before = _lib.load().cs_kernel_launch_count()
    got, first = B.accumulate_numerators(cols, coeffs, 0)
    assert _lib.load().cs_kernel_launch_count() - before == launches
    want, want_first = O.accumulate_numerators(list(vals), 0, coeffs)
    assert list(first) == list(want_first)
    for g, w in zip(got.to_cpu(), want):
        assert np.array_equal(g, w)
