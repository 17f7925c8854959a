"""Words of P in a column count as zeros: its coefficients are canonic words, the same as those of the column
with zeros in their place, at the sizes of every kind of pass (small kernels, one contiguous pass of each
length, the tile kernel, two and three passes)."""
import numpy as np
import pytest
import torch

from proving_gb300.synthetic import m31_columns

P = (1 << 31) - 1
pytestmark = pytest.mark.gpu


def _coefficients(vals, log_n):
    from proving_gb300.backend import BaseColumn, CudaBackend as B, canonic_half_coset
    cols = [BaseColumn.from_cpu(v) for v in vals]
    B.interpolate_columns(cols, B.precompute_twiddles(canonic_half_coset(log_n + 1)))
    torch.cuda.synchronize()
    return [c.to_cpu() for c in cols]


@pytest.mark.parametrize("log_n", [1, 2, 3, 5, 6, 7, 8, 9, 10, 11, 12, 13, 17, 20, 23])
def test_interpolate(log_n):
    zeros = m31_columns(log_n, 3, log_n)
    zeros[0][:] = 0
    zeros[1][::2] = 0
    zeros[2][-1] = 0
    words = np.where(zeros == 0, np.uint32(P), zeros)
    for got, want in zip(_coefficients(words, log_n), _coefficients(zeros, log_n)):
        assert np.array_equal(got, want)
