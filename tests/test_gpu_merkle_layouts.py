"""Merkle trees at the edges of their launches: how the leaf kernel reads its columns (equally spaced
in either direction, a pointer each, lifted) around a block of 16, leaf counts on both sides of the
low-latency compression's limit, and heights around the subtree launches' splits. Roots and layers
equal the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from proving_gb300.synthetic import m31_columns

pytestmark = pytest.mark.gpu


def _columns(vals, layout):
    from proving_gb300.backend import BaseColumn
    n_cols, n = vals.shape
    dev = torch.from_numpy(np.ascontiguousarray(vals).view(np.int32)).cuda()
    if layout == "rows":
        return BaseColumn.rows_of(dev)
    if layout == "reversed":
        return BaseColumn.rows_of(dev.flip(0).contiguous())[::-1]
    # uneven gaps between the columns, all of them only word-aligned
    out = []
    for i in range(n_cols):
        buf = torch.empty(n + 64, dtype=torch.int32, device="cuda")
        buf[i % 7 + 1:i % 7 + 1 + n] = dev[i]
        out.append(BaseColumn(buf[i % 7 + 1:i % 7 + 1 + n]))
    return out


@pytest.mark.parametrize("layout", ["rows", "reversed", "apart"])
@pytest.mark.parametrize("n_cols,log_n", [(1, 5), (15, 7), (16, 6), (17, 9), (33, 10), (2, 15), (3, 16), (17, 16)])
def test_leaf_reads(layout, n_cols, log_n):
    from proving_gb300.backend import CudaBackend as B
    vals = m31_columns(31 * n_cols + log_n, n_cols, log_n)
    tree = B.merkle_commit(_columns(vals, layout), log_n)
    assert tree.root() == O.merkle_commit(list(vals), log_n)


@pytest.mark.parametrize("layout", ["rows", "apart"])
@pytest.mark.parametrize("logs,height", [([6] * 20 + [8] * 5, 9), ([15] * 18 + [16] * 17, 17), ([9] * 33, 12)])
def test_lifted_runs(layout, logs, height):
    from proving_gb300.backend import CudaBackend as B
    vals = [m31_columns(5 + i, 1, n)[0] for i, n in enumerate(logs)]
    cols = []
    for n in sorted(set(logs)):
        cols += _columns(np.stack([v for v, m in zip(vals, logs) if m == n]), layout)
    assert B.merkle_commit(cols, height).root() == O.merkle_commit(vals, height)


@pytest.mark.parametrize("height", [1, 2, 5, 8, 9, 10, 11, 16, 17, 18, 19, 20, 21, 22])
def test_every_layer(height):
    from proving_gb300.backend import CudaBackend as B
    vals = m31_columns(height, 2, height)
    tree = B.merkle_commit(_columns(vals, "rows"), height)
    layer = tree.layer(height)
    for k in range(height - 1, -1, -1):
        layer = B.build_next_layer(layer)
        assert torch.equal(tree.layer(k), layer)
    assert tree.root() == O.merkle_commit(list(vals), height)
