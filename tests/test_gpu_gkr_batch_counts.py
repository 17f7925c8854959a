"""GKR batches by instance count around the launches' shared memory: four instances (the last count whose
tail columns are kept there) with layers long enough for launches of their own, six, 57 to 64 (every
instance's state in shared memory, up to more than four instances' tail columns take) and 65 (none). And one
instance of every kind with 7 and 8 variables, the layers around the longest that the single-block kernel runs
alone. Proofs equal the driver's over the separate operations."""
import pytest

import test_gpu_gkr_native_edges as edges
from test_gpu_gkr_native_edges import GEN, GP, MUL, ONE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 6, 57, 58, 64, 65])
@pytest.mark.parametrize("longest", [3, 10])
def test_batches(n, longest):
    kinds = [GP, GP, ONE, GEN, GP, MUL]
    edges.test_equals_driver([(GEN, longest)] + [(kinds[i % 6], 2 + i % 2) for i in range(n - 1)])


@pytest.mark.parametrize("kind", [GP, GEN, MUL, ONE])
@pytest.mark.parametrize("n_vars", [7, 8, 9])
def test_single_instances(kind, n_vars):
    edges.test_equals_driver([(kind, n_vars)])
