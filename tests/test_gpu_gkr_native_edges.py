"""The device-resident GKR prover at the edges of its launches: layers around the single-block tail's
longest (9 rounds), more instances than keep their tail columns (4) or their state (64) in shared
memory, instances that join late, and every input kind at its smallest. Proof, artifact and channel
equal the driver's over the separate operations."""
import pytest
import torch

from proving_gb300 import _lib
from proving_gb300 import gkr as G
from proving_gb300 import prover as pr

pytestmark = pytest.mark.gpu

GP, GEN, MUL, ONE = G.GRAND_PRODUCT, G.LOGUP_GENERIC, G.LOGUP_MULTIPLICITIES, G.LOGUP_SINGLES


def _layers(spec):
    gen = torch.Generator(device="cuda").manual_seed(sum(7 * k + n for k, n in spec))
    rnd = lambda rows, n: torch.randint(0, pr.P, (rows, 1 << n), dtype=torch.int32, device="cuda", generator=gen)
    out = []
    for kind, n in spec:
        mles = [G.Mle(rnd(4, n), n)]
        if kind == GEN:
            mles.insert(0, G.Mle(rnd(4, n), n))
        if kind == MUL:
            mles.insert(0, G.Mle(rnd(1, n), n, base=True))
        out.append(G.Layer(kind, mles))
    return out


@pytest.mark.parametrize("spec", [
    [(GEN, 1)], [(ONE, 1)], [(ONE, 2)], [(MUL, 2)],
    [(GEN, 9)], [(GEN, 10)], [(MUL, 10)], [(ONE, 11)], [(GP, 11), (GEN, 12)], [(MUL, 12), (GP, 10)],
    [(GEN, 3), (GP, 11), (MUL, 2), (ONE, 11)],
    [(GEN, 11), (GP, 10), (ONE, 9), (MUL, 11), (GP, 2)],        # five: tail columns in global memory
    [(GP, 1 + i % 5) for i in range(65)] + [(GEN, 10)],         # sixty-six: state in global memory too
    [(MUL, 17), (GP, 15)], [(ONE, 16), (GEN, 16)],
])
def test_equals_driver(spec):
    dev, layers = G.DeviceGkrOps(), _layers(spec)
    inputs = [[m.data.clone() for m in lay.mles] for lay in layers]
    ch_a, ch_b = pr.Blake2sChannel(), pr.Blake2sChannel()
    a, art_a = G.prove_batch(dev, ch_a, layers)
    b, art_b = G.prove_batch_native(ch_b, layers)
    assert b.sumcheck_proofs == a.sumcheck_proofs
    assert [[m.columns for m in ms] for ms in b.layer_masks_by_instance] == \
        [[m.columns for m in ms] for ms in a.layer_masks_by_instance]
    assert b.output_claims_by_instance == a.output_claims_by_instance
    assert art_b.ood_point == art_a.ood_point
    assert art_b.claims_to_verify_by_instance == art_a.claims_to_verify_by_instance
    assert (ch_b.digest, ch_b.n_draws) == (ch_a.digest, ch_a.n_draws)
    for lay, kept in zip(layers, inputs):  # the inputs are the caller's
        for m, k in zip(lay.mles, kept):
            assert torch.equal(m.data, k)


def test_unfixed_multiplicities_are_refused():
    with pytest.raises(_lib.CudaBackendError, match="mask of a multiplicities layer"):
        G.prove_batch_native(pr.Blake2sChannel(), _layers([(MUL, 1)]))
