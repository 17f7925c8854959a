"""A GKR batch of more instances than a launch grid has rows (65,535), deep enough for a round of its own launch: every
instance is the same grand product, so each has the output claim of the instance proved alone, and the same
masks as the others."""
import pytest
import torch

from proving_gb300 import gkr as G
from proving_gb300 import prover as pr

pytestmark = pytest.mark.gpu


def test_more_than_65535_instances():
    n_vars, n_inst = 9, 65_536
    gen = torch.Generator(device="cuda").manual_seed(5)
    col = torch.randint(0, pr.P, (4, 1 << n_vars), dtype=torch.int32, device="cuda", generator=gen)
    layer = G.Layer(G.GRAND_PRODUCT, [G.Mle(col, n_vars)])
    alone, _ = G.prove_batch_native(pr.Blake2sChannel(), [layer])
    proof, artifact = G.prove_batch_native(pr.Blake2sChannel(), [layer] * n_inst)
    assert len(proof.output_claims_by_instance) == n_inst
    assert all(c == alone.output_claims_by_instance[0] for c in proof.output_claims_by_instance)
    masks = [[m.columns for m in ms] for ms in proof.layer_masks_by_instance]
    assert len(masks[0]) == n_vars and all(m == masks[0] for m in masks)
    claims = artifact.claims_to_verify_by_instance
    assert all(c == claims[0] for c in claims)
    assert [len(polys) for polys in proof.sumcheck_proofs] == list(range(n_vars))
