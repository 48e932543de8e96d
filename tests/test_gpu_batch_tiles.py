"""A batch's slots give a CTA more pattern tiles than a problem evaluated alone: the same bits."""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle
from test_gpu_fp64_shapes import _alignment

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sites", [95, 700, 1500])
@pytest.mark.parametrize("slots", [2, 8])
def test_batch_matches_single_evaluations(oracle, sites, slots):
    from hyphy3 import _capi
    rng = np.random.default_rng(sites)
    newick = "(" + ",".join(f"(a{i}:0.1,b{i}:0.2):0.1" for i in range(32)) + ");"
    tree = oracle.Tree.parse(newick)
    aln = _alignment(oracle, tree, sites, rng)
    e = oracle.mg94(aln, {"alpha": 1.0, "beta": 0.4, "theta": [0.7, 1.3, 0.9, 1.6, 0.8]})
    bl = np.array(tree.branch_lengths)
    ctx = _capi.Context(0)
    probs = [problem_from_oracle(ctx, oracle, tree, aln) for _ in range(8)]
    alone = []
    for k, pr in enumerate(probs):
        pr.set_model(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"])
        r = pr.eval(bl * (1 + 0.1 * k))
        alone.append((r["lnl"], r["grad_t"].copy()))
    batch = _capi.Batch(ctx, probs, n_slots=slots)
    for pr in probs:
        pr.set_model(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"])
    for (lnl, grad), r in zip(alone, batch.eval([bl * (1 + 0.1 * k) for k in range(8)])):
        assert r["lnl"] == lnl
        assert np.array_equal(r["grad_t"], grad)
    batch.close()
    for pr in probs:
        pr.close()
    ctx.close()
