"""FEL's per-site likelihoods on both sides of the number of requests up to which a request has an SM to itself.

A run's first batch is 12 requests a pattern.  At a fitted (alpha, beta) the reported log-likelihood is the pattern's under
alpha Qs + beta Qn in the main engine."""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle
from test_gpu_fel import _fel_inputs
from test_gpu_fel_levels import _tree
from test_gpu_fp64_shapes import _alignment

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["star_40", "cherries_17", "chain"])
@pytest.mark.parametrize("sites", [12, 13, 40])
def test_reported_likelihood_is_the_engines(oracle, shape, sites):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(_tree(shape))
    aln = _alignment(oracle, tree, sites, np.random.default_rng(sites + len(shape)))
    pi, qs, qn = _fel_inputs(oracle, aln, {"theta": [0.7, 1.3, 0.9, 1.6, 0.8]})
    bl = np.array(tree.branch_lengths)
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    fit = pr.fel_run(pi=pi, Qs=qs, Qn=qn, branch_lengths=bl)
    for p in range(0, pr.P, max(1, pr.P // 12)):
        Q = fit["alpha"][p] * qs + fit["beta"][p] * qn
        np.fill_diagonal(Q, -Q.sum(1))
        pr.set_model(pi=pi, Q=Q)
        site = pr.eval(bl, _capi.WANT_LNL | _capi.WANT_SITE_LNL)["site_lnl"][p]
        # two FP64 evaluations with eigensystems of their own: 1e-9 relative
        assert abs(fit["log_l_alt"][p] - site) <= 1e-9 * max(1.0, abs(site))
    pr.close()
    ctx.close()
