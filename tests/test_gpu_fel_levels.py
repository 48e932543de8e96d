"""FEL's per-site likelihoods over level widths and child counts, against the main engine.

At a fitted (alpha, beta) the reported log-likelihood is the pattern's under alpha Qs + beta Qn with the run's branch
lengths.  Levels narrower and wider than a CTA's warps, odd counts, polytomies, a star, a chain."""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle
from test_gpu_fel import _fel_inputs
from test_gpu_fp64_shapes import _alignment

pytestmark = pytest.mark.gpu


def _tree(shape):
    leaf = iter(f"t{i}:0.{1 + i % 7}" for i in range(200))
    take = lambda k: ",".join(next(leaf) for _ in range(k))
    if shape == "star_40":
        return f"({take(40)});"
    if shape == "cherries_17":
        return "(" + ",".join(f"({take(2)}):0.1" for _ in range(17)) + ");"
    if shape == "mixed_9":
        return "(" + ",".join(f"({take(3)}):0.2" for _ in range(9)) + f",{take(1)});"
    text = f"({take(2)}):0.1"
    for _ in range(20):
        text = f"({text},{take(1)}):0.05"
    return f"({text},{take(2)});"


@pytest.mark.parametrize("shape", ["star_40", "cherries_17", "mixed_9", "chain"])
def test_reported_likelihood_is_the_engines(oracle, shape):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(_tree(shape))
    aln = _alignment(oracle, tree, 4, np.random.default_rng(len(shape)))
    pi, qs, qn = _fel_inputs(oracle, aln, {"theta": [0.7, 1.3, 0.9, 1.6, 0.8]})
    bl = np.array(tree.branch_lengths)
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    fit = pr.fel_run(pi=pi, Qs=qs, Qn=qn, branch_lengths=bl)
    for p in range(pr.P):
        Q = fit["alpha"][p] * qs + fit["beta"][p] * qn
        np.fill_diagonal(Q, -Q.sum(1))
        pr.set_model(pi=pi, Q=Q)
        site = pr.eval(bl, _capi.WANT_LNL | _capi.WANT_SITE_LNL)["site_lnl"][p]
        # two FP64 evaluations with eigensystems of their own: 1e-9 relative
        assert abs(fit["log_l_alt"][p] - site) <= 1e-9 * max(1.0, abs(site))
    pr.close()
    ctx.close()
