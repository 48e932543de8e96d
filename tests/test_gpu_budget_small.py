"""Memory budgets of small problems: one that holds the smallest plan with 256-pattern accumulation chunks is enough."""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle
from test_gpu_fp64_shapes import SHAPES, _alignment

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sites", [300, 900])
@pytest.mark.parametrize("precision_name", ["fp64", "mixed"])
def test_the_smallest_budget_that_holds_large_chunks(oracle, sites, precision_name):
    from hyphy3 import _capi
    prec = _capi.PREC_FP64 if precision_name == "fp64" else _capi.PREC_MIXED
    tree = oracle.Tree.parse(SHAPES["caterpillar"])
    aln = _alignment(oracle, tree, sites, np.random.default_rng(sites))
    e = oracle.mg94(aln, {"alpha": 1.0, "beta": 0.4, "theta": [0.7, 1.3, 0.9, 1.6, 0.8]})
    kw = dict(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], precision=prec)
    bl = np.array(tree.branch_lengths)
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    pr.set_tuning(a_chunk=384)                                    # 3 or 9 tiles of 128 patterns in chunks of 256 and more
    pr.set_model(**kw)
    pr.set_memory_budget(0, 2)
    need = pr.checkpoint_info()["workspace_bytes"]
    pr.close()
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    pr.set_model(**kw)
    ref = pr.eval(bl)
    ref = {"lnl": ref["lnl"], "grad_t": ref["grad_t"].copy()}
    pr.set_memory_budget(need)
    info = pr.checkpoint_info()
    assert info["workspace_bytes"] <= need
    assert info["active"] or precision_name == "mixed"            # (its full workspace may be as small)
    got = pr.eval(bl)
    # the likelihood's order of summation is the same; the gradient's sums of at most 1000 terms are regrouped
    assert got["lnl"] == ref["lnl"]
    tol = 1e-11 if precision_name == "fp64" else 1e-5
    assert np.max(np.abs(got["grad_t"] - ref["grad_t"])) <= tol * np.max(np.abs(ref["grad_t"]))
    with pytest.raises(_capi.H3GError):
        pr.set_memory_budget(need // 2)
    pr.close()
    ctx.close()
