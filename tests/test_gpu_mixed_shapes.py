"""Mixed-precision gradients over tree shapes and pattern counts at the accumulation's edges, against the oracle.

A leaf with one sibling has its gradient formed from the parent's outside vector and the sibling's message (a leaf's,
also with gaps and ambiguity, an internal node's, below the root or not); leaves of polytomies and internal branches
read stored vectors.  Pattern counts around the 64-pattern tile, of which two groups of warps take every other one."""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle
from test_gpu_fp64_shapes import SHAPES, _alignment

pytestmark = pytest.mark.gpu

TWO_AT_ROOT = "(((a:0.1,b:0.2):0.1,(c:0.3,d:0.05):0.2):0.1,e:0.4);"     # the root's two children: a leaf and a subtree


@pytest.mark.parametrize("shape", sorted(SHAPES) + ["two_at_root"])
@pytest.mark.parametrize("sites", [1, 65, 200, 700])
def test_shapes_and_tile_edges(oracle, shape, sites):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(SHAPES.get(shape, TWO_AT_ROOT))
    aln = _alignment(oracle, tree, sites, np.random.default_rng(sites))
    par = {"alpha": 1.0, "beta": 0.4, "theta": [0.7, 1.3, 0.9, 1.6, 0.8]}
    e = oracle.mg94(aln, par)
    bl = list(tree.branch_lengths)
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    lnl, grad = pr.branch_length_gradients(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], bl=np.array(bl),
                                           precision=_capi.PREC_MIXED)
    ref, gref = oracle.branch_length_gradients(tree, aln, par, bl)
    gref = np.array(gref)
    # the mixed path's parity bound: 1e-7 relative in lnL, 1e-5 in the gradient's norm
    assert abs(lnl - ref) <= 1e-7 * abs(ref)
    assert np.linalg.norm(grad - gref) <= 1e-5 * np.linalg.norm(gref)
    pr.close()
    ctx.close()
