"""FP64 pruning and gradient kernels over tree shapes and pattern counts at their tiles' edges, against the oracle.

Shapes: two-leaf nodes, leaves beside internal siblings, polytomies with leaves and internal children, a star;
codons with gaps and IUPAC ambiguity.  Pattern counts around the 32-pattern tile.  (CTAs that take several
tiles run in the full-size parity tests.)"""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle

pytestmark = pytest.mark.gpu

SHAPES = {
    "star": "(a:0.1,b:0.2,c:0.3,d:0.05,e:0.4,f:0.15);",
    "caterpillar": "((((((a:0.1,b:0.2):0.1,c:0.3):0.2,d:0.05):0.1,e:0.4):0.3,f:0.1):0.2,g:0.3,h:0.2);",
    "cherries": "((a:0.1,b:0.2):0.1,(c:0.3,d:0.05):0.1,(e:0.4,f:0.1):0.3);",
    "polytomies": "((a:0.1,b:0.2,(c:0.1,d:0.3):0.2,(e:0.2,f:0.1,g:0.3):0.1):0.2,(h:0.1,i:0.2):0.3,j:0.4,k:0.1);",
}


def _alignment(oracle, tree, sites, rng):
    from hyphy3.simulate import universal_code
    codons, _ = universal_code()
    text = ["".join("ACGT"[x] for x in c) for c in codons] + ["---", "AAR", "CTN", "NNN", "GAY", "ATH"]
    p = np.concatenate([np.full(61, 0.9 / 61), np.full(6, 0.1 / 6)])
    names = [tree.names[i] for i in range(tree.num_nodes()) if tree.is_leaf[i]]
    return oracle.Alignment.from_sequences(names, ["".join(text[k] for k in rng.choice(len(text), size=sites, p=p)) for _ in names])


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("sites", [1, 31, 33, 129])
def test_shapes_and_tile_edges(oracle, shape, sites):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(SHAPES[shape])
    _check(oracle, _capi, tree, _alignment(oracle, tree, sites, np.random.default_rng(sites)))


def _check(oracle, _capi, tree, aln):
    par = {"alpha": 1.0, "beta": 0.4, "theta": [0.7, 1.3, 0.9, 1.6, 0.8]}
    e = oracle.mg94(aln, par)
    bl = list(tree.branch_lengths)
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    lnl, grad = pr.branch_length_gradients(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], bl=np.array(bl))
    ref, gref = oracle.branch_length_gradients(tree, aln, par, bl)
    gref = np.array(gref)
    # the FP64 path's parity bound: 1e-10 relative
    assert abs(lnl - ref) <= 1e-10 * abs(ref)
    assert np.max(np.abs(grad - gref)) <= 1e-10 * max(1.0, np.max(np.abs(gref)))
    pr.close()
    ctx.close()
