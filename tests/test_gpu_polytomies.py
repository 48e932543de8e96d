"""FP64 gradients below nodes of many children, whose leaves have a kernel of their own above nine, against the oracle.

Child counts on both sides of that line, a leaf in the first, second and last place, internal children among the leaves, and
such a node below the root; pattern counts around the 32-pattern tile.  Branches of 0.4 and more: entries of P are
then 1e-5 and more, so their rounding is far below the bound."""
import numpy as np
import pytest

from test_gpu_fp64_shapes import _alignment, _check

pytestmark = pytest.mark.gpu


def _leaves(k, tag="t"):
    return [f"{tag}{i}:{0.4 + 0.03 * (i % 7)}" for i in range(k)]


TREES = {f"star_{k}": "(" + ",".join(_leaves(k)) + ");" for k in (8, 9, 10, 11, 40)}
TREES["internal_first"] = "((a:0.5,b:0.6):0.4," + ",".join(_leaves(10)) + ");"
TREES["internal_second_and_last"] = "(" + ",".join([_leaves(1)[0], "(a:0.5,b:0.6):0.4", *_leaves(9)[1:], "(c:0.5,d:0.4,e:0.7):0.5"]) + ");"
TREES["below_the_root"] = "((" + ",".join(_leaves(12)) + "):0.4,(" + ",".join(_leaves(9, "u")) + "):0.5,v:0.6);"


@pytest.mark.parametrize("shape", sorted(TREES))
@pytest.mark.parametrize("sites", [1, 33, 129])
def test_leaves_of_large_nodes(oracle, shape, sites):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(TREES[shape])
    _check(oracle, _capi, tree, _alignment(oracle, tree, sites, np.random.default_rng(sites)))
