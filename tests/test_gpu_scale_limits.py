"""Likelihoods from given transition matrices whose entries are near the ends of the double range.

The reference prunes in 80-bit floats, whose exponents hold every product here.  Off the diagonal the entries are
about `mag`: a product of two, 1e-300, is still a double, so a pass that scales after each child's message loses
nothing.  "rare": a state that is hardly ever reached, and in which every leaf is; each message is its tiny column."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TREES = {      # parent of each node
    "star": [-1, 0, 0, 0, 0],
    "cherries": [-1, 0, 0, 1, 1, 2, 2],
    "caterpillar": [-1, 0, 0, 2, 2, 4, 4, 6, 6],
    "one_child": [-1, 0, 1, 2, 2, 0],
}


def _site_lnl(parent, states, P, pi):
    n, S = len(parent), pi.size
    kids = [[c for c in range(n) if parent[c] == u] for u in range(n)]
    leaves = [u for u in range(n) if not kids[u]]
    P = P.astype(np.longdouble)

    def below(u, p):
        v = np.ones(S, np.longdouble)
        if not kids[u]:
            return (np.arange(S) == states[p, leaves.index(u)]).astype(np.longdouble)
        for c in kids[u]:
            v = v * (P[c] @ below(c, p))
        return v

    return np.array([float(np.log(pi.astype(np.longdouble) @ below(0, p))) for p in range(len(states))])


@pytest.mark.parametrize("tree", sorted(TREES))
@pytest.mark.parametrize("S", [2, 4, 5, 61])
@pytest.mark.parametrize("mag,rare", [(1e-20, False), (1e-120, False), (1e-150, False), (1e-150, True), (1e-250, True)])
def test_transition_probabilities_near_the_range_ends(tree, S, mag, rare):
    from hyphy3 import _capi
    rng = np.random.default_rng(S)
    parent = np.array(TREES[tree], dtype=np.int32)
    n = parent.size
    leaf = np.array([u not in TREES[tree] for u in range(n)], dtype=np.uint8)
    taxon = np.full(n, -1, dtype=np.int32)
    taxon[leaf == 1] = np.arange(leaf.sum())
    states = rng.integers(0, S, (7, int(leaf.sum()))).astype(np.int8)
    if rare:
        states[:] = S - 1
    P = mag * rng.uniform(0.5, 1.5, (n, S, S))
    if rare:                                                     # every other state is as likely as the next
        P[:, :, :-1] = rng.uniform(0.5, 1.5, (n, S, S - 1)) / S
    else:
        P[:, np.arange(S), np.arange(S)] = 1.0
    pi = np.full(S, 1.0 / S)
    ctx = _capi.Context(0)
    pr = _capi.Problem(ctx, parent, leaf, taxon, states, np.uint64(1) << states.astype(np.uint64), np.ones(len(states)))
    lnl, site = pr.eval_from_P(P, pi)
    ref = _site_lnl(TREES[tree], states, P, pi)
    # at most 9 nodes with sums of 64 rounded products each: 1e-13 of the likelihood, so below 1e-12 of its logarithm
    assert np.max(np.abs(site - ref) / np.maximum(1.0, np.abs(ref))) <= 1e-12
    pr.close()
    ctx.close()
