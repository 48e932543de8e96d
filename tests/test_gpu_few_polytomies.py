"""Nodes of many children, leaves and internal nodes in any order, in the walks for models of at most four states: their
messages are loaded ahead, so every position of a child and every length of the list counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tree(kinds):
    """A root whose children are leaves (0), nodes of two leaves (2) or of three (3)."""
    parent = [-1]
    for k in kinds:
        parent.append(0)
        parent += [len(parent) - 1] * k
    return parent


@pytest.mark.parametrize("kinds", [[0, 0, 2], [2, 0, 0], [0, 2, 0, 0], [2, 2, 2, 2], [0, 0, 3, 0, 2], [3, 0, 0, 0, 0, 0], [0] * 9 + [2],
                                   [0] * 33])
@pytest.mark.parametrize("S,P", [(4, 1), (4, 33), (3, 130)])
def test_values_against_extended_precision(kinds, S, P):
    from hyphy3 import _capi
    rng = np.random.default_rng(len(kinds) + 100 * P)
    parent = np.array(_tree(kinds), dtype=np.int32)
    n = parent.size
    kids = [np.flatnonzero(parent == u) for u in range(n)]
    leaf = np.array([k.size == 0 for k in kids], dtype=np.uint8)
    T = int(leaf.sum())
    taxon = np.full(n, -1, dtype=np.int32)
    taxon[leaf == 1] = np.arange(T)
    masks = rng.integers(1, 2 ** S, (P, T)).astype(np.uint64)            # ambiguous, where more than one bit is set
    one = rng.random((P, T)) < 0.7
    states = np.where(one, rng.integers(0, S, (P, T)), -1).astype(np.int8)
    masks[one] = np.uint64(1) << states[one].astype(np.uint64)
    mats = rng.uniform(0.05, 1.0, (n, S, S))
    mats /= mats.sum(2, keepdims=True)
    pi = rng.dirichlet(np.ones(S))

    def below(u):
        if leaf[u]:
            return ((masks[:, taxon[u], None] >> np.arange(S, dtype=np.uint64)) & np.uint64(1)).astype(np.longdouble)
        v = np.ones((P, S), np.longdouble)
        for c in kids[u]:
            v = v * (below(c) @ mats[c].astype(np.longdouble).T)
        return v

    ctx = _capi.Context(0)
    pr = _capi.Problem(ctx, parent, leaf, taxon, states, masks, np.ones(P))
    _, site = pr.eval_from_P(mats, pi)
    pr.close()
    ctx.close()
    ref = np.log((below(0) @ pi.astype(np.longdouble)).astype(np.longdouble)).astype(float)
    # at most 44 messages of 4 rounded terms each: 44 x 8 x 2^-53 = 4e-14 of the likelihood
    assert np.max(np.abs(site - ref) / np.maximum(1.0, np.abs(ref))) <= 1e-13
