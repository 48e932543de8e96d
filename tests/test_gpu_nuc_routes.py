"""Nucleotide likelihoods from transition matrices around the line between one walk of the tree and a launch per level.

Patterns are independent, so a problem's likelihoods are those of the same patterns in small problems, which walk.  Tree
shapes whose lines lie apart: a star, a chain, a random tree; polytomies; missing and ambiguous states."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _parents(shape, rng):
    if shape == "star":
        return [-1] + [0] * 60
    par = [-1]
    if shape == "chain":
        for k in range(0, 80, 2):
            par += [k, k]
        return par
    leaves = [0]
    while len(leaves) < 90:
        u = leaves.pop(int(rng.integers(len(leaves))))
        for _ in range(3 if shape == "polytomies" and rng.random() < 0.4 else 2):
            leaves.append(len(par))
            par.append(u)
    return par


def _eval(ctx, parent, leaf, taxon, states, masks, weights, P, pi):
    from hyphy3 import _capi
    dp = C.POINTER(C.c_double)
    pr = _capi.Problem(ctx, parent, leaf, taxon, states, masks, weights)
    lnl, site = C.c_double(), np.zeros(len(states))
    ctx.check(ctx.lib.h3g_nuc_eval_from_P(pr.h, P.ctypes.data_as(dp), pi.ctypes.data_as(dp), C.byref(lnl), site.ctypes.data_as(dp)))
    pr.close()
    return lnl.value, site


@pytest.mark.parametrize("shape", ["star", "chain", "random", "polytomies"])
@pytest.mark.parametrize("P", [1, 4736, 4737, 16001, 40000])
def test_routes_agree(shape, P):
    from hyphy3 import _capi
    rng = np.random.default_rng(P)
    parent = np.array(_parents(shape, rng), np.int32)
    n = parent.size
    leaf = np.array([u not in parent for u in range(n)], np.uint8)
    taxon = np.full(n, -1, np.int32)
    T = int(leaf.sum())
    taxon[leaf == 1] = np.arange(T)
    taxon[np.flatnonzero(leaf)[1]] = -1                            # a leaf without data
    states = rng.integers(0, 4, (P, T)).astype(np.int8)
    masks = np.uint64(1) << states.astype(np.uint64)
    lost = rng.random((P, T)) < 0.05
    states[lost] = -1
    masks[lost] = rng.integers(0, 16, int(lost.sum())).astype(np.uint64)
    mat = rng.uniform(0.01, 1.0, (n, 4, 4)) + 3.0 * np.eye(4)
    mat /= mat.sum(2, keepdims=True)
    pi = np.array([0.3, 0.2, 0.1, 0.4])
    weights = rng.integers(1, 4, P).astype(np.float64)
    ctx = _capi.Context(0)
    lnl, site = _eval(ctx, parent, leaf, taxon, states, masks, weights, mat, pi)
    parts = [_eval(ctx, parent, leaf, taxon, states[a:a + 1000], masks[a:a + 1000], weights[a:a + 1000], mat, pi) for a in range(0, P, 1000)]
    assert np.array_equal(site, np.concatenate([s for _, s in parts]))
    total = sum(l for l, _ in parts)
    assert abs(lnl - total) <= 1e-14 * abs(total)                  # compensated sums of one sign, 40 parts
    ctx.close()
