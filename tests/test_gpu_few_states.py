"""Models of at most four states: their walks of the tree against the 64-state passes.

The same model with a fifth state that nothing reaches (zero rates and frequency) runs through the 64-state passes and
has the same likelihood and gradients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TREES = {      # parent of each node, preorder
    "star": [-1, 0, 0, 0, 0, 0, 0, 0],
    "two_at_root": [-1, 0, 1, 1, 0],
    "caterpillar": [-1] + [x for k in range(0, 60, 2) for x in (k, k)],
    "cherries": [-1, 0, 1, 1, 0, 4, 4, 0, 7, 7],
    "polytomies": [-1, 0, 1, 1, 1, 4, 4, 4, 0, 8, 8, 8, 8, 0],
    "wide": [-1] + [0] * 40 + [x for k in range(1, 41) for x in (k, k, k)],
}


def _model(S, K, rng):
    pi = rng.uniform(0.5, 1.5, S)
    pi /= pi.sum()
    Q, lam, U, V, dQ = [], [], [], [], []
    for _ in range(K):
        r = rng.uniform(0.2, 2.0, (S, S))
        q = (r + r.T) * pi[None, :]
        np.fill_diagonal(q, 0.0)
        np.fill_diagonal(q, -q.sum(1))
        sq = np.sqrt(pi)
        sym = sq[:, None] * q / sq[None, :]
        w, e = np.linalg.eigh((sym + sym.T) / 2)
        Q.append(q), lam.append(np.minimum(w, 0.0)), U.append(e / sq[:, None]), V.append(e.T * sq[None, :])
        d = rng.uniform(-1, 1, (2, S, S))
        dQ.append(d - np.einsum("dij,jk->dik", d.sum(2, keepdims=True) * np.ones((1, 1, S)), np.eye(S)) / S)
    return pi, np.array(Q), np.array(lam), np.array(U), np.array(V), np.array(dQ).transpose(1, 0, 2, 3)


def _pad(a, axes):
    width = [(0, 1) if i in axes else (0, 0) for i in range(a.ndim)]
    return np.pad(a, width)


@pytest.mark.parametrize("tree", sorted(TREES))
@pytest.mark.parametrize("S,K,M,P", [(4, 1, 1, 1), (4, 1, 1, 129), (4, 2, 3, 33), (3, 1, 2, 64), (2, 2, 1, 31), (1, 1, 1, 5), (4, 1, 1, 2995)])
def test_against_the_padded_model(tree, S, K, M, P):
    from hyphy3 import _capi
    rng = np.random.default_rng(1000 * S + 100 * K + 10 * M + P)
    parent = np.array(TREES[tree], dtype=np.int32)
    n = parent.size
    leaf = np.array([i not in TREES[tree] for i in range(n)], dtype=np.uint8)
    taxon = np.full(n, -1, dtype=np.int32)
    taxon[leaf == 1] = np.arange(leaf.sum())
    if leaf.sum() > 4:
        taxon[np.flatnonzero(leaf)[1]] = -1                       # a leaf without data
    T = int(leaf.sum())
    states = rng.integers(0, S, (P, T)).astype(np.int8)
    masks = (np.uint64(1) << states.astype(np.uint64))
    lost = rng.random((P, T)) < 0.2
    states[lost] = -1
    masks[lost] = rng.integers(1, 2 ** S, lost.sum()).astype(np.uint64)
    pi, Q, lam, U, V, dQ = _model(S, K, rng)
    bl = rng.uniform(0.01, 0.4, n)
    kw = dict(class_w=rng.dirichlet(np.ones(K)), rates=rng.uniform(0.3, 2.0, M), rate_w=rng.dirichlet(np.ones(M)))
    want = _capi.WANT_LNL | _capi.WANT_SITE_LNL | _capi.WANT_GRAD_T | _capi.WANT_GRAD_GLOBAL
    ctx = _capi.Context(0)
    out = []
    for pad in (False, True):
        # a mask of every state is missing data in both
        mk = np.where(masks == np.uint64(2 ** S - 1), np.uint64(0), masks) if pad else masks
        pr = _capi.Problem(ctx, parent, leaf, taxon, states, mk, np.arange(1, P + 1, dtype=np.float64))
        if pad:
            extra = 5 - S
            q, l, u, v, d, p5 = Q, lam, U, V, dQ, pi
            for _ in range(extra):
                q, l, d, p5 = _pad(q, (1, 2)), _pad(l, (1,)), _pad(d, (2, 3)), np.append(p5, 0.0)
                u, v = _pad(u, (1, 2)), _pad(v, (1, 2))
                u[:, -1, -1] = v[:, -1, -1] = 1.0
            pr.set_model(pi=p5, Q=q, lam=l, U=u, V=v, dQ=d, **kw)
        else:
            pr.set_model(pi=pi, Q=Q, lam=lam, U=U, V=V, dQ=dQ, **kw)
        r = pr.eval(bl, want)
        out.append((r["lnl"], r["site_lnl"].copy(), r["grad_t"].copy(), r["grad_dir"].copy(), r["grad_class_w"].copy(), r["grad_rate_w"].copy()))
        pr.close()
    ctx.close()
    # the same FP64 sums in another order, at most 3000 terms: 3000 x 2^-53 relative to the largest component, times 30
    for a, b in zip(*out):
        scale = max(1.0, float(np.max(np.abs(b))))
        assert np.max(np.abs(np.asarray(a) - np.asarray(b))) <= 1e-11 * scale
