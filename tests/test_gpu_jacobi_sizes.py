"""Device eigensystems (h3g_model_get_eigensystem) over state counts and matrices with degenerate or no couplings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _generator(S, kind, rng):
    pi = rng.uniform(0.5, 1.5, S)
    pi /= pi.sum()
    R = rng.uniform(0.1, 2.0, (S, S))
    R = R + R.T
    if kind == "blocks":                    # two sets of states without transitions between them
        R[: S // 2, S // 2:] = 0.0
        R[S // 2:, : S // 2] = 0.0
    elif kind == "equal":                   # every exchangeability the same: one (S - 1)-fold eigenvalue
        R[:] = 1.0
    elif kind == "none":                    # no transitions at all
        R[:] = 0.0
    Q = R * pi[None, :]
    np.fill_diagonal(Q, 0.0)
    Q[np.diag_indices(S)] = -Q.sum(1)
    return Q, pi


@pytest.mark.parametrize("S", [2, 3, 4, 31, 32, 33, 61, 62, 63, 64])
@pytest.mark.parametrize("kind", ["dense", "blocks", "equal", "none"])
def test_eigensystem_sizes(S, kind):
    from hyphy3 import _capi
    rng = np.random.default_rng(100 * S + len(kind))
    Q, pi = _generator(S, kind, rng)
    ctx = _capi.Context(0)
    states = np.zeros((1, 3), dtype=np.int8)
    pr = _capi.Problem(ctx, [-1, 0, 0, 0], [0, 1, 1, 1], [-1, 0, 1, 2], states, np.full((1, 3), 1, np.uint64), [1.0])
    pr.set_model(pi=pi, Q=Q)
    e = pr.get_eigensystem(0)
    s = np.sqrt(pi)
    lam = np.linalg.eigvalsh(0.5 * ((s[:, None] * Q / s[None]) + (s[:, None] * Q / s[None]).T))
    # backward error of ~10 sweeps of 63 rounds on 64 states: below 64 * 10 * 2^-52 = 1.4e-13 of the norm, times sqrt(pi_max / pi_min) <= 1.8
    scale = max(1.0, float(np.abs(Q).max()) * S ** 0.5)
    assert np.abs(np.sort(e["lam"]) - np.minimum(lam, 0.0)).max() <= 3e-13 * scale
    assert np.abs(e["U"] @ np.diag(e["lam"]) @ e["V"] - Q).max() <= 3e-13 * scale
    assert np.abs(e["U"] @ e["V"] - np.eye(S)).max() <= 3e-13
    pr.close()
    ctx.close()
