"""Mixed-precision models' eigensystems (sweeps on half of the matrix) over state counts and degenerate matrices."""
import numpy as np
import pytest

from test_gpu_jacobi_sizes import _generator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [2, 3, 33, 61, 64])
@pytest.mark.parametrize("kind", ["dense", "blocks", "equal", "none"])
def test_eigensystem_sizes(S, kind):
    from hyphy3 import _capi
    Q, pi = _generator(S, kind, np.random.default_rng(100 * S + len(kind)))
    ctx = _capi.Context(0)
    pr = _capi.Problem(ctx, [-1, 0, 0, 0], [0, 1, 1, 1], [-1, 0, 1, 2], np.zeros((1, 3), dtype=np.int8), np.full((1, 3), 1, np.uint64), [1.0])
    pr.set_model(pi=pi, Q=Q, precision=_capi.PREC_MIXED)
    e = pr.get_eigensystem(0)
    s = np.sqrt(pi)
    sym = s[:, None] * Q / s[None]
    lam = np.linalg.eigvalsh(0.5 * (sym + sym.T))
    # the bounds of the FP64 models' test: about 10 sweeps of 63 rounds on 64 states
    scale = max(1.0, float(np.abs(Q).max()) * S ** 0.5)
    assert np.abs(np.sort(e["lam"]) - np.minimum(lam, 0.0)).max() <= 3e-13 * scale
    assert np.abs(e["U"] @ np.diag(e["lam"]) @ e["V"] - Q).max() <= 3e-13 * scale
    assert np.abs(e["U"] @ e["V"] - np.eye(S)).max() <= 3e-13
    pr.close()
    ctx.close()
