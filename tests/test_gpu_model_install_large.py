"""Models whose arrays are larger than the staging memory: installed in pieces, with little pinned memory.

In a process of its own, where a fake cudaMallocHost refuses blocks above a limit."""
import os
import pathlib
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

FAKE = """
#include <dlfcn.h>
#include <stddef.h>
static size_t limit = (size_t)-1;
int refused = 0;
void set_limit(size_t n) { limit = n; }
int cudaMallocHost(void** p, size_t n) {
    static int (*real)(void**, size_t);
    if (n > limit) { ++refused; return 2; }                       /* cudaErrorMemoryAllocation */
    if (!real) real = (int (*)(void**, size_t))dlsym(dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY), "cudaMallocHost");
    return real(p, n);
}
"""

# 40 taxa, three classes on each of 78 branches: 234 models with 5 dense directions and their own, 49 MB, and no sharing.
# The same three generators on every branch make it a plain mixture of three.  (The results of its 239 directions pin 7.6 MB.)
CHILD = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)          # before the library, which then calls it
import numpy as np
from hyphy3 import _capi
rng = np.random.default_rng(1)
T, S, K = 40, 61, 3
parent, leaves = [-1], [0]
while len(leaves) < T:
    u = leaves.pop(0)
    leaves += [len(parent), len(parent) + 1]
    parent += [u, u]
n = len(parent)
leaf = np.array([u not in parent for u in range(n)], np.uint8)
taxon = np.full(n, -1, np.int32)
taxon[leaf == 1] = np.arange(T)
states = np.where(rng.random((50, T)) < 0.3, rng.integers(0, S, (50, T)), rng.integers(0, S, (50, 1))).astype(np.int8)
pi = rng.uniform(0.5, 1.5, S)
pi /= pi.sum()
Q, dQ = [], rng.standard_normal((6, K, S, S)) * 0.01
dQ -= dQ.mean(-1, keepdims=True)
for k in range(K):
    r = rng.uniform(0.1, 2.0, (S, S))
    q = (r + r.T) * pi[None]
    np.fill_diagonal(q, 0.0)
    np.fill_diagonal(q, -q.sum(1))
    Q.append(q / -(pi * np.diag(q)).sum())
Q = np.array(Q)
w = np.array([0.5, 0.3, 0.2])
bl = rng.exponential(0.1, n)
nb = n - 1
out = []
ctx = _capi.Context(0)
want = _capi.WANT_LNL | _capi.WANT_GRAD_T | _capi.WANT_GRAD_GLOBAL
for large in (False, True):
    pr = _capi.Problem(ctx, parent, leaf, taxon, states, np.uint64(1) << states.astype(np.uint64), np.ones(50))
    if large:
        fake.set_limit(ctypes.c_size_t(int(sys.argv[2])))
        reps = np.tile(np.arange(K), nb)
        off = np.concatenate([[0], np.cumsum(np.where(np.array(parent) < 0, 0, K))]).astype(np.int32)
        pr.set_model(pi=pi, Q=Q[reps], class_w=w[reps], branch_classes=off, dQ=dQ[:5][:, reps], dQ_model=dQ[5][reps])
    else:
        pr.set_model(pi=pi, Q=Q, class_w=w, dQ=dQ[:5], dQ_model=dQ[5])
    r = pr.eval(bl, want)
    g = r["grad_dir"]
    out.append((r["lnl"], r["grad_t"].copy(), g[:5].copy(), g[5:].reshape(-1, K).sum(0)))
    pr.close()
# sums of at most 234 terms and 61 x 61 products, regrouped
for a, b in zip(*out):
    assert np.max(np.abs(np.asarray(a) - b)) <= 1e-10 * np.max(np.abs(b)), (a, b)
# eigensystems as given, each model its own: 1200 of them, 107 MB
pr = _capi.Problem(ctx, [-1, 0, 0, 0], [0, 1, 1, 1], [-1, 0, 1, 2], np.zeros((1, 3), np.int8), np.ones((1, 3), np.uint64), [1.0])
nm = 1200
U, V = rng.standard_normal((2, nm, S, S))
lam = -rng.random((nm, S))
pr.set_model(pi=pi, Q=rng.standard_normal((nm, S, S)), lam=lam, U=U, V=V, class_w=np.full(nm, 1 / nm))
for k in range(nm):
    e = pr.get_eigensystem(k)
    assert np.array_equal(e["lam"], lam[k]) and np.array_equal(e["U"], U[k]) and np.array_equal(e["V"], V[k]), k
assert (ctypes.c_int.in_dll(fake, "refused").value > 0) == (int(sys.argv[2]) < 16 << 20)
pr.close()
ctx.close()
print("installed")
"""


@pytest.mark.parametrize("limit_mb", [16, 9])
def test_install_with_little_pinned_memory(tmp_path, limit_mb):
    (tmp_path / "fake.c").write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "fake.so"), str(tmp_path / "fake.c"), "-ldl"], check=True)
    (tmp_path / "child.py").write_text(textwrap.dedent(CHILD))
    import hyphy3
    env_path = str(pathlib.Path(hyphy3.__file__).resolve().parent.parent)
    r = subprocess.run([sys.executable, str(tmp_path / "child.py"), str(tmp_path / "fake.so"), str(limit_mb << 20)],
                       capture_output=True, text=True, timeout=300, env={**os.environ, "PYTHONPATH": env_path})
    assert r.returncode == 0 and "installed" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
