"""The triangular solve's schedule is chosen by its own measurement wherever the factorization runs
persistently, and the result does not depend on it."""
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
sys.path[:0] = {paths!r}
import numpy as np, scipy.sparse as sp
from inla_b200 import BatchSolver, _lib

def blocks(depth, k, seed):  # binary tree of dense blocks, each coupled to its parent
    rng = np.random.default_rng(seed)
    nb = 2 ** depth - 1
    i, j = [], []
    lo, full = np.tril_indices(k, -1), np.indices((k, k)).reshape(2, -1)
    for b in range(nb):
        i.append(b * k + lo[0]); j.append(b * k + lo[1])
        if b:
            i.append(b * k + full[0]); j.append((b - 1) // 2 * k + full[1])
    i, j = np.concatenate(i), np.concatenate(j)
    a = sp.coo_matrix((rng.uniform(-1, 1, len(i)), (i, j)), shape=(nb * k, nb * k)).tocsc()
    a = a + a.T
    return (a + sp.diags(np.asarray(abs(a).sum(axis=0)).ravel() + 1.0)).tocsc()

for depth, k, B in ((3, 60, 1), (4, 30, 2), (5, 60, 1), (7, 6, 3), (7, 60, 1), (8, 30, 1)):
    q = blocks(depth, k, depth)
    q.sort_indices()
    b = np.random.default_rng(k).standard_normal((B, q.shape[0]))
    out = []
    for mode in (1, 0, 2):
        _lib.check(_lib.lib().inla_set_persistent_schedule(mode))
        if mode == 1:
            print("TREE:", depth, k, B, file=sys.stderr, flush=True)
        sv = BatchSolver(q, max_batch=B)
        sv.factorize(np.tile(q.data, (B, 1)))
        out.append(sv.solve(b))
        assert np.max(np.abs(q @ out[-1].T - b.T)) < 1e-9
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
"""


def test_choice_is_measured():
    root = Path(__file__).resolve().parent.parent
    child = CHILD.format(paths=[str(root / "rust-inla_b200")])
    r = subprocess.run([sys.executable, "-c", child], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "INLA_DEBUG": "1"})
    assert r.returncode == 0, r.stderr[-2000:]
    line = re.compile(r"(schedule|solve) B=\d+: level launches ([\d.]+) ms, persistent ([\d.]+) ms -> (\w+)")
    persistent = False
    for tree in r.stderr.split("TREE:")[1:]:
        picks = {m[0]: m[1:] for m in line.findall(tree)}
        assert "schedule" in picks, tree
        assert ("solve" in picks) == (picks["schedule"][2] == "persistent")
        for levels, queue, pick in picks.values():
            assert levels == queue or pick == ("persistent" if float(queue) < float(levels) else "levels")
        persistent = persistent or "solve" in picks
    assert persistent  # the solve was measured on some tree
