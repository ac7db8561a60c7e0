"""The device memory of a batch left to its default places: problems run alone on
the whole GPU share one set of vectors, the largest one's, and where memory is too
short for the fastest places the teams by qubit count take the problems."""
import numpy as np
import pytest
import torch

import reapers_b200 as rb
from reapers_b200 import _lib

pytestmark = pytest.mark.gpu


def _problem(L, seed):
    rng = np.random.default_rng(seed)
    bits, coeff = rb.syk.xxz_chain(L, 1.0, rng.uniform(-1, 1, L))
    return {"len": L, "bits": bits, "coeff": coeff * 0.3, "w": rb.syk.majorana(2 * L, 1),
            "v": rb.syk.majorana(2 * L, 2), "psi0": rb.random_state(L, "c64", seed=seed)}


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _run(probs, **kw):
    b = rb.BatchOTOC(probs, krydim=8, tol=1e-7, max_restarts=kw.get("max_restarts", 4))
    try:
        return b.run(np.array([0.0, 0.3]))
    finally:
        b.close()


def test_solo_sizes_share_their_vectors(cuda):
    """Of 20, 21 and 22 qubits, out of order: twelve vectors of the largest (400 MB)
    and small change, not 1.75 times that; values and counts as alone."""
    sizes = [20, 22, 21, 22, 20]
    probs = [_problem(L, 10 + i) for i, L in enumerate(sizes)]
    single = [_run([p]) for p in probs]
    free = _free()
    b = rb.BatchOTOC(probs, krydim=8, tol=1e-7, max_restarts=4)
    used = free - _free()
    F, ap = b.run(np.array([0.0, 0.3]))
    assert free - _free() <= used + (2 << 20)      # nothing grows while it runs
    b.close()
    assert used < 12 * (8 << 22) + (64 << 20), used
    assert _free() >= free - (2 << 20)
    for p, (f, a) in enumerate(single):
        assert np.array_equal(F[p], f[0]) and np.array_equal(ap[p], a[0])


def test_short_memory_falls_back_to_teams(cuda):
    """148 problems of 18 qubits go to teams of two (148 slots of 25 MB) and one of
    24 runs alone (1.6 GB): 5.2 GB together, where the teams by qubit count take
    1.6 GB in all."""
    _lib.call("rp_workspace_release")
    shared = [_problem(18, s) for s in range(4)]
    probs = [shared[i % 4] for i in range(148)] + [_problem(24, 9)]
    want = _run([dict(p, team=4 if p["len"] == 18 else 16) for p in probs], max_restarts=1)
    filler = torch.empty(_free() - (3 << 30), dtype=torch.uint8, device="cuda")
    got = _run(probs, max_restarts=1)
    del filler
    torch.cuda.empty_cache()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
