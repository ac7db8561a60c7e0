"""The Krylov exponential's shared memory cycle by cycle: it passes through the
48 KB that a kernel has without asking (16 vectors: 39.0, 43.9, 48.8, 53.7 KB in
cycles 8 to 11; 24: 41.4, 49.3 KB in 4 and 5), each limit reached in a process of
its own, as a larger request before it would hide the failure.  Restart counts
and 1e-10 against the oracle (the bound of the other long evolves)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import numpy as np, torch
import reapers_b200 as rb
from oracle import oracle as O
L, m, cycles = 9, {m}, {cycles}
bits, coeff = rb.syk.xxz_chain(L, 1.0, np.random.default_rng(2).uniform(-2.0, 2.0, L))
v = np.random.default_rng(5).standard_normal(1 << L) + 0j
v /= np.linalg.norm(v)
ham = rb.Hamiltonian(L, bits, coeff, "c128")
x = torch.from_numpy(v).cuda()
st = rb.evolve(ham, x, 6.0, 0.0, m, 0.0, max_iters=cycles)
ref, st2 = O.evolve(L, bits, coeff, v, 6.0, 0.0, m, 0.0, max_iters=cycles)
assert st["restarts"] == st2["restarts"] == cycles, (st, st2)
err = np.linalg.norm(x.cpu().numpy() - ref) / np.linalg.norm(ref)
assert err < 1e-10, err
"""


@pytest.mark.parametrize("m,cycles", [(16, 8), (16, 9), (16, 10), (16, 11), (24, 5), (21, 6)])
def test_every_size_launches(cuda, m, cycles):
    r = subprocess.run([sys.executable, "-c", CODE.format(m=m, cycles=cycles)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
