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


@pytest.mark.parametrize("n", [9, 10, 11])
def test_first_columns_around_the_change_of_threads(cuda, n):
    """Ten rows are the last for a CTA of 256 threads; 1e-13 as for the other sizes
    without squarings (|f A| stays below 5.37 in the 1-norm)."""
    import numpy as np
    import scipy.linalg as sla

    import reapers_b200 as rb
    from reapers_b200 import stepper as SP
    rb.init(0)
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A *= 4.0 / np.abs(A).sum(axis=0).max()
    f = np.exp(2j * np.pi * np.arange(4) / 4) * np.linspace(1.3, 0.01, 4)
    ref = np.stack([sla.expm(v * A)[:, 0] for v in f])
    assert np.max(np.abs(SP.expm_first_columns(A, f) - ref)) <= 1e-13 * max(1.0, np.max(np.abs(ref)))
