"""Imaginary time over many cycles: exp(-beta H) with the ground state's energy at
zero stays below one, but the pieces of its Taylor series around the mean of the
diagonal grow like e^(beta ||H|| / 2), beyond a double for the long times here;
those go to the Pade form, which scales the matrix as a whole.  Against the
eigensystem in numpy; absolute errors are a few u beta ||H|| (below 16 * 1.1e-16
* 2e3), over a result of norm 0.02: 1e-10 holds."""
import numpy as np
import pytest

import reapers_b200 as rb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau,m,phase", [
    (60.0, 32, 1.0),     # exp(-tau H)
    (60.0, 32, -1j),     # the same as exp(-i tau (-i H)), H' = -i H not Hermitian
    (60.0, 24, 1.0),
    (8.0, 24, 1.0),      # short enough for the series
])
def test_long_imaginary_time(cuda, tau, m, phase):
    L = 9
    bits, coeff = rb.syk.xxz_chain(L, 1.0, np.random.default_rng(2).uniform(-2.0, 2.0, L))
    eye = np.eye(1 << L, dtype=np.complex128)
    H = np.stack([O.apply(L, bits, coeff, eye[i]) for i in range(1 << L)], axis=1)
    w, V = np.linalg.eigh(H)
    bits = np.concatenate([bits, [0]]).astype(np.uint64)
    coeff = np.concatenate([coeff, [-w[0]]]) * phase
    ham = rb.Hamiltonian(L, bits, coeff, "c128")
    x = rb.random_state(L, "c128", seed=3)
    ref = V @ (np.exp(-tau * (w - w[0])) * (V.conj().T @ x.cpu().numpy()))
    t, beta = (0.0, tau) if phase == 1.0 else (tau, 0.0)
    st = rb.evolve(ham, x, t, beta, m, 1e-12, max_iters=14)
    assert st["last_err"] < 1e-12, st
    err = np.linalg.norm(x.cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err < 1e-10, (err, st)
    ham.close()
