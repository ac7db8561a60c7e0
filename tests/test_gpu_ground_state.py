"""ground_state beside the other calls and in its result: the last Arnoldi basis
and the evolves' workspace stay as they are, its memory is torch's and is given
back, and the state it returns is a unit vector whose energy is the one it
reports.  The energy comes from the tridiagonal matrix, the state from the
combination of the basis: they agree to the rounding of the steps, a few u per
step of the coefficients' sum (1e-13 in FP64, 1e-5 in FP32 for twelve steps)."""
import numpy as np
import pytest
import torch

import reapers_b200 as rb
from reapers_b200 import _lib, stepper

pytestmark = pytest.mark.gpu


def _chain(L, dtype, seed=1):
    bits, coeff = rb.syk.xxz_chain(L, 0.7, np.random.default_rng(seed).uniform(-1, 1, L))
    return rb.Hamiltonian(L, bits, coeff, dtype), np.abs(coeff).sum()


@pytest.mark.parametrize("dtype,tol", [("c128", 1e-13), ("c64", 1e-5)])
@pytest.mark.parametrize("L,m,iters", [(1, 2, 1), (4, 2, 5), (9, 5, 1), (9, 5, 2), (9, 5, 40), (12, 12, 7), (17, 10, 6)])
def test_state_and_energy_agree(cuda, L, m, iters, dtype, tol):
    ham, size = _chain(L, dtype)
    E, g = rb.ground_state(ham, krydim=m, maxiter=iters, seed=3)
    assert abs(rb.norm(g) - 1.0) < (1e-12 if dtype == "c128" else 1e-6)
    h = torch.empty_like(g)
    ham.apply(h, g)
    assert abs(rb.dot(g, h) - E) <= tol * size
    E2, g2 = rb.ground_state(ham, krydim=m, maxiter=iters, seed=3)
    assert E2 == E and torch.equal(g2, g)
    ham.close()


def test_an_arnoldi_basis_outlives_a_ground_state(cuda):
    ham, _ = _chain(11, "c128")
    psi = rb.random_state(11, "c128", seed=2)
    basis = stepper.arnoldi(ham, psi, 12)
    c = np.linspace(1, 2, basis.m_eff) + 0.5j
    before = stepper.combine(c, torch.empty_like(psi))
    rb.ground_state(ham, krydim=8, maxiter=2)
    assert torch.equal(stepper.combine(c, torch.empty_like(psi)), before)
    ham.close()


def test_device_memory_is_given_back(cuda):
    """A state of 16 MB: after the call as much memory is free as before it (2 MB
    for the library's fixed scratch on the first call)."""
    _lib.call("rp_workspace_release")
    ham, _ = _chain(20, "c128")
    x = rb.random_state(20, "c128", seed=1)
    rb.norm(x)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    E, g = rb.ground_state(ham, krydim=10, maxiter=2)
    del g
    torch.cuda.empty_cache()
    assert torch.cuda.mem_get_info()[0] >= free - (2 << 20)
    ham.close()


def test_as_little_room_as_the_basis_needs(cuda):
    """The start vector and six more: half a vector beyond them is enough."""
    _lib.call("rp_workspace_release")
    torch.cuda.empty_cache()
    L, vec = 24, 8 << 24
    ham, size = _chain(L, "c64")
    want, _ = rb.ground_state(ham, krydim=6, maxiter=3, seed=5)
    _lib.call("rp_workspace_release")
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - 15 * vec // 2, dtype=torch.uint8, device="cuda")
    E, g = rb.ground_state(ham, krydim=6, maxiter=3, seed=5)
    assert abs(E - want) <= 1e-5 * size
    del filler, g
    torch.cuda.empty_cache()
    ham.close()
