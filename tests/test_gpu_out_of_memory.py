"""Calls that find no device memory fail alone: the next call runs.  (The sizes
asked for exceed any GPU's memory, or a filler leaves less than they need.)"""
import ctypes as C

import numpy as np
import pytest
import torch

import reapers_b200 as rb
from reapers_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture
def clean(cuda):
    _lib.call("rp_workspace_release")
    torch.cuda.empty_cache()
    yield
    _lib.call("rp_workspace_release")
    torch.cuda.empty_cache()


@pytest.mark.parametrize("entry", ["rp_evolve", "rp_alloc"])
def test_the_call_after_a_failed_allocation(clean, entry):
    x = torch.ones(64, dtype=torch.complex128, device="cuda")
    if entry == "rp_evolve":   # 66 vectors of 64 GB: refused before the state is read
        ham = rb.Hamiltonian(32, [1], [1.0], "c128")
        with pytest.raises(rb.RPError) as e:
            _lib.call("rp_evolve", ham.handle, C.c_void_p(x.data_ptr()), 1.0, 0.0, 64, 1e-12, 0, None)
        assert e.value.code == -4
        ham.close()
    else:
        p = C.c_void_p()
        with pytest.raises(rb.RPError):
            _lib.call("rp_alloc", C.byref(p), 1 << 50)
    assert rb.norm(x) == 8.0
    small = rb.Hamiltonian(6, [1], [1.0], "c128")
    y = torch.empty_like(x)
    small.apply(y, x)
    rb.evolve(small, x, 0.5, krydim=4)
    assert abs(rb.norm(x) - 8.0) < 1e-12 and np.isfinite(rb.norm(y))
    small.close()


def _leave(nbytes):
    """A tensor that takes all device memory but nbytes."""
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - nbytes, dtype=torch.uint8, device="cuda")


def test_a_basis_that_cannot_grow_gives_back_what_it_took(clean):
    L, vec = 25, 8 << 25
    ham = rb.Hamiltonian(L, *rb.syk.xxz_chain(L, 1.0, np.zeros(L)), "c64")
    x = rb.random_state(L, "c64", seed=1)
    rb.evolve(ham, x, 0.1, krydim=4, max_iters=1)
    filler = _leave(int(3.5 * vec))
    free = torch.cuda.mem_get_info()[0]
    with pytest.raises(rb.RPError) as e:
        rb.evolve(ham, x, 0.1, krydim=20, max_iters=1)
    assert e.value.code == -4
    assert torch.cuda.mem_get_info()[0] == free
    before = x.clone()
    st = rb.evolve(ham, x, 0.1, krydim=5, max_iters=1)   # room for one more
    assert st["applies"] == 5 and not torch.equal(x, before) and abs(rb.norm(x) - 1.0) < 1e-4
    del filler
    ham.close()


def test_a_krylov_matrix_that_cannot_grow_leaves_the_workspace_whole(clean):
    """64 vectors: the matrix and its scratch have 256 rows for four cycles (11 MB)
    and would get 512 (46 MB) in the fifth."""
    L = 9
    ham = rb.Hamiltonian(L, *rb.syk.xxz_chain(L, 1.0, np.linspace(-2, 2, L)), "c128")
    v = rb.random_state(L, "c128", seed=1)
    first, again, x = v.clone(), v.clone(), v.clone()
    rb.evolve(ham, first, 30.0, krydim=64, tol=0.0, max_iters=4)
    filler = _leave(24 << 20)
    with pytest.raises(rb.RPError) as e:
        rb.evolve(ham, x, 30.0, krydim=64, tol=0.0, max_iters=5)
    assert e.value.code == -4
    rb.evolve(ham, again, 30.0, krydim=64, tol=0.0, max_iters=4)
    assert torch.equal(again, first)
    del filler
    torch.cuda.empty_cache()
    rb.evolve(ham, x.copy_(v), 30.0, krydim=64, tol=0.0, max_iters=5)
    _lib.call("rp_workspace_release")
    rb.evolve(ham, again.copy_(v), 30.0, krydim=64, tol=0.0, max_iters=5)
    assert torch.equal(again, x)
    ham.close()
