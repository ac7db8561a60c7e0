"""Term lists between what the row kernel's shared memory takes beside its ring
(about 1400 real strings, 700 complex ones) and the largest row table (2048):
they run, alone and as a problem of a batch left to its default place.  Sampled
rows against the oracle (FP64 1e-12, FP32 1e-5, the suite's bounds for sums of a
thousand terms); the OTOC of the default place against a team's (FP32 states,
2e-6 as between the other places)."""
import numpy as np
import pytest
import torch

import reapers_b200 as rb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _strings(rng, L, T, diag=0):
    x, z = rng.integers(1, 1 << L, T), rng.integers(0, 1 << L, T)
    x[:diag] = 0
    bits = np.zeros(T, np.uint64)
    for i in range(L):
        bits |= (((x >> i) & 1) << (2 * i)).astype(np.uint64)
        bits |= (((z >> i) & 1) << (2 * i + 1)).astype(np.uint64)
    return bits


@pytest.mark.parametrize("L,dtype,T,diag,cplx,rows", [
    (20, "c64", 1250, 0, False, True),      # fits
    (20, "c64", 1500, 0, False, False),
    (19, "c128", 1900, 0, False, False),
    (19, "c64", 1000, 0, True, False),      # 2000 records
    (20, "c128", 2000, 900, False, False),  # terms and diagonal
    (22, "c64", 4090, 2045, False, False),  # the largest tables
])
def test_lists_near_the_limit(cuda, L, dtype, T, diag, cplx, rows):
    rng = np.random.default_rng(T)
    bits = _strings(rng, L, T, diag)
    coeff = rng.standard_normal(T) + (1j * rng.standard_normal(T) if cplx else 0.0)
    ham = rb.Hamiltonian(L, bits, coeff, dtype)
    assert (ham.info()["kernel"] == 2) == rows
    x = rb.random_state(L, dtype, seed=5, normalize=False)
    out = torch.full_like(x, float("nan"))
    ham.apply(out, x)
    host, got = x.cpu().numpy().astype(np.complex128), out.cpu().numpy()
    idx = np.unique(np.concatenate([[0, 1, (1 << L) - 1], rng.integers(0, 1 << L, 1500)])).astype(np.uint64)
    ref = O.apply_at(bits, coeff, idx, lambda k: host[k])
    err = np.linalg.norm(got[idx] - ref) / np.linalg.norm(ref)
    assert err < (1e-12 if dtype == "c128" else 1e-5), err
    ham.close()


def test_default_place_of_a_long_list(cuda):
    L, T = 19, 1500
    rng = np.random.default_rng(4)
    bits, coeff = _strings(rng, L, T), rng.standard_normal(T) * 0.02 + 0j
    p = {"len": L, "bits": bits, "coeff": coeff, "w": rb.syk.majorana(2 * L, 1), "v": rb.syk.majorana(2 * L, 2),
         "psi0": rb.random_state(L, "c64", seed=6)}
    F = []
    for team in (0, 8):
        b = rb.BatchOTOC([dict(p, team=team)], krydim=8, tol=1e-7)
        F.append(b.run(np.array([0.3]))[0][0, 0])
        b.close()
    assert abs(F[0] - F[1]) < 2e-6, F
