"""Term lists too long for the row kernel's table on states of its size: the run
kernel where terms share X masks, the tiled kernel where (almost) every term has
its own, against the oracle on sampled rows (FP64 1e-12, FP32 1e-5, the suite's
bounds for sums of a few thousand terms) and with accumulation."""
import numpy as np
import pytest
import torch

import reapers_b200 as rb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TILED, RUNS = 1, 4


def _strings(rng, L, T, share):
    """T strings over `share` T distinct X masks."""
    X = int(T * share)
    masks = rng.choice((1 << L) - 1, X, replace=False) + 1
    x, z = np.concatenate([masks, rng.choice(masks, T - X)]), rng.integers(0, 1 << L, T)
    bits = np.zeros(T, np.uint64)
    for i in range(L):
        bits |= (((x >> i) & 1) << (2 * i)).astype(np.uint64)
        bits |= (((z >> i) & 1) << (2 * i + 1)).astype(np.uint64)
    return bits


@pytest.mark.parametrize("L,dtype,T,share,cplx,kernel", [
    (20, "c64", 2500, 1.0, False, TILED),
    (20, "c128", 2500, 1.0, False, TILED),
    (22, "c64", 2100, 1.0, False, TILED),
    (20, "c64", 2500, 0.8, True, TILED),
    (21, "c128", 2200, 0.8, True, TILED),
    (20, "c64", 2500, 0.7, False, RUNS),
    (20, "c128", 2500, 0.9, False, RUNS),
    (20, "c128", 2500, 0.5, True, RUNS),
    (19, "c64", 2500, 1.0, False, RUNS),
    (19, "c128", 2500, 1.0, True, RUNS),
    (20, "c64", 9000, 0.01, False, RUNS),
])
def test_kernel_and_values(cuda, L, dtype, T, share, cplx, kernel):
    rng = np.random.default_rng(T + L)
    bits = _strings(rng, L, T, share)
    coeff = rng.standard_normal(T) + (1j * rng.standard_normal(T) if cplx else 0.0)
    ham = rb.Hamiltonian(L, bits, coeff, dtype)
    assert ham.info()["kernel"] == kernel
    x = rb.random_state(L, dtype, seed=5, normalize=False)
    out = torch.full_like(x, float("nan"))
    ham.apply(out, x)
    host, got = x.cpu().numpy().astype(np.complex128), out.cpu().numpy()
    idx = np.unique(np.concatenate([[0, 1, (1 << L) - 1], rng.integers(0, 1 << L, 1000)])).astype(np.uint64)
    ref = O.apply_at(bits, coeff, idx, lambda k: host[k])
    tol = 1e-12 if dtype == "c128" else 1e-5
    assert np.linalg.norm(got[idx] - ref) / np.linalg.norm(ref) < tol
    ham.apply(out, x, accumulate=True)
    err = np.linalg.norm(out.cpu().numpy()[idx] - 2 * ref) / np.linalg.norm(ref)
    assert err < 2 * tol, err
    ham.close()
