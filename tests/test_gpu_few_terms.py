"""Lists of a few strings below the row kernel's size: the kernel that is taken on
both sides of the rule, and values against the oracle (FP64 1e-13, FP32 1e-6: sums
of at most eight terms)."""
import numpy as np
import pytest
import torch

import reapers_b200 as rb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TILED, RUNS = 1, 4


@pytest.mark.parametrize("L,dtype,T,kernel", [
    (16, "c64", 1, RUNS), (17, "c64", 1, TILED), (17, "c128", 1, TILED), (17, "c64", 2, RUNS), (17, "c128", 2, TILED),
    (17, "c128", 3, RUNS),
    (18, "c64", 1, TILED), (18, "c64", 6, TILED), (18, "c64", 7, RUNS)])
def test_kernel_and_values(cuda, L, dtype, T, kernel):
    rng = np.random.default_rng(10 * L + T)
    x, z = rng.integers(0, 1 << L, T), rng.integers(0, 1 << L, T)
    bits = np.zeros(T, np.uint64)
    for i in range(L):
        bits |= (((x >> i) & 1) << (2 * i)).astype(np.uint64) | (((z >> i) & 1) << (2 * i + 1)).astype(np.uint64)
    coeff = rng.standard_normal(T) + 1j * rng.standard_normal(T)
    ham = rb.Hamiltonian(L, bits, coeff, dtype)
    assert ham.info()["kernel"] == kernel
    v = rb.random_state(L, dtype, seed=3, normalize=False)
    out = torch.full_like(v, float("nan"))
    ham.apply(out, v)
    ref = O.apply(L, bits, coeff, v.cpu().numpy().astype(np.complex128))
    assert np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref) < (1e-13 if dtype == "c128" else 1e-6)
    ham.close()
