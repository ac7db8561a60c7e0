"""Row plans with a fused diagonal on both sides of the rule that merges them (2^22
elements): diagonal lists that fold little or much, lists without terms to sum,
and lists with them, against the oracle on sampled rows (FP64 1e-12, FP32 1e-5, the
suite's bounds for sums of some hundred terms) and bit for bit in two shards."""
import numpy as np
import pytest
import torch

import reapers_b200 as rb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

L = 22


def _masks(kind, rng):
    pairs = [(1 << i) | (1 << j) for i in range(L) for j in range(i)]
    if kind == "four Z strings":
        return [0] * 4, rng.integers(1, 1 << L, 4)
    if kind == "Z strings of the tile":
        return [0] * 60, [int(z) << 12 for z in rng.integers(1, 1 << (L - 12), 60)]
    if kind == "transverse Ising":
        return [1 << i for i in range(L)] + [0] * (L - 1), [0] * L + [3 << i for i in range(L - 1)]
    if kind == "all ZZ and X":
        return [1 << i for i in range(L)] + [0] * len(pairs), [0] * L + pairs
    if kind == "all XX, YY and Z":
        return pairs + pairs + [0] * L, [0] * len(pairs) + pairs + [1 << i for i in range(L)]
    x = rng.integers(1, 1 << L, 60)      # random
    x[:30] = 0
    return x, rng.integers(1, 1 << L, 60)


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("kind", ["four Z strings", "Z strings of the tile", "transverse Ising", "all ZZ and X",
                                  "all XX, YY and Z", "random"])
def test_values(cuda, kind, dtype):
    rng = np.random.default_rng(3)
    x, z = (np.array([int(v) for v in m], dtype=np.int64) for m in _masks(kind, rng))
    bits = np.zeros(len(x), np.uint64)
    for i in range(L):
        bits |= (((x >> i) & 1) << (2 * i)).astype(np.uint64) | (((z >> i) & 1) << (2 * i + 1)).astype(np.uint64)
    coeff = rng.standard_normal(len(bits)) + 0j
    ham = rb.Hamiltonian(L, bits, coeff, dtype)
    assert ham.info()["kernel"] == 2 and ham.info()["diag_terms"] >= 4
    v = rb.random_state(L, dtype, seed=5, normalize=False)
    out = torch.full_like(v, float("nan"))
    ham.apply(out, v)
    host, got = v.cpu().numpy().astype(np.complex128), out.cpu().numpy()
    idx = np.unique(np.concatenate([[0, 1, (1 << L) - 1], rng.integers(0, 1 << L, 3000)])).astype(np.uint64)
    ref = O.apply_at(bits, coeff, idx, lambda k: host[k])
    err = np.linalg.norm(got[idx] - ref) / np.linalg.norm(ref)
    assert err < (1e-12 if dtype == "c128" else 1e-5), err
    half = (1 << L) // 2
    for r in range(2):
        part = torch.empty_like(v[:half])
        ham.apply_shard(part, [v[:half].clone(), v[half:].clone()], r)
        assert torch.equal(part, out[r * half:(r + 1) * half])
    ham.close()
