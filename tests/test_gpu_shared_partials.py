"""The run kernel's partial sums are one buffer for all Hamiltonians: products of
several, of different sizes, precisions and numbers of CTAs per block, enqueued
without a wait between them give the bits that each gives alone, also after a
shutdown of the library (in a process of its own, so that the shutdown does not
disturb the other tests')."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import numpy as np, torch
import reapers_b200 as rb
from reapers_b200 import _lib
rb.init(0)
cases = [("dense", 12, "c128"), ("dense", 8, "c64"), ("dense", 10, "c64"), ("sparse", 14, "c128"),
         ("sparse", 15, "c64"), ("dense", 14, "c128"), ("dense", 5, "c128")]
hams, x, want, out = [], [], [], []
for model, L, dtype in cases:
    terms = rb.syk.dense_syk(2 * L, seed=L) if model == "dense" else rb.syk.sparse_syk(2 * L, 8, seed=L)
    hams.append(rb.Hamiltonian(L, *terms, dtype))
    x.append(rb.random_state(L, dtype, seed=L))
    want.append(torch.empty_like(x[-1]))
    out.append(torch.empty_like(x[-1]))
    hams[-1].apply(want[-1], x[-1])
    rb.synchronize()
for again in range(2):
    order = np.random.default_rng(again).integers(0, len(cases), 400)
    for o in out:
        o.fill_(float("nan"))
    for i in order:
        hams[i].apply(out[i], x[i])
    rb.synchronize()
    for i in set(order.tolist()):
        assert torch.equal(out[i], want[i]), cases[i]
    if not again:
        _lib.call("rp_shutdown")
        rb.init(0)
"""


def test_interleaved_products(cuda):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
