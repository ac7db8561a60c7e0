"""Products captured into CUDA graphs: two graphs of one Hamiltonian, replayed on two
streams at once, give what the plain calls give (sums in another order: 1e-13 in
FP64, 1e-5 in FP32 for lists of a few thousand terms), and so does a replay beside
plain calls.  States of several blocks whose terms are dealt out to several CTAs,
of one CTA per block, and of the split kernel."""
import numpy as np
import pytest
import torch

import reapers_b200 as rb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [("c128", 1e-13), ("c64", 1e-5)])
@pytest.mark.parametrize("model,L", [("dense", 8), ("dense", 12), ("sparse", 14), ("sparse", 16), ("sparse", 17),
                                     ("chain", 9)])
def test_two_graphs_of_one_hamiltonian(cuda, model, L, dtype, tol):
    if model == "dense":
        bits, coeff = rb.syk.dense_syk(2 * L, seed=3)
    elif model == "sparse":
        bits, coeff = rb.syk.sparse_syk(2 * L, 8, seed=3)
    else:
        bits, coeff = rb.syk.xxz_chain(L, 1.0, np.linspace(-1, 1, L))
    ham = rb.Hamiltonian(L, bits, coeff, dtype)
    x = [rb.random_state(L, dtype, seed=s) for s in (1, 2, 3)]
    want = [torch.empty_like(v) for v in x]
    for w, v in zip(want, x):
        ham.apply(w, v)
    rb.synchronize()
    out = [torch.empty_like(v) for v in x]
    graphs = []
    for k in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=rb.stream(), capture_error_mode="thread_local"):
            for _ in range(8):
                ham.apply(out[k], x[k])
        graphs.append(g)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for o in out:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        ham.apply(out[2], x[2])
        rb.synchronize()
        torch.cuda.synchronize()
        for o, w in zip(out, want):
            err = torch.linalg.vector_norm(o - w) / torch.linalg.vector_norm(w)
            assert err.item() < tol, err
    assert torch.equal(out[2], want[2])
    del graphs
    ham.close()
