"""The network's gradient is summed over samples in FP64: n equal samples (n a power
of two, so that the mean's factor is exact) give the gradient of one of them bit
for bit.  A product of two FP32 numbers has 48 bits, so a CTA's sum of up to 32
equal ones is exact, and the rest of the sum errs by 2^-53, far below the last
rounding to FP32.  One sweep of four samples per CTA, several in shared memory, and
several in the partial itself (256 inputs)."""
import numpy as np
import pytest

import reapers_b200  # noqa: F401
from reapers_b200 import stepper as SP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out", [(21, 2), (3, 1), (256, 8)])
@pytest.mark.parametrize("n", [4, 64, 512, 4096])
def test_equal_samples_give_one_samples_gradient(cuda, n, n_in, n_out):
    rng = np.random.default_rng(n_in)
    x = rng.standard_normal((1, n_in)).astype(np.float32)
    y = rng.standard_normal((1, n_out)).astype(np.float32)
    net = SP.Mlp(n_in, n_out, seed=7)
    _, one = net.grad(x, y)
    _, many = net.grad(np.repeat(x, n, axis=0), np.repeat(y, n, axis=0))
    assert np.array_equal(many, one)
    net.close()


def test_an_epoch_of_more_steps_than_one_launch_takes(cuda):
    """2^16 + 3 batches of one sample, all equal, so that the shuffle does not
    matter: the same parameters as 2^16 of them and three more in a second call,
    and the mean of the losses of both."""
    rng = np.random.default_rng(5)
    n, x, y = (1 << 16) + 3, rng.standard_normal((1, 2)).astype(np.float32), np.ones((1, 1), np.float32)
    nets = [SP.Mlp(2, 1, seed=3), SP.Mlp(2, 1, seed=3)]
    loss = nets[0].train(np.repeat(x, n, axis=0), np.repeat(y, n, axis=0), epochs=1, batch=1, lr=1e-5)
    first = nets[1].train(np.repeat(x, n - 3, axis=0), np.repeat(y, n - 3, axis=0), epochs=1, batch=1, lr=1e-5)
    last = nets[1].train(np.repeat(x, 3, axis=0), np.repeat(y, 3, axis=0), epochs=1, batch=1, lr=1e-5)
    assert np.array_equal(nets[0].get_params(), nets[1].get_params())
    assert abs(loss - (first * (n - 3) + last * 3) / n) <= 1e-6 * loss
    for net in nets:
        net.close()
