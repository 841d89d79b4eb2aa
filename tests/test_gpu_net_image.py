"""The trainer's BF16 image of the weights, which each Adam step updates in place
beside the FP32 blob: after any number of steps the gradient equals, bit for bit,
that of a new trainer made from the blob, whose image is built anew; at batches on
both sides of a tile of 128 samples and of eight tiles' partials."""
import numpy as np
import pytest

from wrapd_b200 import prox_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(1, 1), (127, 127), (129, 128), (300, 129), (1153, 1024), (1153, 1153)])
def test_image_follows_the_blob(lib_built, n, batch):
    rng = np.random.default_rng(n + batch)
    X = rng.uniform(0.5, 1.5, (n, 5)).astype(np.float32)
    T = (X[:, :3] * rng.uniform(0.9, 1.1, (n, 3))).astype(np.float32)
    blob = prox_net.init_blob(X, T, 1)
    a = prox_net.Trainer(blob)
    a.set_data(X, T)
    a.train(epochs=3, batch=batch, lr=1e-2, lr_end=1e-3, seed=2)
    after = a.blob()
    assert not np.array_equal(after, blob)
    b = prox_net.Trainer(after)
    b.set_data(X, T)
    la, ga = a.grad(0, n)
    lb, gb = b.grad(0, n)
    a.close()
    b.close()
    np.testing.assert_array_equal(ga, gb)
    assert la == lb
