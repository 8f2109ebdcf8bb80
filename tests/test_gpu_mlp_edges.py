"""The surrogate's kernels at the edges of their tiles and pipeline: widths off the 8 values of a padded row,
inner sizes of less than one, of one and of more than four 64-wide tiles, batches of one row and off the
32-row and 128-row tiles, against the CPU check on the same BF16 rounding points. A sum that falls on the
other side of a rounding moves a hidden value by 2^-8 of itself, which in a layer of few units is not
averaged out: 2^-7 on outputs, twice that on gradients, whose factors both can move."""
import numpy as np
import pytest

from oracle import mlp_ref as MR
from test_gpu_mlp import make, relnorm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [1, 0])
@pytest.mark.parametrize("dims,B", [([3, 5, 2], 1), ([7, 11, 9, 5], 33), ([64, 64, 64, 64], 64), ([65, 130, 63, 17], 129),
                                    ([321, 72, 257, 1], 7)])
def test_layers_at_tile_edges(dims, B, kind):
    net, layers = make(dims, kind=kind)
    rng = np.random.Generator(np.random.PCG64(11))
    x = rng.standard_normal((B, dims[0])).astype(np.float32)
    t = rng.standard_normal((B, dims[-1])).astype(np.float32)
    zs, _ = MR.forward(layers, x)
    assert relnorm(net.forward(x), zs[-1]) < 2.0**-7
    loss, g = net.train_step(x, t, lr=0.0, grads=True)
    loss0, g0 = MR.grads(layers, x, t)
    assert abs(loss - loss0) < 2.0**-6 * abs(loss0)
    for l in range(len(dims) - 1):
        assert relnorm(g[l][0], g0[l][0]) < 2.0**-6, l
        assert relnorm(g[l][1], g0[l][1]) < 2.0**-6, l


def test_adam_step_of_ragged_layers():
    """One Adam step from zero moments moves every weight by lr g / (|g| + eps): the tiled update reaches all
    of a ragged layer's weights and biases once. Where |g| is far above eps the step is lr to FP32 rounding
    of the weight (2^-23 of at most 1)."""
    dims, B, lr = [33, 65, 7], 40, 1e-2
    net, layers = make(dims, seed=3)
    rng = np.random.Generator(np.random.PCG64(13))
    x = rng.standard_normal((B, dims[0])).astype(np.float32)
    t = rng.standard_normal((B, dims[-1])).astype(np.float32)
    _, g = net.train_step(x, t, lr=0.0, grads=True)
    net, layers = make(dims, seed=3)
    net.train_step(x, t, lr=lr)
    for l in range(len(dims) - 1):
        W, b = net.get_layer(l)
        for new, old, gr in ((W, layers[l][0], g[l][0]), (b, layers[l][1], g[l][1])):
            step = np.asarray(new, np.float64) - np.asarray(old, np.float64)
            big = np.abs(gr) > 1e-4
            assert big.mean() > 0.5
            np.testing.assert_allclose(step[big], -lr * np.sign(np.asarray(gr))[big], rtol=1e-3)
