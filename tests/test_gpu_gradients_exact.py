"""The gradients of a chain without scattering, where every history is the same and
both have a closed form: each cell's term on its own, the chain's first and last cells
included, in both forms of the kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,mu,width", [(1, 1.0, .3), (2, .6, .1), (40, .7, .01), (256, 1.0, 2e-3), (257, 1.0, 2e-3),
                                        (300, .8, 5e-3), (700, .5, 1e-3), (300, .9, .05)])
def test_every_cell_of_an_unscattered_flight(mcg, mode, m, mu, width):
    """Flight lengths l = dx / mu; W_c the weight after cell c, G the loss, P_c its
    part up to cell c: dF/dsig_a = l (w_c W_c - (G - P_c)), dF/dsig_s = -l (G - P_(c-1)).
    A float32 deposit is off by up to 2^-25 of the weight, width / mu of which it is:
    3e-5 of it at the thinnest, the weight as much after 700 cells; the sums of 64
    equal terms are exact to 2^-18.  In all below 3e-4 of the largest component."""
    rng = np.random.default_rng(m)
    sa = (width * m * rng.uniform(0.5, 1.5, m)).astype(f32)
    w = rng.standard_normal(m).astype(f32)
    w[0], w[-1] = 3.0, -4.0
    n = 64
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, np.full(m, 5e-5, f32), 0.0)
        ctx.adjoint_set_weights(w)
        ctx.adjoint_run(0, n, mu0=mu)
        loss, ga, gs = ctx.adjoint_read()
        assert ctx.counters()["steps"] == n * m
    faces = (np.arange(m + 1, dtype=np.float64).astype(f32) * f32(1.0 / m)).astype(float)
    length = np.diff(faces) / float(f32(mu))
    left = np.exp(-np.cumsum(sa.astype(float) * length))
    before = np.concatenate([[1.0], left[:-1]])
    part = w.astype(float) * (before - left)
    rest = np.concatenate([np.cumsum(part[::-1])[::-1], [0.0]])
    want_a = length * (w * left - rest[1:])
    want_s = -length * rest[:-1]
    assert abs(loss - rest[0]) <= 3e-4 * np.abs(part).sum()
    assert np.abs(ga - want_a).max() <= 3e-4 * np.abs(want_a).max()
    assert np.abs(gs - want_s).max() <= 3e-4 * np.abs(want_s).max()
