"""The sums that the gradients keep between a forward pass and its replay: in
turns when there are more of them than are kept, in smaller ones when there is no
device memory, and a failed set-up of a fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


def _fit(rng, cells, histories):
    total = int(np.sum(cells))
    slabs = [dict(n_cells=int(m), n_histories=int(n), base_seed=11 + 7 * s, seed_mode=0, isotropic=0,
                  mu0=1.0, w0=1.0) for s, (m, n) in enumerate(zip(cells, histories))]
    return slabs, rng.uniform(0.2, 2, total).astype(f32), rng.uniform(0.5, 5, total).astype(f32)


def _close(a, b):
    """Equal but for the order of the float32 sums of a slab's histories."""
    assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()


def test_fit_of_many_items(mcg):
    """2100 items, and the same slabs in two halves."""
    rng = np.random.default_rng(8)
    cells = rng.integers(1, 9, 2100)
    slabs, sa, ss = _fit(rng, cells, rng.integers(1, 60, 2100))
    w = rng.standard_normal(len(sa))
    cut = int(cells[:1000].sum())
    with mcg.Context(mode="fast") as ctx:
        ctx.fit_set(slabs, sa, ss, np.zeros(len(sa)), max_steps=2)
        t, g = ctx.fit_gradient(w)
        ctx.fit_run(2)
        sig, loss = ctx.fit_read()
        for part, k in ((slabs[:1000], slice(0, cut)), (slabs[1000:], slice(cut, None))):
            ctx.fit_set(part, sa[k], ss[k], np.zeros(len(sa[k])), max_steps=2)
            t1, g1 = ctx.fit_gradient(w[k])
            assert np.array_equal(t[k], t1)
            _close(g[k], g1)
            ctx.fit_run(2)
            # Adam's first steps are of the learning rate's size whatever the
            # gradient's; cells without a gradient to speak of may go either way
            far = np.abs(ctx.fit_read()[0] - sig[k]) > 1e-3
            assert far.sum() <= 0.01 * far.size
    assert loss.shape == (2,) and np.isfinite(loss).all()


@pytest.mark.parametrize("turns", [1, 3])
def test_fit_of_long_short_and_thick_slabs(mcg, fail_allocation, turns):
    """Slabs that go to the two forward kernels of the fit, in one turn and in
    several (a failed allocation halves the sums): the tracker's tallies, and the
    adjoint's gradients but for the order of the float32 sums."""
    rng = np.random.default_rng(6)
    cells = np.array([1, 20, 64, 100, 101, 300, 500, 40])
    histories = [5000, 9000, 2048, 2049, 3000, 8193, 700, 1]
    width = [.2, .01, .3, 1e-3, .005, .3, .002, .1]
    per = np.repeat(cells, cells)
    sa = (np.repeat(width, cells) * per * rng.uniform(0.5, 1.5, per.size)).astype(f32)
    ss = (0.7 * np.repeat(width, cells) * per * rng.uniform(0.5, 1.5, per.size)).astype(f32)
    w = rng.standard_normal(per.size).astype(f32)
    slabs = [dict(n_cells=int(m), n_histories=int(n), base_seed=11 + s, seed_mode=0, isotropic=0, mu0=1.0, w0=1.0)
             for s, (m, n) in enumerate(zip(cells, histories))]
    with mcg.Context(mode="fast") as ctx:
        if turns > 1:
            fail_allocation(1)
        ctx.fit_set(slabs, sa, ss, np.zeros(per.size), max_steps=1)
        t, g = ctx.fit_gradient(w)
    o = 0
    for d in slabs:
        m, n, k = d["n_cells"], d["n_histories"], slice(o, o + d["n_cells"])
        o += m
        with mcg.Context(mode="fast") as ctx:
            ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa[k], ss[k], 1e-12)
            ctx.adjoint_set_weights(w[k])
            ctx.adjoint_run(0, n, base_seed=d["base_seed"])
            assert np.array_equal(t[k], ctx.tally() / n)
            _close(g[k], ctx.adjoint_read()[1])


@pytest.fixture
def fail_allocation(mcg):
    lib = mcg.load_library()
    yield lib.mcg_testing_fail_allocation
    lib.mcg_testing_fail_allocation(-1)


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_adjoint_with_less_memory(mcg, mode, fail_allocation):
    """Without memory for every history's sum the run takes turns of half as
    many (tally and loss are exact sums); below 4096 it fails and says so."""
    m, n = 300, 20_000
    rng = np.random.default_rng(1)
    sa, ss = rng.uniform(0.2, 2, (2, m)).astype(f32)
    w = rng.standard_normal(m).astype(f32)
    out = []
    for short in (False, True):
        with mcg.Context(mode=mode) as ctx:
            ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, ss, 1e-12)
            ctx.adjoint_set_weights(w)
            if short:
                fail_allocation(0)
                with pytest.raises(mcg.MCGError) as e:
                    ctx.adjoint_run(0, 4000)
                assert e.value.code == 2  # MCG_ERR_CUDA
                fail_allocation(0)
            ctx.adjoint_run(0, n)
            out.append((ctx.tally_q(), *ctx.adjoint_read()))
            # the failure was used up: a set-up's allocations succeed
            ctx.set_layers_xs([0], [m + 1], [f32(0.001)], np.ones(m + 1), np.ones(m + 1), 1e-12)
    (q0, l0, a0, s0), (q1, l1, a1, s1) = out
    assert np.array_equal(q0, q1) and l0 == l1
    _close(a0, a1)
    _close(s0, s1)


def test_fit_with_less_memory(mcg, fail_allocation):
    """Half the sums: the same tally; none, or no memory at all: no fit is set."""
    rng = np.random.default_rng(2)
    slabs, sa, ss = _fit(rng, [40, 30, 20], [9000, 100, 8192])  # four items
    zero, w = np.zeros(90), rng.standard_normal(90)
    with mcg.Context(mode="fast") as ctx:
        ctx.fit_set(slabs, sa, ss, zero, max_steps=1)
        t, g = ctx.fit_gradient(w)
        fail_allocation(1)
        ctx.fit_set(slabs, sa, ss, zero, max_steps=1)
        t1, g1 = ctx.fit_gradient(w)
        assert np.array_equal(t, t1)
        _close(g, g1)
        for one, after in ((False, 0), (True, 1)):
            fail_allocation(after)
            with pytest.raises(mcg.MCGError) as e:
                ctx.fit_set(slabs[1:2] if one else slabs, sa, ss, zero, max_steps=1)
            assert e.value.code == 2  # MCG_ERR_CUDA
            with pytest.raises(mcg.MCGError) as e:
                ctx.fit_run(0)
            assert e.value.code == 5  # MCG_ERR_STATE
        ctx.fit_set(slabs, sa, ss, zero, max_steps=1)
        assert np.array_equal(ctx.fit_gradient(w)[0], t)
