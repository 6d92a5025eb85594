"""The adjoint's forms on chains of thick cells: without a gradient a lane per
history, with one both passes in one kernel, also on chains longer than the short
ones.  The tally and the loss are exact: event mode's, and the sum of its products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("gradient", [False, True])
@pytest.mark.parametrize("m,wa,ws", [(1, .3, .3), (7, .01, .01), (8, .01, .01), (40, .1, .01), (40, .01, .6),
                                     (257, .05, .01), (300, .3, .2), (300, .01, .3), (700, .034, .02),
                                     (700, .036, .02), (3500, .2, .01), (14_000, .1, .01)])
def test_thick_forms(mcg, mode, gradient, m, wa, ws):
    rng = np.random.default_rng(m)
    sa = (wa * m * rng.uniform(0.5, 1.5, m)).astype(f32)
    ss = (ws * m * rng.uniform(0.5, 1.5, m)).astype(f32)
    w = rng.standard_normal(m).astype(f32)
    with mcg.Context(mode=mode) as ctx:
        for min_w, n in ((1e-12, 2000), (0.3, 1), (1e-12, 33)):
            ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, ss, min_w)
            ctx.adjoint_set_weights(w)
            ctx.set_algorithm("event", 1)
            ctx.simulate_source(7, n)
            want, cnt = ctx.tally_q(), ctx.counters()
            ctx.set_algorithm("history")
            ctx.adjoint_reset()
            ctx.adjoint_run(7, n, with_gradient=gradient)
            assert np.array_equal(ctx.tally_q(), want)
            got = ctx.counters()
            assert all(got[k] == cnt[k] for k in ("histories", "steps", "scatters"))
            loss, ga, gs = ctx.adjoint_read()
            # float-float sums of products rounded to 24 bits, over at most unit weight
            assert abs(loss - (ctx.tally() * w).sum() / n) <= 2.0 ** -23 * np.abs(w).max()
            assert np.isfinite(ga).all() and np.isfinite(gs).all()
            assert (ga != 0).any() == gradient


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_forward_pass_costs_what_the_tracker_does(mcg, mode):
    """40 thick cells, 5e5 histories, against the tracker on the same chain (by tiles
    the forward pass took four times as long)."""
    m, n = 40, 500_000
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, 0.3 * m), np.full(m, 0.001 * m), 1e-12)
        ctx.adjoint_set_weights(np.ones(m, f32))
        times = []
        for run in (lambda: ctx.simulate_source(0, n), lambda: ctx.adjoint_run(0, n, with_gradient=False)):
            best = []
            for _ in range(4):
                run()
                best.append(ctx.last_kernel_ms())
            times.append(min(best))
    assert times[1] < 2 * times[0], times


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("refill", [1, 3, 200])
def test_refill_steps_of_the_one_kernel(mcg, mode, refill):
    """mcg_set_launch's steps between two looks for new histories: the same sums."""
    m, n = 40, 3000
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, 0.3 * m), np.full(m, 0.3 * m), 1e-12)
        ctx.adjoint_set_weights(np.ones(m, f32))
        out = []
        for steps in (0, refill):
            ctx.set_launch(refill_steps=steps)
            ctx.adjoint_reset()
            ctx.adjoint_run(0, n)
            out.append((ctx.tally_q().tobytes(), ctx.adjoint_read()[0], ctx.counters()))
        assert out[0] == out[1]
