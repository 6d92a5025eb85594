"""The asynchronous workers' two forms, tiles and a lane per particle, on both sides of
the rule's lines: sub-domains of few cells, thick cells, and many histories that
stream through a short chain.  Event mode gives the same sums by another path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,layers,wa,ws,n", [
    (30, 1, .3, .3, 3000), (30, 1, .029, .01, 3000), (30, 1, .032, .01, 3000), (300, 4, .01, .3, 2000),
    (300, 4, .01, .2, 2000), (400, 4, .1, .01, 2000), (400, 4, .08, .01, 2000), (16_000, 64, .1, .01, 500),
    (28_000, 3, .3, .01, 200), (60, 2, 1e-5, 1e-5, 70_000), (60, 2, .0019, .0019, 70_000),
    (100, 2, .0021, .0021, 70_000), (101, 2, .001, .001, 70_000), (499, 3, 5e-5, 5e-5, 66_000),
    (500, 3, 5e-5, 5e-5, 66_000), (300, 10, 5e-5, 5e-5, 65_535), (48, 2, 1e-3, 1e-3, 400)])
def test_async_forms_match_event_mode(mcg, mode, m, layers, wa, ws, n):
    rng = np.random.default_rng(m + layers)
    st, lm, dx, _, _ = mcg.layer_decomposition(0.0, 1.0, m, layers)
    sa, ss = (wa * m * rng.uniform(0.9, 1.1, m)).astype(f32), (ws * m * rng.uniform(0.9, 1.1, m)).astype(f32)
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs(st, lm, dx, sa, ss, 1e-12)
        ctx.set_algorithm("event", 1)
        ctx.simulate_source(0, n)
        want, c = ctx.tally_q(), ctx.counters()
        ctx.set_algorithm("history")
        ctx.tally_reset()
        ctx.worker_run_async(n)
        assert np.array_equal(ctx.tally_q(), want)
        got = ctx.counters()
        assert all(got[k] == c[k] for k in ("histories", "steps", "scatters"))


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_thick_sub_domains_cost_what_the_tracker_does(mcg, mode):
    """30 cells of width .3 that hardly scatter, 5e5 histories, against the tracker (by
    tiles the workers took five times as long as by lanes)."""
    m, n = 30, 500_000
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, 0.3 * m), np.full(m, 0.001 * m), 1e-12)
        times = []
        for run in (lambda: ctx.simulate_source(0, n), lambda: ctx.worker_run_async(n)):
            best = []
            for _ in range(5):
                run()
                best.append(ctx.last_kernel_ms())
            times.append(min(best))
    assert times[1] < 4 * times[0], times
