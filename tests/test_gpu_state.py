"""Settings and state that outlive one call: what a context keeps between runs
must follow its setters, and contexts must not disturb one another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


def _batch(n_slabs=12, low=10, high=200, histories=500, seed=3):
    rng = np.random.default_rng(seed)
    cells = rng.integers(low, high + 1, n_slabs)
    total = int(cells.sum())
    slabs = [dict(n_cells=int(k), n_histories=histories, base_seed=31 + s, seed_mode=s % 2,
                  isotropic=s % 3, mu0=1.0, w0=1.0) for s, k in enumerate(cells)]
    return slabs, rng.uniform(0.5, 5, total).astype(f32), rng.uniform(0.1, 0.9, total).astype(f32)


@pytest.mark.parametrize("first", ["strict", "fast"])
def test_batch_follows_settings_made_after_its_first_run(mcg, first):
    """The captured graph holds the arithmetic, the tally scale, the step limit
    and the tile window by value: after each setter a run gives what a fresh
    context with those settings gives."""
    slabs, sigs, rates = _batch()
    other = {"strict": "fast", "fast": "strict"}[first]

    def fresh(mode, scale, limit):
        with mcg.Context(mode=mode) as c:
            c.set_tally_scale(scale)
            mcg._check(c.lib.mcg_set_step_limit(c.h, limit))
            c.batch_set(slabs, sigs, rates, 1e-12)
            try:
                c.batch_run()
                code = 0
            except mcg.MCGError as e:
                code = e.code
            return c.batch_tally_q(), c.counters()["steps"], code

    with mcg.Context(mode=first) as c:
        c.batch_set(slabs, sigs, rates, 1e-12)
        c.batch_run()
        for mode, scale, limit, window in ((first, 33, 1 << 28, 0), (other, 33, 1 << 28, 5),
                                           (other, 33, 40, 5), (first, 40, 1 << 28, 0)):
            c.set_mode(mode)
            c.set_tally_scale(scale)
            mcg._check(c.lib.mcg_set_step_limit(c.h, limit))
            c.set_launch(refill_steps=window)
            c.batch_tally_reset()
            try:
                c.batch_run()
                code = 0
            except mcg.MCGError as e:
                code = e.code
            q, steps, want = fresh(mode, scale, limit)
            assert np.array_equal(c.batch_tally_q(), q)
            assert (c.counters()["steps"], code) == (steps, want)
            assert (code != 0) == (limit == 40)


@pytest.mark.parametrize("kind", ["batch", "per_slab", "adjoint", "fit", "event"])
def test_contexts_of_two_threads_do_not_lower_each_others_shared_memory(mcg, kind):
    """A launch's limit of shared memory belongs to the kernel, not to the
    context: one host thread runs small problems while another runs large ones of
    the same kernels.  A lowered limit is a failed launch (an error code)."""
    def runner(m, n):
        c = mcg.Context(mode="fast")
        sa = np.full(m, 0.002 * m, f32)
        slabs = [dict(n_cells=m, n_histories=n, base_seed=5, seed_mode=0, isotropic=0, mu0=1.0, w0=1.0)]
        if kind in ("batch", "per_slab"):
            c.batch_set(slabs, 2 * sa, np.full(m, 0.5, f32), 1e-12)

            def run():
                if kind == "per_slab":
                    c.batch_run_per_slab()
                    return
                c.batch_set_launch(block=512)  # configured and captured anew
                c.batch_run()
        elif kind == "fit":
            c.fit_set(slabs, sa, sa, np.zeros(m), max_steps=1)

            def run():
                c.fit_gradient(np.ones(m))
        else:
            c.set_layers_xs([0], [m], [f32(1.0 / m)], sa, sa, 1e-12)
            if kind == "event":
                c.set_algorithm("event", 4)

                def run():
                    c.simulate_source(0, n)
            else:
                c.adjoint_set_weights(np.ones(m, f32))

                def run():
                    c.adjoint_run(0, n)
        return c, run

    failed = []

    def loop(run, times):
        try:
            for _ in range(times):
                run()
        except mcg.MCGError as e:
            failed.append(str(e))

    (a, small), (b, large) = runner(300, 20), runner(10_000, 20)
    try:
        times = 100 if kind == "event" else 400
        threads = [threading.Thread(target=loop, args=(f, times)) for f in (small, large)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        a.close()
        b.close()
    assert not failed


@pytest.mark.parametrize("width", [1e-4, 3e-4, 4.9e-4, 5.1e-4, 2e-3])
def test_synchronous_workers_around_the_thin_step(mcg, width):
    """Strict workers' cycles on both sides of the line of the thin-cell step
    (5e-4) and of the tiles' lower one, against event mode."""
    m, layers, n = 1000, 8, 3000
    rng = np.random.default_rng(4)
    st, lm, dx, _, _ = mcg.layer_decomposition(0.0, 1.0, m, layers)
    sa, ss = rng.uniform(0.3, 1.0, (2, m)) * width * m
    sa[500] = width * m
    with mcg.Context(mode="strict") as ctx:
        ctx.set_layers_xs(st, lm, dx, sa, ss, 1e-12)
        ctx.set_algorithm("event", 1)
        ctx.simulate_source(0, n)
        want, c = ctx.tally_q(), ctx.counters()
        ctx.set_algorithm("history")
        ctx.tally_reset()
        ctx.worker_run(n, per_cycle=500)
        assert np.array_equal(ctx.tally_q(), want)
        assert all(ctx.counters()[k] == c[k] for k in ("steps", "scatters"))


@pytest.mark.parametrize("xs", [False, True])
def test_memory_and_time_of_a_long_chain(mcg, xs):
    """A chain that is never thin keeps 56 bytes per cell (cells of both arithmetics,
    tile table, tally), not the thin tables' 16 more; and its cross sections given
    directly do not cost a second upload."""
    import time
    import torch
    m = 2_000_000
    a, b = np.full(m, 0.01 * m, f32), np.full(m, 0.5, f32)
    with mcg.Context(mode="fast") as ctx:
        ctx.set_layers([0], [10], [f32(0.1)], np.ones(10), np.full(10, 0.5), 1e-12)
        free = torch.cuda.mem_get_info()[0]
        (ctx.set_layers_xs if xs else ctx.set_layers)([0], [m], [f32(1.0 / m)], a, b, 1e-12)
        assert free - torch.cuda.mem_get_info()[0] < 60 * m + (16 << 20)
        times = []
        for f in (ctx.set_layers, ctx.set_layers_xs):
            best = []
            for _ in range(4):
                t = time.perf_counter()
                f([0], [m], [f32(1.0 / m)], a, b, 1e-12)
                best.append(time.perf_counter() - t)
            times.append(min(best))
        assert times[1] < 1.5 * times[0], times


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_chains_of_one_length_with_and_without_thin_tables(mcg, mode):
    """The buffers are kept for as many cells; the thin tables come with the first
    chain that may use them, and are that chain's own each time."""
    m = 6000
    with mcg.Context(mode=mode) as ctx:
        for width in (0.01, 2e-5, 0.03, 5e-5, 5e-5, 0.005):
            sa, ss = np.full(m, width * m), np.full(m, 0.7 * width * m)
            if width == 5e-5:
                sa[::2] = 0.0
            ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, ss, 1e-12)
            out = []
            for algorithm in ("event", "history"):
                ctx.set_algorithm(algorithm, 1)
                ctx.tally_reset()
                ctx.simulate_source(0, 300)
                out.append((ctx.tally_q().tobytes(), ctx.counters()))
            assert out[0] == out[1]


def test_chain_longer_than_the_thin_kernel_holds(mcg):
    """100,000 thin cells: no thin tables, the other tiles."""
    m = 100_000
    with mcg.Context(mode="strict") as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, 1.0), np.full(m, 2.0), 1e-12)
        out = []
        for algorithm in ("event", "history"):
            ctx.set_algorithm(algorithm, 1)
            ctx.tally_reset()
            ctx.simulate_source(0, 100)
            out.append((ctx.tally_q().tobytes(), ctx.counters()))
        assert out[0] == out[1]


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_small_refill_steps_are_not_a_tile_each(mcg, mode):
    """A caller's refill_steps of 1 or 4 took six and two times as long as 8, a tile's
    fixed costs for as many steps."""
    m = 1000
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, 2.0), np.full(m, 2.0), 1e-12)
        times = {}
        for steps in (8, 4, 1):
            ctx.set_launch(refill_steps=steps)
            best = []
            for _ in range(4):
                ctx.simulate_source(0, 300_000)
                best.append(ctx.last_kernel_ms())
            times[steps] = min(best)
        assert max(times[1], times[4]) < 1.3 * times[8], times


@pytest.mark.parametrize("kept", [False, True])
def test_failed_thin_tables_leave_no_geometry(mcg, kept):
    """The thin tables' allocation fails: with buffers of the same chain length kept,
    where it is the only one, or after four others."""
    m = 300
    thin = ([0], [m], [f32(1.0 / m)], np.full(m, 1e-5 * m), np.full(m, 1e-5 * m), 1e-12)
    with mcg.Context(mode="fast") as ctx:
        n = m if kept else m + 1
        ctx.set_layers_xs([0], [n], [f32(1.0 / n)], np.full(n, 0.01 * n), np.full(n, 0.01 * n), 1e-12)
        ctx.lib.mcg_testing_fail_allocation(0 if kept else 4)
        try:
            with pytest.raises(mcg.MCGError) as e:
                ctx.set_layers_xs(*thin)
            assert e.value.code == 2  # MCG_ERR_CUDA
        finally:
            ctx.lib.mcg_testing_fail_allocation(-1)
        with pytest.raises(mcg.MCGError) as e:
            ctx.simulate_source(0, 10)
        assert e.value.code == 5  # MCG_ERR_STATE
        ctx.set_layers_xs(*thin)
        ctx.simulate_source(0, 1000)
        assert ctx.counters()["histories"] == 1000
