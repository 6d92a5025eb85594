"""Batches in which some slabs take a lane per history and others tiles: two
kernels side by side, or one of them alone.  The event-based form gives the same
sums by another path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


def _slabs(rng, cells, widths, histories):
    """widths: optical widths (sig_a, sig_s) of a slab's cells, on average."""
    per = np.repeat(cells, cells)
    sa, ss = (np.repeat([w[k] for w in widths], cells) * per * rng.uniform(0.3, 1.7, per.size) for k in (0, 1))
    sa[::13] = 0.0
    ss[5::17] = 0.0
    sigs = (sa + ss).astype(f32)
    rates = np.where(sigs > 0, sa / np.where(sigs > 0, sigs, 1), 0).astype(f32)
    slabs = [dict(n_cells=int(m), n_histories=int(n), base_seed=17 + 3 * s, seed_mode=s % 2, isotropic=s % 3,
                  mu0=1.0, w0=1.0) for s, (m, n) in enumerate(zip(cells, histories))]
    return slabs, sigs, rates


CASES = {
    # both kernels: slabs on either side of the lines of length and width
    "mixed": ([1, 99, 100, 101, 102, 300, 300, 300, 700, 16], [(.01, .01)] * 5 + [(.2, .2), (.01, .6), (.005, .005)] +
              [(.01, .01), (1, 1)], [3000, 500, 900, 200, 700, 300, 64, 100, 150, 5000]),
    "lanes alone": ([1, 2, 3, 31, 64, 40, 7], [(1e-5, 1e-5), (.5, 1e-3), (.1, .1), (3, 1), (.3, .3), (0, .5), (.02, 2)],
                    [1, 31, 513, 2000, 100, 0, 300]),
    "tiles alone": ([200, 333], [(.01, .01), (1e-4, 1e-4)], [300, 77]),
    # a tenth of the work in short slabs: by tiles with the others
    "few short ones": ([30, 30, 2000], [(.1, .1), (.01, .01), (1e-3, 1e-3)], [100, 100, 500]),
    # thick slabs beyond the shared-memory tally of the other kernel
    "long and thick": ([28_000, 20, 25_000], [(.3, .01), (.5, .5), (.2, .3)], [200, 3000, 100]),
}


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("name", CASES)
def test_mixed_batches_match_event_mode(mcg, mode, name):
    rng = np.random.default_rng(len(name))
    slabs, sigs, rates = _slabs(rng, *CASES[name])
    with mcg.Context(mode=mode) as ctx:
        for min_w, limit in ((1e-12, 1 << 28), (0.3, 1 << 28), (1e-12, 9)):
            mcg._check(ctx.lib.mcg_set_step_limit(ctx.h, limit))
            ctx.batch_set(slabs, sigs, rates, min_w)
            want = None
            for algorithm, block, item, tally in (("event", 256, 64, 1), ("history", 256, 1, 1),
                                                  ("history", 1024, 1 << 16, 0), ("history", 512, 700, 2)):
                ctx.batch_set_algorithm(algorithm, 2)
                ctx.batch_set_launch(block, item, tally)
                ctx.batch_tally_reset()
                for again in range(2 if limit > 9 else 1):  # the graph, then its replay
                    try:
                        ctx.batch_run()
                    except mcg.MCGError as e:
                        assert e.code == 7 and limit == 9  # MCG_ERR_LIMIT
                got = (ctx.batch_tally_q(), ctx.counters())
                if want is None:
                    want = got
                else:
                    assert np.array_equal(got[0], want[0]), (min_w, block, item, tally)
                    assert got[1] == want[1]
            if limit > 9:
                ctx.batch_tally_reset()
                ctx.batch_run_per_slab()
                assert np.array_equal(2 * ctx.batch_tally_q(), want[0])


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_autotuned_mixed_batch(mcg, mode):
    rng = np.random.default_rng(1)
    cells = rng.integers(2, 220, 40)
    slabs, sigs, rates = _slabs(rng, cells, [(.02, .05)] * 40, rng.integers(200, 3000, 40))
    with mcg.Context(mode=mode) as ctx:
        ctx.batch_set(slabs, sigs, rates, 1e-12)
        ctx.batch_set_algorithm("event", 4)
        ctx.batch_run()
        want = ctx.batch_tally_q()
        ctx.batch_set_algorithm("history")
        ctx.batch_autotune(0.5)
        ctx.batch_set_algorithm("history")
        ctx.batch_tally_reset()
        ctx.batch_run()
        assert np.array_equal(ctx.batch_tally_q(), want)


@pytest.mark.parametrize("mode,bound", [("strict", 2.0), ("fast", 2.0)])
@pytest.mark.parametrize("width", [1e-4, 0.3])
def test_short_slabs_cost_what_short_chains_do(mcg, mode, bound, width):
    """Time per step of 2000 short slabs against one chain of such cells and as many
    histories (by tiles they took three to eight times as long)."""
    m, n, slabs = 40, 2000, 2000
    sa = np.full(m, width * m, f32)
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, sa, 1e-12)
        chain = []
        for _ in range(4):
            ctx.simulate_source(0, n * slabs)
            chain.append(ctx.last_kernel_ms())
        ctx.batch_set([dict(n_cells=m, n_histories=n, base_seed=5 + s, seed_mode=0, isotropic=0, mu0=1.0, w0=1.0)
                       for s in range(slabs)], np.tile(2 * sa, slabs), np.full(m * slabs, 0.5, f32), 1e-12)
        batch = []
        for _ in range(4):
            ctx.batch_run()
            batch.append(ctx.last_kernel_ms())
    assert min(batch) < bound * min(chain), (min(batch), min(chain))
