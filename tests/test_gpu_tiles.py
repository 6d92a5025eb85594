"""The tiled tracker (a warp advances each of its histories by a tile of up to
16 or 32 certain crossings) against the event-based tracker, whose single
crossings and full steps are another path of the same arithmetic: per particle
and per cell identical, over chain lengths around the tile sizes, thin and
thick cells, one and several layers of different spacing, and particles inside
and outside their cells, with directions, weights and seeds at the edges of
what the tiles accept.  Results are exact, so nothing is tolerated."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


def _particles(mcg, rng, m, dx, n):
    p = np.zeros(n, mcg.PARTICLE_DTYPE)
    p["seed"] = rng.integers(0, 2 ** 63, n, dtype=np.uint64)
    p["seed"][::17] |= np.uint64(1) << np.uint64(63)
    p["index"] = rng.integers(0, m, n)
    p["x"] = ((p["index"] + rng.random(n)) * dx).astype(f32)
    p["x"][::5] = (p["index"][::5] * dx).astype(f32)            # on the left face
    p["x"][1::11] = ((p["index"][1::11] + 1) * dx).astype(f32)  # on the right face
    p["x"][2::13] = ((p["index"][2::13] - 0.5) * dx).astype(f32)  # outside the cell
    p["mu"] = (2 * rng.random(n) - 1).astype(f32)
    for k, v in enumerate((1.0, -1.0, 0.0, -0.0, 1e-4, -1e-4, 1.1e-4, 1e-3, -0.03, 0.06)):
        p["mu"][k::29] = v
    p["wmc"] = 1.0
    for k, v in enumerate((1e-12, 2e-12, 0.9e-12, 1e-30, 0.3, 1e20, 0.0)):
        p["wmc"][k::23] = v
    p["index"][3::31] = -1
    p["index"][4::37] = m
    return p


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("thin", [False, True])
@pytest.mark.parametrize("m,layers", [(1, 1), (2, 2), (15, 1), (16, 3), (17, 1), (31, 1), (32, 1),
                                      (33, 7), (64, 1), (700, 9)])
def test_tiles_match_event_mode(mcg, mode, thin, m, layers):
    rng = np.random.default_rng(m * 100 + layers)
    st, lm, dx, _, _ = mcg.layer_decomposition(0.0, 1.0, m, layers)
    # optical widths: thin below 2e-4 in sigma_a and 4e-4 in sigma_s; thick from
    # far below to far above the tiles' ranges, some cells empty or scattering only
    if thin:
        sa, ss = 1.9e-4 * m * rng.random(m), 2e-4 * m * rng.random(m)
    else:
        sa, ss = m * 10.0 ** rng.uniform(-5, 0.5, m), m * 10.0 ** rng.uniform(-5, 0, m)
    sa[::7], ss[3::8] = 0.0, 5e-5
    sigs = (sa + ss).astype(f32)
    rates = np.where(sigs > 0, sa / np.where(sigs > 0, sigs, 1), 0).astype(f32)
    with mcg.Context(mode=mode) as ctx:
        for min_w, scale, n, launch in ((1e-12, 40, 2500, {}), (0.3, 35, 33, {}), (0.0, 20, 1, {}),
                                        (-np.inf, 35, 400, dict(block=1024, refill_steps=3)),
                                        (1e-12, 44, 999, dict(block=64, blocks_per_sm=1))):
            ctx.set_layers(st, lm, dx, sigs, rates, min_w)
            ctx.set_tally_scale(scale)
            ctx.set_launch(**launch)
            p = _particles(mcg, rng, m, 1.0 / m, n)
            out = []
            for algorithm in ("history", "event"):
                ctx.set_algorithm(algorithm, 1)
                ctx.tally_reset()
                q = p.copy()
                r = ctx.simulate(q)
                out.append((q, r, ctx.tally_q(), ctx.counters()))
            (pa, ra, qa, ca), (pb, rb, qb, cb) = out
            assert pa.tobytes() == pb.tobytes()
            for key in ("results", "steps", "scatters"):
                assert np.array_equal(ra[key], rb[key]), key
            assert np.array_equal(qa, qb)
            assert ca == cb


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("sizes", [(1, 40), (15, 700), (20_000, 25_000)])
def test_batch_items_match_event_mode(mcg, mode, sizes):
    """Work items down to one history, so that blocks change slabs while their
    warps keep histories of earlier ones (whose deposits then go to the global
    tally), in every tally mode and block size: the event-based form's tallies
    and counters.  The largest slabs are beyond the shared-memory tally."""
    rng = np.random.default_rng(sizes[1])
    n_slabs = 60 if sizes[1] < 1000 else 3
    cells = rng.integers(sizes[0], sizes[1] + 1, n_slabs)
    total = int(cells.sum())
    sa = np.repeat(10.0 ** rng.uniform(-2, 1, n_slabs), cells) * rng.random(total)
    ss = np.repeat(10.0 ** rng.uniform(-2, 1.3, n_slabs), cells) * rng.random(total)
    sigs = (sa + ss).astype(f32)
    rates = (sa / np.maximum(sa + ss, 1e-30)).astype(f32)
    slabs = [dict(n_cells=int(cells[s]), n_histories=int(rng.integers(0, 300)), base_seed=17 + s,
                  seed_mode=s % 2, isotropic=s % 3, mu0=1.0, w0=1.0) for s in range(n_slabs)]
    with mcg.Context(mode=mode) as ctx:
        ctx.batch_set(slabs, sigs, rates, 1e-12)
        ctx.batch_set_algorithm("event", 2)
        ctx.batch_run()
        want, counters = ctx.batch_tally_q(), ctx.counters()
        ctx.batch_set_algorithm("history")
        for block, item, tally, defer in ((256, 1, 1, 0), (512, 7, 0, 1), (1024, 64, 2, 32),
                                          (1024, 1 << 20, 1, 4)):
            ctx.batch_set_launch(block, item, tally)
            ctx.batch_set_deferral(defer)
            ctx.batch_tally_reset()
            ctx.batch_run()
            assert np.array_equal(ctx.batch_tally_q(), want), (block, item, tally)
            assert ctx.counters() == counters


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,layers,width,n", [
    (1, 1, 0.5, 5), (7, 7, 3.0, 2000), (20, 20, 1e-3, 120_000), (33, 2, 0.2, 700),
    (700, 16, 1e-2, 5000), (3000, 5, 1.5e-4, 300), (16_000, 64, 1e-4, 300), (30_000, 3, 1e-4, 40)])
def test_async_workers_match_event_mode(mcg, mode, m, layers, width, n):
    """Sub-domains from one cell up, thin and thick chains (width: the largest
    optical width of a cell), fewer histories than a warp has lanes and more than
    the grid has, and chains beyond each form of the shared-memory tally."""
    rng = np.random.default_rng(m)
    st, lm, dx, _, _ = mcg.layer_decomposition(0.0, 1.0, m, layers)
    sa, ss = rng.uniform(0.1, width * m / 2, (2, m)) if width * m > 0.4 else np.full((2, m), 0.1)
    sigs = (sa + ss).astype(f32)
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers(st, lm, dx, sigs, (sa / sigs).astype(f32), 1e-12)
        ctx.set_algorithm("event", 1)
        ctx.simulate_source(0, n)
        want, c = ctx.tally_q(), ctx.counters()
        ctx.tally_reset()
        ctx.worker_run_async(n)
        assert np.array_equal(ctx.tally_q(), want)
        got = ctx.counters()
        assert all(got[k] == c[k] for k in ("histories", "steps", "scatters"))


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,layers,width", [(1, 1, 2.0), (16, 1, 0.3), (40, 3, 0.021), (40, 3, 0.019),
                                            (300, 2, 0.1), (5000, 1, 1.0), (27_000, 1, 0.5)])
def test_thick_chains_match_event_mode(mcg, mode, m, layers, width):
    """Chains of thick cells run a lane per history (width: every cell's optical
    width, on both sides of the rule's line and beyond the shared tally): host
    particles and born ones, the weight cut-off and the tally modes."""
    rng = np.random.default_rng(m)
    st, lm, dx, _, _ = mcg.layer_decomposition(0.0, 1.0, m, layers)
    sigs = np.full(m, 2 * width * m, f32)
    rates = np.full(m, 0.5, f32)
    with mcg.Context(mode=mode) as ctx:
        for min_w, tally, launch in ((1e-12, 0, {}), (0.2, 1, dict(block=128)),
                                     (1e-12, 2, dict(block=1024, blocks_per_sm=1))):
            ctx.set_layers(st, lm, dx, sigs, rates, min_w)
            ctx.set_tally_mode(tally)
            ctx.set_launch(**launch)
            p = _particles(mcg, rng, m, 1.0 / m, 700)
            out = []
            for algorithm in ("history", "event"):
                ctx.set_algorithm(algorithm, 1)
                ctx.tally_reset()
                q = p.copy()
                r = ctx.simulate(q)
                ctx.simulate_source(3, 1500)
                out.append((q, r, ctx.tally_q(), ctx.counters()))
            (pa, ra, qa, ca), (pb, rb, qb, cb) = out
            assert pa.tobytes() == pb.tobytes()
            for key in ("results", "steps", "scatters"):
                assert np.array_equal(ra[key], rb[key]), key
            assert np.array_equal(qa, qb)
            assert ca == cb
