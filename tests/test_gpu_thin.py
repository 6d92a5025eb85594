"""Thin chains, whose tiles test a whole flight against the chain's widest cell,
where the cells are not alike: cells whose steps the tiles must leave to the
full step (negative absorption, faces that do not fit between layers), and cells
that are wider when entered from a neighbouring layer than between their own
faces.  The event-based tracker, which has neither tiles nor bounds per flight,
gives the same arithmetic by another path; results are exact."""
import numpy as np
import pytest

from test_gpu_tiles import _particles

pytestmark = pytest.mark.gpu
f32 = np.float32


def _entry_widths(st, m, dx):
    """Length of the flight that enters each cell by its left and right face, over
    the cell's own, as the tracker forms them (float32 faces index * dx)."""
    lo, hi = [np.concatenate([(np.arange(s + k, s + k + n).astype(f32) * f32(d)) for s, n, d in
                              zip(st, m, dx)]) for k in (0, 1)]
    left, right = hi.copy(), -lo
    left[1:] -= hi[:-1]
    left[0] -= lo[0]
    right[:-1] += lo[1:]
    right[-1] += hi[-1]
    return left / (hi - lo), right / (hi - lo)


def _same_as_event_mode(ctx, n, **source):
    """In the launch shape of the library's choice, and with a block size that
    makes a thin chain take the thin form whether it pays or not."""
    out = []
    for algorithm, launch in (("event", {}), ("history", {}), ("history", dict(block=768))):
        ctx.set_algorithm(algorithm, 1)
        ctx.set_launch(**launch)
        ctx.tally_reset()
        ctx.simulate_source(0, n, **source)
        out.append((ctx.tally_q(), ctx.counters()))
    ctx.set_launch()
    for q, c in out[1:]:
        assert np.array_equal(out[0][0], q)
        assert out[0][1] == c
    ctx.tally_reset()
    ctx.worker_run_async(n, **source)
    assert np.array_equal(out[0][0], ctx.tally_q())
    return out[0]


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,sign", [(64, -1), (700, -1), (3000, -1), (700, 1)])
def test_cells_without_a_tile_length(mcg, mode, m, sign):
    """Every 37th cell amplifies the weight, or (sign 1) has no length at all
    because its layer starts where the previous one's cells already are."""
    rng = np.random.default_rng(m)
    sa, ss = rng.uniform(0.2, 1.0, (2, m)) * 1.5e-4 * m
    if sign < 0:
        st, lm, dx = [0], [m], [f32(1.0 / m)]
        sa[5::37] *= -1
    else:
        # layers of 37 cells, each a little finer than the one before: the first
        # face of a layer lies before the last face of the previous one
        st = np.arange(0, m, 37)
        lm = np.minimum(37, m - st)
        dx = (1.0 / m) * np.cumprod(np.concatenate([[1.0], 1 - 1.25 / st[1:]]))
        left, _ = _entry_widths(st, lm, dx)
        assert (left <= 0).sum() >= len(st) // 2
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs(st, lm, dx, sa, ss, 1e-12)
        q, c = _same_as_event_mode(ctx, 3000)
        assert c["histories"] == 3000
        if sign < 0:
            assert (q < 0).sum() == (sa < 0).sum()


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_fine_decomposition(mcg, mode):
    """1000 sub-domains of 20 cells, as the library decomposes the slab: the
    layers' float32 faces do not meet, and some cells have no length."""
    m, layers = 20_000, 1000
    st, lm, dx, _, _ = mcg.layer_decomposition(0.0, 1.0, m, layers)
    left, right = _entry_widths(st, lm, dx)
    assert min(left.min(), right.min()) <= 0
    rng = np.random.default_rng(3)
    sa, ss = rng.uniform(0.2, 1.0, (2, m)) * 1e-4 * m
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs(st, lm, dx, sa, ss, 1e-12)
        _same_as_event_mode(ctx, 2000)


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("gap", [0.5, 3.0])
def test_cells_wider_from_the_next_layer(mcg, mode, gap):
    """50 layers, each a little coarser than the one before, so that a layer
    starts `gap` cells after the previous one ends: those cells are entered from
    farther away than they are wide, in both directions."""
    m, k = 1000, 20
    st = np.arange(0, m, k)
    dx = (1.0 / m) * np.cumprod(np.concatenate([[1.0], 1 + gap / st[1:]]))
    left, right = _entry_widths(st, np.full(m // k, k), dx)
    assert min((w > 1 + 0.9 * gap).sum() for w in (left, right)) >= m // k - 3
    wide = dx.repeat(k)
    # strict thin chains may scatter strongly, fast ones are thin in both
    wa, ws = (1e-4, 2e-2) if mode == "strict" else (3e-4, 3e-4)
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs(st, np.full(m // k, k), dx, wa / wide, ws / wide, 1e-12)
        _same_as_event_mode(ctx, 2000 if mode == "strict" else 400_000)


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_uniform_decomposed_slab(mcg, mode):
    """12,000 equal cells in 64 sub-domains: a few per cent wider at some of the
    sub-domains' ends."""
    m = 12_000
    st, lm, dx, _, _ = mcg.layer_decomposition(0.0, 1.0, m, 64)
    left, right = _entry_widths(st, lm, dx)
    assert max(left.max(), right.max()) > 1.02
    wa, ws = (5e-5, 2e-3) if mode == "strict" else (5e-5, 3.9e-4)
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs(st, lm, dx, np.full(m, wa * m), np.full(m, ws * m), 1e-12)
        _same_as_event_mode(ctx, 20_000)


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_thick_cells_with_short_entries(mcg, mode):
    """Layers of one cell whose right faces coincide: no flight to the right has a
    length, and those to the left are 1 / g of the cells' own width, so that the
    chain is thin by the tiles' lengths and thick by its cells."""
    m = 1000
    g = np.arange(m)
    dx = 1.0 / (g + 1)
    left, right = _entry_widths(g, np.ones(m, int), dx)
    assert np.abs(left[1:]).max() < 1e-3 and np.median(right) < 1e-2
    sa = 1e-4 * (g + 1) * (g + 2)
    sa[0] = sa[-1] = 0.0
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs(g, np.ones(m, int), dx, sa, 0.9 * sa, 1e-12)
        p = _particles(mcg, np.random.default_rng(1), m, 1.0, 1500)
        p["x"] = ((p["index"] + 0.5) * dx[np.clip(p["index"], 0, m - 1)]).astype(f32)
        out = []
        for algorithm in ("event", "history"):
            ctx.set_algorithm(algorithm, 1)
            ctx.tally_reset()
            q = p.copy()
            ctx.simulate(q)
            out.append((q.tobytes(), ctx.tally_q().tobytes(), ctx.counters()))
        assert out[0] == out[1]
        _same_as_event_mode(ctx, 3000)


def _kernel_ms(ctx, n, **source):
    times = []
    for _ in range(4):
        ctx.simulate_source(0, n, **source)
        times.append(ctx.last_kernel_ms())
    return min(times)


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("scale,w0", [(40, 30.0), (40, 1e6), (50, 1.0), (58, 1.0), (62, 1e-3), (62, 1.0), (0, 1e18)])
def test_large_deposits(mcg, mode, scale, w0):
    """Deposits around and above the 31 bits of a low word, up to beyond the 62
    that the tiles take (sums wrap alike)."""
    rng = np.random.default_rng(9)
    m = 1000
    sa, ss = rng.uniform(0.2, 1.0, (2, m)) * 1.5e-4 * m
    sa[::9] = 0.0
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, ss, 1e-12)
        ctx.set_tally_scale(scale)
        _same_as_event_mode(ctx, 3000, w0=w0)


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_large_deposits_stay_in_the_tiles(mcg, mode):
    """The same histories with a weight of 1000 and of 1, born or as particles: a
    full step for every crossing takes 40 times as long, the form with wider
    deposits two to three times."""
    m, n = 10_000, 20_000
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, 5e-5 * m), np.full(m, 2e-4 * m), 1e-12)
        assert _kernel_ms(ctx, n, w0=1000.0) < 8 * _kernel_ms(ctx, n)
        p = np.zeros(n, mcg.PARTICLE_DTYPE)
        p["seed"] = np.arange(1, n + 1, dtype=np.uint64) * np.uint64(7919 * 10 ** 9)
        p["mu"] = 1.0
        times = []
        for w in (1.0, 1000.0):
            p["wmc"] = w
            best = []
            for _ in range(3):
                ctx.simulate(p.copy())
                best.append(ctx.last_kernel_ms())
            times.append(min(best))
        assert times[1] < 8 * times[0]


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("heavy", [False, True])
@pytest.mark.parametrize("m", [1, 31, 33, 700])
def test_thin_particles(mcg, mode, heavy, m):
    """Host particles on both sides of the line between the two forms, which is
    drawn on the device from their weights: one heavy particle decides."""
    rng = np.random.default_rng(m)
    sa, ss = rng.uniform(0.2, 1.0, (2, m)) * 1.5e-4 * m
    p = _particles(mcg, rng, m, 1.0 / m, 2500)
    p["wmc"] = np.minimum(p["wmc"], 1.0)
    if heavy:
        p["wmc"][1234] = -1e9 if m == 31 else np.nan if m == 33 else 1e9
    with mcg.Context(mode=mode) as ctx:
        for min_w, scale in ((1e-12, 40), (-np.inf, 35), (0.3, 30)):
            ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, ss, min_w)
            ctx.set_tally_scale(scale)
            out = []
            for algorithm, launch in (("event", {}), ("history", {}), ("history", dict(block=512))):
                ctx.set_algorithm(algorithm, 1)
                ctx.set_launch(**launch)
                ctx.tally_reset()
                q = p.copy()
                r = ctx.simulate(q)
                out.append((q, r, ctx.tally_q(), ctx.counters()))
            pa, ra, qa, ca = out[0]
            for pb, rb, qb, cb in out[1:]:
                assert pa.tobytes() == pb.tobytes()
                for key in ("results", "steps", "scatters"):
                    assert np.array_equal(ra[key], rb[key]), key
                assert np.array_equal(qa, qb)
                assert ca == cb


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m", [1, 16, 64, 300])
def test_short_chains_are_not_slower_for_being_thin(mcg, mode, m):
    """Two million histories through chains of almost nothing, on which the thin
    form's one block per SM took twice as long as cells of width 5e-3 do."""
    times = []
    with mcg.Context(mode=mode) as ctx:
        for width in (1e-7, 5e-3):
            ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, width * m), np.full(m, width * m), 1e-12)
            times.append(_kernel_ms(ctx, 2_000_000 if m < 64 else 500_000))
    assert times[0] < 1.25 * times[1], times
