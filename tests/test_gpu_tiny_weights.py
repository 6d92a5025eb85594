"""Weights far below one, down to the subnormal numbers where a deposit rounds to
nothing: runs without a minimum weight carry their histories on until they leave.
The event-based tracker gives the same arithmetic by another path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


def _chain(m, wa, ws, seed=0):
    rng = np.random.default_rng(seed)
    sa, ss = (wa * m * rng.uniform(0.2, 1.0, m)).astype(f32), (ws * m * rng.uniform(0.2, 1.0, m)).astype(f32)
    sa[7::11] = 0.0
    return [0], [m], [f32(1.0 / m)], sa, ss


def _particles(mcg, m, n):
    rng = np.random.default_rng(n)
    p = np.zeros(n, mcg.PARTICLE_DTYPE)
    p["seed"] = rng.integers(0, 2 ** 63, n, dtype=np.uint64)
    p["index"] = rng.integers(0, m, n)
    p["x"] = ((p["index"] + 0.5) / m).astype(f32)
    p["mu"] = (2 * rng.random(n) - 1).astype(f32)
    # from normal numbers through the line of 2^-60 to zero, of both signs
    p["wmc"] = np.where(rng.random(n) < 0.8, 1, -1) * 2.0 ** rng.uniform(-152, 3, n)
    p["wmc"][::41] = 0.0
    p["wmc"][1::43] = 2.0 ** -60
    p["wmc"][2::47] = np.nextafter(f32(2.0 ** -60), f32(0))
    p["wmc"][3::53] = -(2.0 ** -60)
    return p


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,wa,ws", [(40, 0.015, 0.1), (900, 0.015, 0.002), (900, 0.05, 0.001), (1500, 1e-4, 1e-4)])
def test_tiny_weights_match_event_mode(mcg, mode, m, wa, ws):
    with mcg.Context(mode=mode) as ctx:
        for min_w, scale in ((-np.inf, 40), (0.0, 58), (0.0, 59), (-1e-25, 35), (1e-30, 35), (1e-41, 40), (-1.0, 62)):
            ctx.set_layers_xs(*_chain(m, wa, ws), min_w)
            ctx.set_tally_scale(scale)
            p = _particles(mcg, m, 1500)
            out = []
            for algorithm in ("history", "event"):
                ctx.set_algorithm(algorithm, 1)
                ctx.tally_reset()
                q = p.copy()
                r = ctx.simulate(q)
                ctx.simulate_source(5, 300)
                out.append((q, r, ctx.tally_q(), ctx.counters()))
            (pa, ra, qa, ca), (pb, rb, qb, cb) = out
            assert pa.tobytes() == pb.tobytes()
            for key in ("results", "steps", "scatters"):
                assert np.array_equal(ra[key], rb[key]), key
            assert np.array_equal(qa, qb)
            assert ca == cb


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_batch_and_loss_without_a_minimum_weight(mcg, mode):
    """A deep slab as one of a batch, and under the adjoint's forward pass, whose
    loss is the sum of the deposits' products."""
    m, n = 900, 400
    geo = _chain(m, 0.015, 0.002)
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs(*geo, 0.0)
        ctx.set_algorithm("event", 1)
        ctx.simulate_source(0, n)
        want = ctx.tally_q()
        w = np.random.default_rng(2).standard_normal(m).astype(f32)
        ctx.tally_reset()
        ctx.adjoint_set_weights(w)
        ctx.adjoint_run(0, n)
        assert np.array_equal(ctx.tally_q(), want)
        loss, ga, gs = ctx.adjoint_read()
        # float-float sums of products rounded to 24 bits, over at most unit weight
        assert abs(loss - (ctx.tally() * w).sum() / n) <= 2.0 ** -23 * np.abs(w).max()
        assert np.isfinite(ga).all() and np.isfinite(gs).all()
        slab = dict(n_cells=m, n_histories=n, base_seed=5127801, seed_mode=0, isotropic=0, mu0=1.0, w0=1.0)
        sigs = (geo[3] + geo[4]).astype(f32)
        ctx.batch_set([slab, slab], np.tile(sigs, 2), np.tile((geo[3] / sigs).astype(f32), 2), 0.0)
        ctx.batch_set_algorithm("event", 1)
        ctx.batch_run()
        want = ctx.batch_tally_q()
        ctx.batch_set_algorithm("history")
        ctx.batch_tally_reset()
        ctx.batch_run()
        assert np.array_equal(ctx.batch_tally_q(), want)


@pytest.mark.parametrize("mode", ["strict", "fast"])
def test_tiny_weights_stay_in_the_tiles(mcg, mode):
    """The same histories with a weight of 1e-25 and of 1: a full step for every
    crossing takes several times as long."""
    m = 1000
    times = []
    with mcg.Context(mode=mode) as ctx:
        ctx.set_layers_xs([0], [m], [f32(1.0 / m)], np.full(m, 1e-3 * m), np.full(m, 1e-3 * m), 0.0)
        for w0 in (1.0, 1e-25):
            best = []
            for _ in range(4):
                ctx.simulate_source(0, 300_000, w0=w0)
                best.append(ctx.last_kernel_ms())
            times.append(min(best))
    assert times[1] < 2 * times[0], times
