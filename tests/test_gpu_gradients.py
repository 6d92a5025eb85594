"""Gradient kernels: the lanes cross cells on their own and take the full steps
together, so a history's terms are computed in rounds.  Checked at chain lengths
and cross sections where the two kinds of step mix differently (thin cells:
almost only crossings; thick ones: almost only full steps), at one history, a
warp's worth and more than a block's share, with the step's weight cut-off, and
for chains whose arrays leave no room for the seed chain's table.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

f32 = np.float32


def _problem(m, low, high):
    rng = np.random.default_rng(m)
    sa, ss = (m * 10.0 ** rng.uniform(low, high, (2, m))).astype(f32)
    return sa, ss, rng.standard_normal(m).astype(f32)


def _ctx(mcg, mode, sa, ss, w, min_w=1e-12):
    m = len(sa)
    ctx = mcg.Context(mode=mode)
    ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa, ss, min_w)
    ctx.adjoint_set_weights(w)
    return ctx


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,low,high", [(1, -2, 0), (2, -4, -2), (33, -3, 0.5), (40, -1, 0.5),
                                        (1000, -3.5, -2), (6900, -4, -3.5)])
@pytest.mark.parametrize("min_w", [1e-12, 0.5])
def test_forward_pass_equals_event_mode(mcg, mode, m, low, high, min_w):
    sa, ss, w = _problem(m, low, high)
    with _ctx(mcg, mode, sa, ss, w, min_w) as ctx:
        ctx.set_algorithm("event", 1)
        for n in (1, 31, 3000):
            ctx.tally_reset()
            ctx.simulate_source(7, n)
            ref, cnt = ctx.tally_q(), ctx.counters()
            ctx.tally_reset()
            ctx.adjoint_reset()
            ctx.adjoint_run(7, n)
            loss, _, _ = ctx.adjoint_read()
            assert np.array_equal(ctx.tally_q(), ref)
            assert [ctx.counters()[k] for k in ("steps", "scatters")] == [cnt[k] for k in ("steps", "scatters")]
            # float-float sums of products rounded to 24 bits, over at most unit weight
            assert abs(loss - (ctx.tally() * w).sum() / n) <= 2.0 ** -23 * np.abs(w).max()


@pytest.mark.parametrize("mode", ["strict", "fast"])
@pytest.mark.parametrize("m,low,high", [(1, -2, 0), (2, -4, -2), (33, -3, 0.5), (40, -1, 0.5),
                                        (256, -3, -1.5), (257, -3, -1.5), (400, -2, 0.5)])
def test_gradients_match_fp64_on_the_same_histories(mcg, oracle, mode, m, low, high):
    """The 64-bit estimator follows the same random numbers, so all but a few
    histories take the same path: a deposit's float32 rounding is at most about
    1e-4 of it, and a step goes the other way in about 1e-6 of all cases, which
    for 20000 histories of under 500 steps is ten of them: sqrt(2 * 10 / 20000) =
    3.2 % of a gradient that is all noise."""
    n = 20000
    sa, ss, w = _problem(m, low, high)
    with _ctx(mcg, mode, sa, ss, w) as ctx:
        ctx.adjoint_reset()
        ctx.adjoint_run(0, n)
        _, ga, gs = ctx.adjoint_read()
    p = np.zeros(n, oracle.PARTICLE_DTYPE)
    p["seed"] = oracle.rnd_seed_chain(5127801, n)
    p["mu"], p["wmc"] = 1.0, 1.0
    _, ra, rs = oracle.fp64_adjoint([oracle.layer_make(0.0, 1.0, 0, m)], sa.astype(float),
                                    ss.astype(float), w, 1e-12, p)
    for got, ref in ((ga, ra / n), (gs, rs / n)):
        assert np.linalg.norm(got - ref) <= 0.05 * np.linalg.norm(ref)


def test_more_histories_than_one_part(mcg):
    """Above 2^24 histories the forward pass and the replay take turns: the sums
    over two shorter runs, and the tracker's tally."""
    m, n = 257, (1 << 24) + 777
    sa, ss, w = _problem(m, -2, -1)
    with _ctx(mcg, "fast", sa, ss, w) as ctx:
        ctx.simulate_source(0, n)
        ref = ctx.tally_q()
        out = []
        for cuts in ((0, n), (0, 9_000_000, n)):
            ctx.tally_reset()
            ctx.adjoint_reset()
            for a, b in zip(cuts, cuts[1:]):
                ctx.adjoint_run(a, b - a)
            out.append(ctx.adjoint_read())
            assert np.array_equal(ctx.tally_q(), ref)
    (la, a0, s0), (lb, a1, s1) = out
    assert la == lb
    for x, y in ((a0, a1), (s0, s1)):
        assert np.abs(x - y).max() <= 1e-3 * np.abs(y).max()


@pytest.mark.parametrize("cells,histories", [((1, 2, 33, 700), (1, 31, 9000, 20000)),
                                             ((9000, 15000), (300, 300))])
def test_fit_pass_equals_adjoint(mcg, cells, histories):
    """Several slabs in one launch, one with two work items, two without room for
    the seed chain's table: the tallies of the adjoint kernel and its gradients
    but for the order of the float32 sums (a relative 1e-4 of the largest)."""
    rng = np.random.default_rng(5)
    slabs = [dict(n_cells=m, n_histories=n, base_seed=11 + m, seed_mode=0, isotropic=0, mu0=1.0,
                  w0=1.0) for m, n in zip(cells, histories)]
    total = sum(cells)
    sa, ss = rng.uniform(0.2, 2, total).astype(f32), rng.uniform(0.5, 5, total).astype(f32)
    w = rng.standard_normal(total).astype(f32)
    with mcg.Context(mode="fast") as ctx:
        ctx.fit_set(slabs, sa, ss, np.zeros(total), max_steps=1)
        t, g = ctx.fit_gradient(w)
    o = 0
    for d in slabs:
        m, n, k = d["n_cells"], d["n_histories"], slice(o, o + d["n_cells"])
        o += m
        if m > 14000:  # beyond the adjoint kernel's arrays: the tally alone
            with mcg.Context(mode="fast") as ctx:
                ctx.set_layers_xs([0], [m], [f32(1.0 / m)], sa[k], ss[k], 1e-12)
                ctx.simulate_source(0, n, seed_mode=0, base_seed=d["base_seed"])
                assert np.array_equal(t[k], ctx.tally() / n)
            continue
        with _ctx(mcg, "fast", sa[k], ss[k], w[k]) as ctx:
            ctx.adjoint_reset()
            ctx.adjoint_run(0, n, with_gradient=True, seed_mode=0, base_seed=d["base_seed"])
            _, ref, _ = ctx.adjoint_read()
            assert np.array_equal(t[k], ctx.tally() / n)
        assert np.abs(g[k] - ref).max() <= 1e-4 * np.abs(ref).max()
