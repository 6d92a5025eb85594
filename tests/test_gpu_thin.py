"""Thin chains, whose tiles test a whole flight against the chain's widest cell,
where the cells are not alike: cells whose steps the tiles must leave to the
full step (negative absorption, faces that do not fit between layers), and cells
that are wider when entered from a neighbouring layer than between their own
faces.  The event-based tracker, which has neither tiles nor bounds per flight,
gives the same arithmetic by another path; results are exact."""
import numpy as np
import pytest

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
    out = []
    for algorithm in ("event", "history"):
        ctx.set_algorithm(algorithm, 1)
        ctx.tally_reset()
        ctx.simulate_source(0, n, **source)
        out.append((ctx.tally_q(), ctx.counters()))
    ctx.set_algorithm("history")
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
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
