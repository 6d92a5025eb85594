"""The work a user of this framework has it do, as measurable cases.

One pass is what a program does per call: clear the tally, run the
histories through a public entry point, read the tally and the counters
back.  Sizes and physics are those of the workload module, the benchmark and
the tests: the 100-cell ramp slab, the 1000-cell default layer of the
reference, the 10,000-cell sine slab in 64 sub-domains, batches of uneven
slabs, the 1000-cell differentiation slab, the inverse fit and the
hand-over workers.

Case fields: kind (which entry point), mode (strict or fast arithmetic) and
the sizes.  Everything random comes from the seed given to prepare().
"""
import importlib.util
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MASK63 = (1 << 63) - 1
CHAIN_G, CHAIN_C = 5177284530976225183, 2096348467109453893  # the seed chain
REAL_G, REAL_C = 6364136223846793005, 1442695040888963407    # the sample stream
EPS = 1e-4
MIN_W = 1e-12


def _package():
    if "mc_mpi_gb300" not in sys.modules:
        pkg = os.path.join(ROOT, "mc-mpi_gb300")
        spec = importlib.util.spec_from_file_location(
            "mc_mpi_gb300", os.path.join(pkg, "__init__.py"), submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["mc_mpi_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["mc_mpi_gb300"]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference's GPU seam as its Layer calls it: a few particles
        # from host arrays, geometry passed on every call
        dict(name="seam_100x1000", kind="seam", physics="decay", cells=100, histories=1000),
        # the small plain slab from host particles, every per-particle output wanted
        dict(name="host_100x1e5_strict", kind="host", mode="strict", physics="ramp", cells=100,
             layers=1, source="beam", histories=100_000),
        # the reference's default layer (isotropic source inside) on particles
        # that already live on the GPU
        dict(name="device_1000x1e6_fast", kind="device", mode="fast", physics="decay", cells=1000,
             layers=1, source="inside", histories=1_000_000),
        # the fine decomposed slab with few histories: a parameter scan's call
        dict(name="slab10k_1e5_strict", kind="source", mode="strict", physics="sine", cells=10_000,
             layers=64, source="beam", histories=100_000),
        # the same slab at production size (the largest case)
        dict(name="slab10k_2e7_strict", kind="device", mode="strict", physics="sine",
             cells=10_000, layers=64, source="beam", histories=20_000_000),
        dict(name="slab10k_4e6_fast", kind="source", mode="fast", physics="sine", cells=10_000,
             layers=64, source="beam", histories=4_000_000),
        # a few uneven slabs in one launch
        dict(name="batch_37_strict", kind="batch", mode="strict", slabs=37, max_cells=1031,
             max_histories=20_000),
        # thousands of uneven slabs in one launch, both arithmetics
        dict(name="batch_4096_strict", kind="batch", mode="strict", slabs=4096, max_cells=4096,
             max_histories=50_000),
        dict(name="batch_4096_fast", kind="batch", mode="fast", slabs=4096, max_cells=4096,
             max_histories=50_000),
        # forward tally, loss and both gradients of a differentiation step
        dict(name="adjoint_1000x2e6_strict", kind="adjoint", mode="strict", cells=1000,
             histories=2_000_000),
        # an inverse fit from its start: 64 slabs, Adam steps of batched
        # forward + adjoint launches
        dict(name="fit_64x5_steps", kind="fit", slabs=64, max_cells=1024, histories=100_000,
             steps=5),
        # the asynchronous hand-over workers on the decomposed slab
        dict(name="workers_10k_1e6_strict", kind="workers", mode="strict", physics="sine",
             cells=10_000, layers=64, source="beam", histories=1_000_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["seam", "host", "device", "source", "source", "batch", "batch", "adjoint",
                       "fit", "workers"])
    mode = rng.choice(["strict", "strict", "fast"])
    if kind == "seam":
        return dict(kind=kind, physics=rng.choice(["decay", "ramp"]),
                    cells=_log_int(rng, 16, 2000), histories=_log_int(rng, 64, 20_000))
    if kind == "batch":
        return dict(kind=kind, mode=mode, slabs=_log_int(rng, 16, 4096),
                    max_cells=_log_int(rng, 64, 4096), max_histories=_log_int(rng, 2000, 50_000))
    if kind == "adjoint":
        return dict(kind=kind, mode=mode, cells=_log_int(rng, 50, 4000),
                    histories=_log_int(rng, 5000, 1_000_000))
    if kind == "fit":
        return dict(kind=kind, slabs=rng.randint(5, 64), max_cells=_log_int(rng, 80, 1024),
                    histories=_log_int(rng, 5000, 100_000), steps=rng.randint(2, 5))
    cells = _log_int(rng, 16, 16_000)
    layers = 1 if kind != "workers" and rng.random() < 0.5 else rng.randint(2, min(64, cells))
    most = min(2e7 if kind == "source" else 2e6, 5e10 / cells)
    return dict(kind=kind, mode=mode, physics=rng.choice(["ramp", "decay", "sine"]), cells=cells,
                layers=layers, source=rng.choice(["beam", "inside"]),
                histories=_log_int(rng, 1000, most))


# ------------------------------------------------------------------ inputs
def _xs(case, rng):
    """sigma_a, sigma_s per cell of a plain case, float32; the seed shifts the
    profile a little."""
    m = case["cells"]
    x = (np.arange(m, dtype=np.float64) + 0.5) / m
    k = 1.0 + 0.05 * rng.random()
    if case["physics"] == "ramp":      # sigma_a = 0.2 + 1.8 x, sigma_s = 1
        sa, ss = 0.2 + 1.8 * k * x, np.ones(m)
    elif case["physics"] == "sine":    # the fine slab
        sa, ss = 0.5 + 0.4 * np.sin(6 * np.pi * x * k), 2.0 + 1.5 * np.cos(4 * np.pi * x)
    else:                              # the Layer constructor: exp(-x), half absorbed
        sa = ss = 0.5 * np.exp(-k * x)
    return sa.astype(np.float32), ss.astype(np.float32)


def _sigs_rates(sa, ss):
    sigs = (sa + ss).astype(np.float32)
    return sigs, (sa / sigs).astype(np.float32)


def _source(case, seed):
    """Keyword arguments of a device-born source."""
    base = 5127801 + 7919 * int(seed)
    if case.get("source", "beam") == "beam":
        return dict(seed_mode=0, base_seed=base, x0=0.0, mu0=1.0, w0=1.0, isotropic=0, cell0=0)
    x0 = np.float32(np.sqrt(2.0) / 2.0)
    cell = int(x0 / (np.float32(1.0) / np.float32(case["cells"])))
    return dict(seed_mode=0, base_seed=base, x0=float(x0), mu0=1.0, w0=1.0, isotropic=1,
                cell0=min(cell, case["cells"] - 1))


def _particles(case, seed):
    """The source's particles as a host array (the seed chain on the GPU)."""
    pkg = _package()
    src = _source(case, seed)
    s = _seed_chain(src["base_seed"], case["histories"])
    mu = torch.ones(len(s), dtype=torch.float32, device="cuda")
    if src["isotropic"]:
        s = _lcg(s)
        mu = 2.0 * (s.to(torch.float32) * 2.0 ** -63) - 1.0
    p = np.zeros(len(s), pkg.PARTICLE_DTYPE)
    p["seed"], p["mu"] = s.cpu().numpy().astype(np.uint64), mu.cpu().numpy()
    p["x"], p["wmc"], p["index"] = src["x0"], src["w0"], src["cell0"]
    return p


def _chain_context(case, seed):
    pkg = _package()
    sigs, rates = _sigs_rates(*_xs(case, np.random.default_rng([int(seed), 1])))
    st, m, dx, _, _ = pkg.layer_decomposition(0.0, 1.0, case["cells"], case["layers"])
    ctx = pkg.Context(mode=case["mode"])
    ctx.set_layers(st, m, dx, sigs, rates, MIN_W)
    ctx.set_tally_scale(35)
    return ctx


def _slabs(case, seed):
    """Uneven slabs: cells uniform, lengths U[0.5, 5], sigma_a U[0.1, 5],
    sigma_s U[0, 10], histories log-uniform; beam and half-isotropic sources.
    The sizes belong to the case, the physics and the particles to the seed."""
    rng, sizes = np.random.default_rng([int(seed), 2]), np.random.default_rng(case["slabs"])
    n = case["slabs"]
    cells = sizes.integers(16, case["max_cells"] + 1, n)
    hist = np.exp(sizes.uniform(np.log(50), np.log(case["max_histories"]), n)).astype(int) + 1
    total = int(cells.sum())
    length = np.repeat(rng.uniform(0.5, 5.0, n).astype(np.float32), cells)
    sa = rng.uniform(0.1, 5.0, total).astype(np.float32)
    ss = rng.uniform(0.0, 10.0, total).astype(np.float32)
    sigs, rates = _sigs_rates(sa, ss)
    slabs = [dict(n_cells=int(cells[s]), n_histories=int(hist[s]),
                  base_seed=5127801 + 7919 * s + 104729 * int(seed), seed_mode=0,
                  isotropic=0 if s % 2 == 0 else 2, mu0=1.0, w0=1.0) for s in range(n)]
    return slabs, (sigs * length).astype(np.float32), rates


def _adjoint_inputs(case, seed):
    rng = np.random.default_rng([int(seed), 3])
    m = case["cells"]
    sa = (2.0 * rng.uniform(0.2, 2.0, m)).astype(np.float32)
    ss = (2.0 * rng.uniform(0.5, 5.0, m)).astype(np.float32)
    return sa, ss, rng.standard_normal(m).astype(np.float32)


def _fit_inputs(case, seed):
    """Slabs with a hidden sine sigma_a; the targets are its analytic
    uncollided-beam absorption with a few per cent of noise, as a measured
    tally would have."""
    rng, sizes = np.random.default_rng([int(seed), 4]), np.random.default_rng(case["slabs"])
    slabs, target = [], []
    for s in range(case["slabs"]):
        m = int(sizes.integers(min(64, case["max_cells"] // 2), case["max_cells"] + 1))
        x = (np.arange(m) + 0.5) / m
        hidden = 1.0 + 0.8 * np.sin(2 * np.pi * rng.integers(1, 5) * x + rng.uniform(0, 6.28))
        left = np.exp(-np.concatenate([[0.0], np.cumsum(hidden / m)]))
        target.append((left[:-1] - left[1:]) * (1.0 + 0.03 * rng.standard_normal(m)))
        slabs.append(dict(n_cells=m, n_histories=case["histories"], seed_mode=0, isotropic=0,
                          base_seed=5127801 + 104729 * s + 7919 * int(seed), mu0=1.0, w0=1.0))
    target = np.concatenate(target)
    return dict(slabs=slabs, target=target, sig_a0=np.ones(len(target), np.float32),
                sig_s=np.full(len(target), 1.5, np.float32))


def prepare(case, seed):
    pkg = _package()
    kind, n = case["kind"], case.get("histories")
    if kind == "seam":
        sigs, rates = _sigs_rates(*_xs(case, np.random.default_rng([int(seed), 1])))
        return dict(kind=kind, sigs=sigs, rates=rates, dx=1.0 / case["cells"],
                    particles=_particles(dict(case, source="inside"), seed))
    if kind == "batch":
        ctx = pkg.Context(mode=case["mode"])
        ctx.batch_set(*_slabs(case, seed), MIN_W)
        return dict(kind=kind, ctx=ctx)
    if kind == "adjoint":
        sa, ss, w = _adjoint_inputs(case, seed)
        ctx = pkg.Context(mode=case["mode"])
        m = case["cells"]
        ctx.set_layers_xs([0], [m], [np.float32(1.0) / np.float32(m)], sa, ss, MIN_W)
        ctx.adjoint_set_weights(w)
        return dict(kind=kind, ctx=ctx, n=n, source=_source(case, seed))
    if kind == "fit":
        return dict(kind=kind, ctx=pkg.Context(mode="fast"), steps=case["steps"],
                    **_fit_inputs(case, seed))
    state = dict(kind=kind, ctx=_chain_context(case, seed), n=n, source=_source(case, seed))
    if kind == "host":
        state["particles"] = _particles(case, seed)
    elif kind == "device":
        state["born"] = torch.from_numpy(_particles(case, seed).view(np.uint8)).cuda()
        state["particles"] = torch.empty_like(state["born"])
        state["results"] = torch.empty(n, dtype=torch.int32, device="cuda")
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "seam":
        p = state["particles"].copy()
        absorbed = np.zeros(len(state["sigs"]), np.float32)
        _package().cusimulate(p, state["sigs"], state["rates"], absorbed, 0, len(absorbed),
                              state["dx"])
        return dict(particles=p.view(np.uint8), absorbed=absorbed)
    ctx = state["ctx"]
    if kind == "batch":
        ctx.batch_tally_reset()
        ctx.batch_run()
        return dict(tally=ctx.batch_tally_q(), counters=list(ctx.counters().values()))
    if kind == "adjoint":
        ctx.adjoint_reset()
        ctx.adjoint_run(0, state["n"], **state["source"])
        loss, ga, gs = ctx.adjoint_read()
        return dict(loss=loss, grad_a=ga, grad_s=gs, tally=ctx.tally(), tally_q=ctx.tally_q())
    if kind == "fit":
        ctx.fit_set(state["slabs"], state["sig_a0"], state["sig_s"], state["target"],
                    max_steps=state["steps"])
        ctx.fit_run(state["steps"])
        sig, loss = ctx.fit_read()
        return dict(sig_a=sig, loss=loss)
    ctx.tally_reset()
    out = {}
    if kind == "host":
        p = state["particles"].copy()
        out = ctx.simulate(p)
        out["particles"] = p.view(np.uint8)
    elif kind == "device":
        state["particles"].copy_(state["born"])
        ctx.simulate_device_ptr(state["particles"].data_ptr(), state["n"],
                                state["results"].data_ptr())
        out = dict(particles=state["particles"], results=state["results"])
    elif kind == "workers":
        ctx.worker_run_async(state["n"], **state["source"])
    else:
        ctx.simulate_source(0, state["n"], **state["source"])
    out.update(tally=ctx.tally(), tally_q=ctx.tally_q())
    c = ctx.counters()
    if kind == "workers":  # the workers count finished histories and steps only
        c = {k: c[k] for k in ("histories", "steps", "scatters")}
    out["counters"] = list(c.values())
    return out


# ------------------------------------------------------------------ work
# steps per history and cell of each physics (a property of the workload:
# counted once, beam / interior source), about 20 operations a step
STEPS_PER_CELL = dict(ramp=(1.06, 0.70), decay=(0.99, 0.58), sine=(1.10, 0.89))
OPS_PER_STEP = 20.0


def work(case):
    kind = case["kind"]
    if kind == "batch":
        span = np.log(case["max_histories"] / 50.0)
        n = case["slabs"] * (case["max_histories"] - 50.0) / span
        m = (16 + case["max_cells"]) / 2
        return dict(bytes=case["slabs"] * m * 24.0, flops=n * m * 0.67 * OPS_PER_STEP)
    if kind == "fit":
        m = (64 + case["max_cells"]) / 2
        n = case["slabs"] * case["histories"] * case["steps"]
        return dict(bytes=case["slabs"] * m * (40.0 + 48.0 * case["steps"]),
                    flops=n * m * 1.0 * 3 * OPS_PER_STEP)
    if kind == "adjoint":
        return dict(bytes=case["cells"] * 48.0,
                    flops=case["histories"] * case["cells"] * 1.2 * 3 * OPS_PER_STEP)
    per = STEPS_PER_CELL[case["physics"]][0 if case.get("source") == "beam" else 1]
    moved = case["cells"] * 16.0
    if kind in ("seam", "host", "device"):
        moved += case["histories"] * (52.0 if kind != "host" else 68.0)
    return dict(bytes=moved, flops=case["histories"] * case["cells"] * per * OPS_PER_STEP)


# ------------------------------------------------------------------ 64 bits
def _lcg(s, g=REAL_G, c=REAL_C):
    return (s * g + c) & MASK63


def _seed_chain(base, n):
    """First n states of the seed chain after `base` (int64 on the GPU)."""
    out = torch.empty(n, dtype=torch.int64, device="cuda")
    s = torch.tensor(int(base) & MASK63, dtype=torch.int64, device="cuda")
    out[0] = _lcg(s, CHAIN_G, CHAIN_C)
    g, c, have = CHAIN_G, CHAIN_C, 1
    while have < n:  # states k + have are the have-step jump of states k
        k = min(have, n - have)
        gs = torch.tensor(g - (1 << 63) * (g >> 63), dtype=torch.int64, device="cuda")
        out[have:have + k] = (out[:k] * gs + c) & MASK63
        g, c, have = (g * g) & MASK63, (g * c + c) & MASK63, have + k
    return out


def _histories64(sa, ss, lo, hi, s, x, mu, cell, min_w, weights=None):
    """The step of the tracker in double: absorbed weight per cell and, with
    loss weights, the summed loss and both gradients (path replayed)."""
    dev, m = s.device, len(sa)
    sa, ss, lo, hi = (torch.from_numpy(np.asarray(v, np.float64)).to(dev) for v in (sa, ss, lo, hi))
    tally = torch.zeros(m, dtype=torch.float64, device=dev)
    grad_a, grad_s = torch.zeros_like(tally), torch.zeros_like(tally)
    loss = torch.zeros(len(s), dtype=torch.float64, device=dev)
    lw = None if weights is None else torch.from_numpy(weights.astype(np.float64)).to(dev)
    born = s, x, mu, cell
    for phase in range(1 if lw is None else 2):
        s, x, mu, cell = (v.clone() for v in born)
        w, done = torch.ones_like(x), torch.zeros_like(x)
        ids = torch.arange(len(s), device=dev)
        for it in range(1 << 20):
            if it % 16 == 0:
                k = (w >= min_w) & (cell >= 0) & (cell < m)
                if not bool(k.any()):
                    break
                s, x, mu, cell, w, done, ids = (v[k] for v in (s, x, mu, cell, w, done, ids))
            live = (w >= min_w) & (cell >= 0) & (cell < m)
            c = cell.clamp(0, m - 1)
            s1 = _lcg(s)
            h = s1.to(torch.float64) * 2.0 ** -63
            a, i = sa[c], ss[c]
            di = torch.where(i > EPS, -torch.log(h) / i, torch.inf)
            edge = torch.where(mu < 0, lo[c], hi[c])
            de = torch.where(mu.abs() > EPS, (edge - x) / mu, torch.inf)
            coll = di < de
            s2 = _lcg(s1)
            f = torch.where(coll, di, de)
            dep = torch.where(live, -torch.expm1(-a * f) * w, 0.0)
            w = w - dep
            if phase == 0:
                tally.index_add_(0, c, dep)
                if lw is not None:
                    loss.index_add_(0, ids, lw[c] * dep)
            else:
                before = loss[ids] - done
                done = done + lw[c] * dep
                score = torch.where(coll, 1.0 / i.clamp_min(EPS), 0.0) - f
                z = torch.zeros_like(f)
                grad_a.index_add_(0, c, torch.where(live, f * (lw[c] * w - (loss[ids] - done)), z))
                grad_s.index_add_(0, c, torch.where(live, score * before, z))
            x = torch.where(live, torch.where(coll, x + di * mu, edge), x)
            nmu = 2.0 * (s2.to(torch.float64) * 2.0 ** -63) - 1.0
            cell = torch.where(live & ~coll, torch.where(mu < 0, cell - 1, cell + 1), cell)
            mu = torch.where(live & coll, nmu, mu)
            s = torch.where(coll, s2, s1)
    return tally, loss, grad_a, grad_s


def exact(case, seed):
    kind, n = case["kind"], case.get("histories", 0)
    if kind in ("batch", "fit", "workers") or case["cells"] > 1500 or n > 2_100_000:
        return None  # too many passes of the step loop for plain torch
    m = case["cells"]
    s = _seed_chain(_source(case, seed)["base_seed"], n)
    dx = np.float32(1.0) / np.float32(m)
    if case.get("layers", 1) > 1:  # contiguous layers, each with its own float spacing
        parts = np.array([len(v) for v in np.array_split(np.arange(m), case["layers"])])
        first = np.concatenate([[0], np.cumsum(parts)])
        at = first.astype(np.float32) * dx
        dx = np.repeat((at[1:] - at[:-1]) / parts.astype(np.float32), parts)
    lo = np.arange(m, dtype=np.float32) * dx
    hi = np.arange(1, m + 1, dtype=np.float32) * dx
    if kind == "adjoint":
        sa, ss, weights = _adjoint_inputs(case, seed)
    else:
        sigs, rates = _sigs_rates(*_xs(case, np.random.default_rng([int(seed), 1])))
        sa, ss, weights = sigs * rates, sigs * (1.0 - rates.astype(np.float64)), None
    src = _source(dict(case, source="inside") if kind == "seam" else case, seed)
    mu = torch.full((n,), 1.0, dtype=torch.float64, device="cuda")
    if src["isotropic"]:
        s = _lcg(s)
        mu = 2.0 * (s.to(torch.float64) * 2.0 ** -63) - 1.0
    x = torch.full((n,), src["x0"], dtype=torch.float64, device="cuda")
    cell = torch.full((n,), src["cell0"], dtype=torch.int64, device="cuda")
    tally, loss, ga, gs = _histories64(sa, ss, lo, hi, s, x, mu, cell,
                                       -np.inf if kind == "seam" else MIN_W, weights)
    if kind == "seam":
        return dict(particles=None, absorbed=tally)
    if kind == "adjoint":
        return dict(loss=float(loss.sum()) / n, grad_a=ga / n, grad_s=gs / n, tally=tally,
                    tally_q=None)
    out = dict(tally=tally, tally_q=None, counters=None)
    if kind == "host":
        out.update(results=None, steps=None, scatters=None, particles=None)
    elif kind == "device":
        out.update(particles=None, results=None)
    return out
