"""Batched few-body systems (config 4 shape: n ~ U[3, 64], Plummer with
virial radius 1e-3, eps = 0) in one persistent kernel, against smallN's
integrator restated in the oracle (itself bit-identical to smallN built from
the reference sources with dt_crit = 0, tests/test_batch_oracle.py)."""
import numpy as np
import pytest

import amuse_gb300 as ag
import oracle
from amuse_gb300 import ic

pytestmark = pytest.mark.gpu


def _systems(nsys, nmin, nmax, seed):
    ns, m, x, v, tcr = ic.encounter_batch(nsys, nmin, nmax, seed=seed)
    return ns, m, x, v, tcr


def test_exact_mode_is_bit_identical_to_smalln(g6):
    ns, m, x, v, tcr = _systems(24, 3, 40, seed=5)
    t_end = np.full(len(ns), 1.0 * tcr)
    r = g6.batch_run(ns, t_end, m, x, v, eta=0.14, exact=True)
    off = np.concatenate([[0], np.cumsum(ns)])
    for s in range(len(ns)):
        a, b = off[s], off[s + 1]
        px, pv, tf, st = oracle.smalln(m[a:b], x[a:b], v[a:b], 0.14, t_end[s])
        assert r["status"][s] == 0
        assert r["steps"][s] == st, s
        assert r["t_final"][s] == tf, s
        assert np.array_equal(r["pos"][a:b], px), s
        assert np.array_equal(r["vel"][a:b], pv), s


def test_exact_mode_matches_reference_smalln_fixtures(g6):
    """Against smallN built from the reference sources (tests/golden/
    smalln_systems.npz): n = 3 ... 64, two crossing times, bit for bit."""
    from conftest import golden
    g = golden("smalln_systems.npz")
    k = int(g["nsys"])
    ns = np.array([len(g[f"s{i}_mass"]) for i in range(k)], np.int32)
    cat = lambda key: np.concatenate([g[f"s{i}_{key}"] for i in range(k)])
    t_end = np.full(k, float(g["t_end"]))
    r = g6.batch_run(ns, t_end, cat("mass"), cat("pos0"), cat("vel0"), eta=float(g["eta"]),
                     exact=True)
    assert np.array_equal(r["pos"], cat("pos")) and np.array_equal(r["vel"], cat("vel"))
    assert np.array_equal(r["t_final"], np.array([float(g[f"s{i}_t"]) for i in range(k)]))


def _energy(m, x, v):
    k = 0.5 * np.sum(m * np.sum(v * v, 1))
    d = x[:, None, :] - x[None, :, :]
    r = np.sqrt(np.sum(d * d, -1))
    iu = np.triu_indices(len(m), 1)
    return k - np.sum(m[iu[0]] * m[iu[1]] / r[iu])


def test_fast_mode_conserves_energy_like_exact(g6):
    ns, m, x, v, tcr = _systems(64, 3, 64, seed=6)
    t_end = np.full(len(ns), 2.0 * tcr)
    fast = g6.batch_run(ns, t_end, m, x, v, exact=False)
    exact = g6.batch_run(ns, t_end, m, x, v, exact=True)
    off = np.concatenate([[0], np.cumsum(ns)])
    de_f, de_e = [], []
    for s in range(len(ns)):
        a, b = off[s], off[s + 1]
        e0 = _energy(m[a:b], x[a:b], v[a:b])
        de_f.append(abs((_energy(m[a:b], fast["pos"][a:b], fast["vel"][a:b]) - e0) / e0))
        de_e.append(abs((_energy(m[a:b], exact["pos"][a:b], exact["vel"][a:b]) - e0) / e0))
    print(f"median |dE/E| fast {np.median(de_f):.2e} exact {np.median(de_e):.2e}; "
          f"max fast {max(de_f):.2e} exact {max(de_e):.2e}")
    assert np.all(fast["status"] == 0) and np.all(fast["t_final"] >= t_end)
    # the scheme's own truncation error dominates: both modes agree on it
    assert np.median(de_f) < 2 * np.median(de_e) + 1e-12
    assert max(de_f) < 3 * max(de_e) + 1e-12


def test_split_mode_energy_and_short_time_agreement(g6):
    """Split mode (FP32 pair terms from double-single positions): over two
    crossing times its energy error stays at the scheme's truncation level
    (within 10x of exact mode, or 1e-7), and over a short time, before the
    systems' chaos amplifies rounding, it tracks the exact mode closely."""
    ns, m, x, v, tcr = _systems(64, 3, 64, seed=6)
    t_end = np.full(len(ns), 2.0 * tcr)
    split = g6.batch_run(ns, t_end, m, x, v, mode="split")
    exact = g6.batch_run(ns, t_end, m, x, v, mode="exact")
    off = np.concatenate([[0], np.cumsum(ns)])
    de_s, de_e = [], []
    for s in range(len(ns)):
        a, b = off[s], off[s + 1]
        e0 = _energy(m[a:b], x[a:b], v[a:b])
        de_s.append(abs((_energy(m[a:b], split["pos"][a:b], split["vel"][a:b]) - e0) / e0))
        de_e.append(abs((_energy(m[a:b], exact["pos"][a:b], exact["vel"][a:b]) - e0) / e0))
    print(f"median |dE/E| split {np.median(de_s):.2e} exact {np.median(de_e):.2e}; "
          f"max split {max(de_s):.2e} exact {max(de_e):.2e}")
    assert np.all(split["status"] == 0) and np.all(split["t_final"] >= t_end)
    assert np.median(de_s) < 10 * np.median(de_e) + 1e-7
    short = np.full(len(ns), 0.02 * tcr)
    rs = g6.batch_run(ns, short, m, x, v, mode="split")
    re = g6.batch_run(ns, short, m, x, v, mode="exact")
    scale = np.abs(re["pos"]).max()
    assert np.abs(rs["pos"] - re["pos"]).max() <= 1e-5 * scale


def test_step_budget_and_queue(g6):
    ns, m, x, v, tcr = _systems(500, 3, 64, seed=7)
    r = g6.batch_run(ns, 5 * tcr, m, x, v, max_steps=10)
    assert np.all(r["steps"] == 10) and np.all(r["status"] == 1)
    r = g6.batch_run(ns, 0.05 * tcr, m, x, v)
    assert np.all(r["status"] == 0) and np.all(r["t_final"] >= 0.05 * tcr)
    assert np.all(r["wall_ms"] > 0)


def test_autotuner(g6):
    ns, m, x, v, tcr = _systems(300, 3, 64, seed=8)
    best = g6.batch_tune(ns, tcr, m, x, v, frac=0.02)
    assert best["warps_per_cta"] >= 1 and best["ctas_per_sm"] >= 1 and best["ms"] > 0
    r = g6.batch_run(ns, 0.05 * tcr, m, x, v)
    assert np.all(r["status"] == 0)


# --- smallN's unperturbed binaries --------------------------------------------

def _unpert_fixture():
    from conftest import golden
    g = golden("smalln_unpert.npz")
    k = int(g["nsys"])
    ns = np.array([len(g[f"s{i}_mass"]) for i in range(k)], np.int32)
    cat = lambda key: np.concatenate([g[f"s{i}_{key}"] for i in range(k)])
    t_end = np.array([float(g[f"s{i}_t_end"]) for i in range(k)])
    return g, k, ns, cat, t_end


@pytest.mark.parametrize("mode", ["fast", "split"])
def test_unperturbed_binaries_follow_oracle_and_smalln(g6, mode):
    """Hierarchical systems with hard binaries (tests/golden/smalln_unpert.npz,
    written by the unmodified smallN with its unperturbed binaries): the batch
    kernel with the same treatment ends where the oracle's restatement
    (orc_smalln_unpert) and smallN end, to 1e-4 of the system size (fast:
    FP64 pair terms; split: FP32 pair terms), having made binaries, in far
    fewer steps than without them."""
    g, k, ns, cat, t_end = _unpert_fixture()
    g6.batch_unperturbed(True)
    try:
        r = g6.batch_run(ns, t_end, cat("mass"), cat("pos0"), cat("vel0"), eta=0.14, mode=mode)
        nbin = g6.batch_binaries(k)
    finally:
        g6.batch_unperturbed(False)
    plain = g6.batch_run(ns, t_end, cat("mass"), cat("pos0"), cat("vel0"), eta=0.14, mode=mode)
    off = np.concatenate([[0], np.cumsum(ns)])
    for s in range(k):
        a, b = off[s], off[s + 1]
        m, x0, v0 = g[f"s{s}_mass"], g[f"s{s}_pos0"], g[f"s{s}_vel0"]
        po, vo, to, so, nbo = oracle.smalln_unpert(m, x0, v0, 0.14, t_end[s])
        scale = np.abs(x0).max()
        d_or = np.abs(r["pos"][a:b] - po).max() / scale
        d_ref = np.abs(r["pos"][a:b] - g[f"s{s}_pos"]).max() / scale
        print(f"system {s} ({mode}): steps {r['steps'][s]} (plain {plain['steps'][s]}, oracle "
              f"{so}), binaries {nbin[s]} (oracle {nbo}), |dx| vs oracle {d_or:.1e}, "
              f"vs smallN {d_ref:.1e}")
        assert r["status"][s] == 0
        assert nbin[s] >= 1
        assert d_or <= 1e-4 and d_ref <= 1e-4
        assert r["steps"][s] < plain["steps"][s]


def test_unperturbed_refused_in_exact_mode(g6):
    g, k, ns, cat, t_end = _unpert_fixture()
    g6.batch_unperturbed(True)
    try:
        with pytest.raises(ag.G6Error, match="exact"):
            g6.batch_run(ns, t_end, cat("mass"), cat("pos0"), cat("vel0"), mode="exact")
    finally:
        g6.batch_unperturbed(False)


def test_unperturbed_batching_workload_completes(g6):
    """The batching configuration's systems (n ~ U[3, 64], Plummer r_vir =
    1e-3, eps = 0) to 10 crossing times with the unperturbed treatment: no
    system reaches the step budget, and the per-system energy error stays at
    the level of the scheme's truncation error."""
    ns, m, x, v, tcr = _systems(256, 3, 64, seed=9)
    t_end = np.full(len(ns), 10.0 * tcr)
    g6.batch_unperturbed(True)
    try:
        r = g6.batch_run(ns, t_end, m, x, v, mode="split", max_steps=2_000_000)
        nbin = g6.batch_binaries(len(ns))
    finally:
        g6.batch_unperturbed(False)
    off = np.concatenate([[0], np.cumsum(ns)])
    de = []
    for s in range(len(ns)):
        a, b = off[s], off[s + 1]
        e0 = _energy(m[a:b], x[a:b], v[a:b])
        de.append(abs((_energy(m[a:b], r["pos"][a:b], r["vel"][a:b]) - e0) / e0))
    de = np.array(de)
    print(f"binaries made: {nbin.sum()} in {np.sum(nbin > 0)} systems; |dE/E| median "
          f"{np.median(de):.2e} p99 {np.percentile(de, 99):.2e} max {de.max():.2e}; steps max "
          f"{r['steps'].max()}")
    assert np.all(r["status"] == 0) and np.all(r["t_final"] >= t_end)
    assert np.all(np.isfinite(de)) and np.median(de) < 1e-3


@pytest.mark.parametrize("first,then", [((4, 60), (40, 3)), ((40, 3), (6, 60)), ((5, 3), (90, 40))])
def test_batch_growing_in_systems_or_bodies(lib_built, first, then):
    """A second batch that outgrows the per-system buffers alone (more but
    smaller systems), the per-body buffers alone, or both: the launch must
    see the reallocated buffers."""
    g6 = ag.G6X(0)
    g6.close()  # start from empty batch buffers
    g6 = ag.G6X(0)
    for nsys, n in (first, then):
        ns, m, x, v, tcr = _systems(nsys, n, n, seed=nsys)
        r = g6.batch_run(ns, 0.05 * tcr, m, x, v, eta=0.14, exact=True, max_steps=100000)
        for s in range(0, nsys, 7):
            a, b = s * n, (s + 1) * n
            px, pv, tf, st = oracle.smalln(m[a:b], x[a:b], v[a:b], 0.14, 0.05 * tcr)
            assert r["status"][s] == 0 and r["steps"][s] == st and r["t_final"][s] == tf
            assert np.array_equal(r["pos"][a:b], px) and np.array_equal(r["vel"][a:b], pv)


@pytest.mark.parametrize("mode,tol", [("fast", 1e-9), ("split", 1e-6)])
@pytest.mark.parametrize("unp", [False, True])
def test_component_layout_edges(g6, mode, tol, unp):
    """Sizes at the edges of the component slots (3n = 32 k) and of the two
    leaves per lane, a few steps, against smallN: FP64 roundings amplified by
    at most 1e6, FP32 pair terms moving bodies by 1e-7 of a t^2 / 2 ~ 2e-3 of
    the size, amplified by 1e3 at the closest pair."""
    sizes = [2, 3, 10, 11, 21, 22, 32, 33, 42, 43, 53, 54, 63, 64]
    rng = np.random.RandomState(12)
    sysm = [ic.plummer(n, do_scale=True, rng=rng) for n in sizes]
    ns = np.array(sizes, np.int32)
    m = np.concatenate([s[0] for s in sysm])
    x = np.concatenate([s[1] for s in sysm]) * 1e-3
    v = np.concatenate([s[2] for s in sysm]) / np.sqrt(1e-3)
    t_end = 0.02 * 2 * np.sqrt(2) * 1e-3 ** 1.5
    # dt_crit = 0 makes no binaries: the tree's code with smallN's trajectory
    g6.batch_unperturbed(unp, dt_crit=0.0)
    try:
        r = g6.batch_run(ns, t_end, m, x, v, mode=mode, max_steps=100000)
    finally:
        g6.batch_unperturbed(False)
    off = np.concatenate([[0], np.cumsum(ns)])
    for s, n in enumerate(sizes):
        a, b = off[s], off[s + 1]
        px, pv, tf, st = oracle.smalln(m[a:b], x[a:b], v[a:b], 0.14, t_end)
        assert r["status"][s] == 0
        if mode == "fast":
            assert r["steps"][s] == st, n
        assert np.abs(r["pos"][a:b] - px).max() <= tol * 1e-3, n
        assert np.abs(r["vel"][a:b] - pv).max() <= tol * 1e3 * np.abs(pv).max(), n


@pytest.mark.parametrize("unp", [False, True])
def test_split_step_with_equal_pairs(g6, unp):
    """Rings in circular motion: every body has two nearest pairs of the same
    step, so the step comes from the quotients of all pairs, for one and two
    leaves per lane.  Over 0.2 of the dynamical time (R = 1) FP32 terms move a
    body by 1e-7 of a t^2 / 2 <= 0.1 and the end time by 1e-7 of a step; the
    ring's own instability grows at most by e^0.8."""
    sizes = [2, 3, 4, 31, 32, 33, 63, 64]
    ms, xs, vs = [], [], []
    for n in sizes:
        a = 2 * np.pi * np.arange(n) / n
        x = np.stack([np.cos(a), np.sin(a), 0 * a], 1)
        pull = (1.0 / n) * (1 / (4 * np.sin(np.pi * np.arange(1, n) / n))).sum()
        vs.append(np.sqrt(pull) * np.stack([-np.sin(a), np.cos(a), 0 * a], 1))
        ms.append(np.full(n, 1.0 / n))
        xs.append(x)
    g6.batch_unperturbed(unp, dt_crit=0.0)
    try:
        r = g6.batch_run(np.array(sizes, np.int32), 0.2, np.concatenate(ms), np.concatenate(xs),
                         np.concatenate(vs), mode="split", max_steps=100000)
    finally:
        g6.batch_unperturbed(False)
    off = np.concatenate([[0], np.cumsum(sizes)])
    for s, n in enumerate(sizes):
        px, pv, tf, st = oracle.smalln(ms[s], xs[s], vs[s], 0.14, 0.2)
        assert r["status"][s] == 0 and r["steps"][s] == st, n
        assert abs(r["t_final"][s] - tf) <= 1e-6
        assert np.abs(r["pos"][off[s]:off[s + 1]] - px).max() <= 1e-6, n
        assert np.abs(r["vel"][off[s]:off[s + 1]] - pv).max() <= 1e-6 * np.abs(pv).max(), n


@pytest.mark.parametrize("mode,unp", [("split", False), ("fast", True), ("exact", False)])
def test_shape_beyond_residency(g6, mode, unp):
    """More CTAs per SM asked for than fit (4 x 3 and 4 x 4 warps) leave no
    system waiting for a whole CTA to end: 400 equal systems, fewer than the
    warps that fit at once, would take twice as long as at 4 x 2."""
    m, x, v = ic.plummer(24, do_scale=True, rng=np.random.RandomState(13))
    ns = np.full(400, 24, np.int32)
    m, x, v = np.tile(m, 400), np.tile(x, (400, 1)) * 1e-3, np.tile(v, (400, 1)) / np.sqrt(1e-3)
    t_end = 0.01 * 2 * np.sqrt(2) * 1e-3 ** 1.5
    g6.batch_unperturbed(unp)
    ms, pos = [], []
    try:
        for shape in ((4, 2), (4, 3), (4, 4)):
            g6.batch_config(*shape)
            r = [g6.batch_run(ns, t_end, m, x, v, mode=mode, max_steps=100000) for _ in range(4)]
            ms.append(min(q["elapsed_ms"] for q in r[1:]))
            pos.append(r[-1]["pos"])
    finally:
        g6.batch_unperturbed(False)
        g6.batch_config(4, 2)
    assert np.array_equal(pos[0], pos[1]) and np.array_equal(pos[0], pos[2])
    assert max(ms) <= 1.4 * ms[0], ms


def _with_binaries(n, pairs, rng):
    """A Plummer system in which the two bodies of each pair circle the first
    one's place, 1e-3 of the nearest other body apart, e = 0.6, inbound."""
    m, x, v = ic.plummer(n, do_scale=True, rng=rng)
    for a, b in pairs:
        d = np.sqrt(((x - x[a]) ** 2).sum(1))
        d[[a, b]] = np.inf
        sma, mt, e, ea = 1e-3 * d.min(), m[a] + m[b], 0.6, 1.5 * np.pi
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        w = np.cross(u, rng.normal(size=3))
        w /= np.linalg.norm(w)
        f, g = np.sqrt(1 - e * e), np.sqrt(mt / sma) / (1 - e * np.cos(ea))
        r = sma * ((np.cos(ea) - e) * u + f * np.sin(ea) * w)
        s = g * (-np.sin(ea) * u + f * np.cos(ea) * w)
        c, cv = x[a].copy(), v[a].copy()
        x[a], x[b] = c - m[b] / mt * r, c + m[a] / mt * r
        v[a], v[b] = cv - m[b] / mt * s, cv + m[a] / mt * s
    return m, x * 1e-3, v / np.sqrt(1e-3)


BINARIES = {11: [(0, 10)], 21: [(0, 20)], 22: [(3, 21)], 32: [(0, 31), (5, 17)], 33: [(4, 32)],
            43: [(31, 32), (7, 42)], 54: [(9, 50), (33, 34)], 63: [(0, 62), (31, 33)],
            64: [(0, 63), (30, 40), (7, 8)]}


@pytest.mark.parametrize("mode", ["fast", "split"])
@pytest.mark.parametrize("full,t", [(True, 0.02), (False, 0.0005)], ids=["frozen", "dissolving"])
def test_binaries_at_layout_edges(g6, mode, full, t):
    """Hard binaries inside systems at the edges of the component slots, members
    on both sides of the 32nd slot, against orc_smalln_unpert: frozen over whole
    periods, or made and dissolved every period (up to 46 times here).  Inputs
    moved by 1e-15 of themselves move the oracle's end by up to 1e-13 of the size,
    1e-11 of the end time and 1e-9 of the velocities (fast: a hundred times that
    allowed and more); by 1e-8, 1e-4 of a binary's separation, by 1e-6, 1e-4 and
    1e-2 (split: FP32 terms are a thousand times more exact than that)."""
    tx, tt, tv = (1e-9, 1e-7, 1e-6) if mode == "fast" else (1e-6, 1e-4, 1e-2)
    made = {n: _with_binaries(n, p, np.random.RandomState(n)) for n, p in BINARIES.items()}
    ns = np.array(list(made), np.int32)
    m, x, v = (np.concatenate([made[n][k] for n in made]) for k in range(3))
    t_end = t * 2 * np.sqrt(2) * 1e-3 ** 1.5
    g6.batch_unperturbed(True, allow_full=full)
    try:
        r = g6.batch_run(ns, t_end, m, x, v, mode=mode, max_steps=100000)
        nbin = g6.batch_binaries(len(ns))
    finally:
        g6.batch_unperturbed(False)
    off = np.concatenate([[0], np.cumsum(ns)])
    for s, n in enumerate(ns):
        a, b = off[s], off[s + 1]
        px, pv, tf, st, nb = oracle.smalln_unpert(m[a:b], x[a:b], v[a:b], 0.14, t_end,
                                                  allow_full=full, max_steps=100000)
        assert r["status"][s] == 0 and nbin[s] >= len(BINARIES[n]), n
        if mode == "fast":
            assert r["steps"][s] == st and nbin[s] == nb, n
        assert abs(r["t_final"][s] - tf) <= tt * tf, n
        assert np.abs(r["pos"][a:b] - px).max() <= tx * 1e-3, n
        assert np.abs(r["vel"][a:b] - pv).max() <= tv * np.abs(pv).max(), n
