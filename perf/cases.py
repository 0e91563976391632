"""The work that a user of this library has it do, as cases that can be timed.

Each case is one call (or the few calls of one block step) through the public
Python entry points of ``amuse_gb300``, which are the C ABI's.  The kinds:

  abi     one block of ph4's GPU loop through the GRAPE-6 calls with host
          arrays: g6_set_j_particle for the block's particles, then
          g6_set_ti and g6calc_firsthalf / lasthalf(2) on them
  all     a shared step of a phiGRAPE- or hermite-like caller: every particle
          sent with g6_set_j_particle, then the force on all of them
  slots   a block of the device-resident loop: the force on listed slots,
          results left on the GPU
  dev     the force on explicit device arrays of i-particles
  fixed   the shared force of the fixed-step path, device arrays in and out
  run     device-resident block steps from the initial state (load, first
          forces, a number of blocks, read back): ph4's evolve_model
  knn     the k nearest neighbours (ph4's get_densities_on_gpu)
  adjoint the differentiable fixed-step integrator, forward and backward
  batch   many few-body systems in one launch (smallN's scheme)
  scatter one increment of the multiples hand-off: binary-single encounters

A program keeps one j-system on the GPU and calls with other blocks and times,
so for abi, slots, dev and knn the j-system belongs to the case and the seed
draws the block and the time.
"""
import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

import amuse_gb300 as ag
from amuse_gb300 import ic
from amuse_gb300.adjoint import hermite_fixed

TINY = 2.0 ** -52  # ph4 adds it to the softened distance
_PD = ctypes.POINTER(ctypes.c_double)
_PI = ctypes.POINTER(ctypes.c_int)


def listed():
    return [
        # ph4 at its smallest: N = 1024, a handful of active particles, with
        # the neighbour search; all latency
        dict(name="abi_tiny", kind="abi", n=1024, ni=8, imf="equal", eps2=1e-4, nn=True,
             prec="split"),
        # the mean block of the N = 65536 Salpeter run, neighbours wanted
        dict(name="abi_block", kind="abi", n=65536, ni=722, imf="salpeter", eps2=1e-6, nn=True,
             prec="split"),
        # a shared step with host arrays
        dict(name="abi_all", kind="all", n=32768, imf="equal", eps2=1e-4, nn=False),
        # the mean block of the N = 2^20 run
        dict(name="slots_1m", kind="slots", n=1 << 20, ni=11719, imf="equal", eps2=1e-6,
             nn=False, prec="split"),
        # the shared force of a large fixed-step run
        dict(name="fixed_131k", kind="fixed", n=131072, eps2=1e-4, prec="split", jerk="hermite"),
        # the FP64 mode (G6_PRECISION=fp64) on a block, neighbours wanted
        dict(name="fp64_block", kind="dev", n=16384, ni=501, imf="equal", eps2=1e-4, nn=True,
             prec="fp64"),
        # N = 1024 at eta = 0.01, where block steps want FP64 forces
        dict(name="run_fp64", kind="run", n=1024, imf="equal", eps2=1e-4, eta=0.01, blocks=128,
             prec="fp64"),
        # block steps with a mass spectrum at ph4's default eta
        dict(name="run_split", kind="run", n=16384, imf="salpeter", eps2=1e-6, eta=0.14,
             blocks=128, prec="split"),
        # ph4's knn = 12 of every particle
        dict(name="knn_all", kind="knn", n=65536, ni=65536, k=12),
        # gradient of a short fixed-step run
        dict(name="adjoint", kind="adjoint", n=8192, nsteps=16, checkpoint=8, eps2=1e-4,
             prec="split", jerk="hermite"),
        # uneven few-body systems, smallN's unperturbed binaries on
        dict(name="batch_mixed", kind="batch", nsys=1024, nmin=3, nmax=64, mode="split", unp=True,
             tcr=0.05),
        # the multiples hand-off's most common encounter
        dict(name="scatter", kind="scatter", nsys=4096, mode="split", unp=True, t_end=10.0),
    ]


def _log(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm, half of them odd."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v | 1 if rng.random() < 0.5 else v))


def draw(rng):
    kind = rng.choice(["abi", "abi", "all", "slots", "dev", "dev", "fixed", "run", "knn",
                       "adjoint", "batch", "scatter"])
    c = dict(kind=kind)
    imf = rng.choice(["equal", "salpeter"])
    nn = rng.random() < 0.5
    prec = "split" if rng.random() < 0.7 else "fp64"
    if kind == "abi":
        n = _log(rng, 256, 131072)
        c.update(n=n, ni=_log(rng, 1, min(n, 4096)), imf=imf, eps2=rng.choice([1e-4, 1e-6]),
                 nn=nn, prec="split")
    elif kind == "all":
        c.update(n=_log(rng, 512, 32768), imf=imf, eps2=1e-4, nn=nn)
    elif kind in ("slots", "dev"):
        if prec == "fp64":
            n = _log(rng, 512, 32768)
            ni = _log(rng, 1, min(n, (1 << 23) // n))
        else:
            n = _log(rng, 4096, 1 << 20)
            ni = _log(rng, 1, min(n, (3 << 32) // n))
        c.update(n=n, ni=ni, imf=imf, eps2=rng.choice([1e-4, 1e-6]), nn=nn, prec=prec)
    elif kind == "fixed":
        n = _log(rng, 512, 131072) if prec == "split" else _log(rng, 256, 4096)
        c.update(n=n, eps2=1e-4, prec=prec, jerk=rng.choice(["hermite", "softened"]))
    elif kind == "run":
        c.update(n=_log(rng, 256, 16384 if prec == "split" else 2048), imf=imf, eps2=1e-4,
                 eta=0.14 if prec == "split" else 0.01, blocks=rng.choice([32, 64, 128]),
                 prec=prec)
    elif kind == "knn":
        n = _log(rng, 4096, 65536)
        c.update(n=n, ni=n if rng.random() < 0.5 else _log(rng, 64, n), k=rng.choice([6, 12, 24]))
    elif kind == "adjoint":
        c.update(n=_log(rng, 256, 8192) if prec == "split" else _log(rng, 128, 1024),
                 nsteps=rng.choice([4, 8, 16]), checkpoint=rng.choice([4, 8, 16]), eps2=1e-4,
                 prec=prec, jerk=rng.choice(["hermite", "softened"]))
    elif kind == "batch":
        mode = rng.choice(["split", "fast", "exact"])
        lo = rng.choice([3, 3, 8, 24])
        c.update(nsys=_log(rng, 32, 1024), nmin=lo, nmax=rng.choice([lo + 4, 40, 64]), mode=mode,
                 unp=mode != "exact" and rng.random() < 0.5,
                 tcr=0.05 if mode == "split" else 0.01)
    else:
        c.update(nsys=_log(rng, 16, 4096), mode=rng.choice(["split", "split", "fast"]), unp=True,
                 t_end=rng.choice([5.0, 10.0]))
    return c


# ------------------------------------------------------------ particles ---
def _cluster(n, imf, seed):
    """mass, pos, vel of a cluster in N-body units, bodies as AMUSE draws them."""
    rng = np.random.RandomState(seed & 0x7FFFFFFF)
    m, x, v = ic.plummer(n, rng=rng)
    if imf == "salpeter":
        m = ic.salpeter_masses(n, -2.35, 0.1, 100.0, rng=rng)
        ic.move_to_center(m, x, v)
    return m, x, v


def _mean_field(x, v):
    """Acceleration and jerk of the Plummer model's mean field (M = 1): what
    the j-particles of a running system carry, near enough."""
    s = ((x * x).sum(1) + (3 * math.pi / 16) ** 2)[:, None]
    rv = (x * v).sum(1)[:, None]
    return -x * s ** -1.5, -v * s ** -1.5 + 3 * rv * x * s ** -2.5


_host = {"key": None}  # the j-system of the current case, host arrays
_gpu = {"key": None}   # which j-system the library holds


def _system(c):
    key = (c["n"], c.get("imf", "equal"))
    if _host["key"] != key:
        m, x, v = _cluster(c["n"], key[1], 1000003 + c["n"])
        a, j = _mean_field(x, v)
        n = c["n"]
        _host.update(key=key, m=m, x=x, v=v, a=a, j=j, t=np.zeros(n), dt=np.full(n, 2.0 ** -7),
                     ids=np.arange(1, n + 1, dtype=np.int32))
    return _host


def _library(prec):
    g6 = ag.G6X(0)
    want = ag.FP64 if prec == "fp64" else ag.SPLIT
    if g6.get_precision() != want:
        g6.set_precision(want)
    return g6


def _hold(s):
    """The library with this state's j-system in it."""
    g6 = _library(s["prec"])
    if _gpu["key"] != s["key"]:
        h = s["sys"]
        g6.load_particles(h["m"], h["x"], h["v"], h["a"], h["j"], h["t"], h["dt"], h["ids"])
        _gpu["key"] = s["key"]
    return g6


def _predict(h, k, t):
    d = (t - h["t"][k])[:, None]
    x = h["x"][k] + d * (h["v"][k] + 0.5 * d * (h["a"][k] + d * h["j"][k] / 3))
    return x, h["v"][k] + d * (h["a"][k] + 0.5 * d * h["j"][k])


def _d(a):
    return a.ctypes.data_as(_PD)


def _i(a):
    return a.ctypes.data_as(_PI)


_reserved = []


def _reserve():
    """One launch of the largest batch, ending after its first step: the
    library's batch buffers then hold every batch of this program."""
    if not _reserved:
        r = np.random.RandomState(5)
        n, k = 4096, 16
        _library("split").batch_run(np.full(n, k, np.int32), 1e-9, np.full(n * k, 1.0 / k),
                                    r.normal(size=(n * k, 3)), r.normal(size=(n * k, 3)))
        _reserved.append(True)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _encounters(nsys, seed):
    """Binary-single scatterings: a binary of 0.5 + 0.5 with a = 1, e to 0.7,
    random phase and orientation, and a single of 0.5 from d = 15 at 0.6."""
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    e, E = r.uniform(0, 0.7, nsys), r.uniform(0, 2 * np.pi, nsys)
    w = np.sqrt(1 - e * e)
    s = 1 / (1 - e * np.cos(E))
    zero = np.zeros(nsys)
    xr = np.stack([np.cos(E) - e, w * np.sin(E), zero], 1)
    vr = np.stack([-s * np.sin(E), s * w * np.cos(E), zero], 1)
    q = np.linalg.qr(r.normal(size=(nsys, 3, 3)))[0]
    xr, vr = np.einsum("nij,nj->ni", q, xr), np.einsum("nij,nj->ni", q, vr)
    b = 1.5 * np.sqrt(r.uniform(size=nsys))
    far = np.stack([np.full(nsys, -15.0), b, zero], 1)
    x = np.stack([-0.5 * xr, 0.5 * xr, far], 1)
    v = np.stack([-0.5 * vr, 0.5 * vr, np.stack([np.full(nsys, 0.6), zero, zero], 1)], 1)
    x -= x.mean(1, keepdims=True)
    v -= v.mean(1, keepdims=True)
    return np.full(nsys, 3, np.int32), np.full(3 * nsys, 0.5), x.reshape(-1, 3), v.reshape(-1, 3)


# --------------------------------------------------------------- prepare ---
def prepare(case, seed):
    c, kind = case, case["kind"]
    rng = np.random.RandomState((seed * 7919 + c.get("n", c.get("nsys", 1))) & 0x7FFFFFFF)
    s = dict(case=c, kind=kind, prec=c.get("prec", "split"))
    if kind in ("abi", "slots", "dev", "knn"):
        h = _system(c)
        s.update(sys=dict(h), key=(kind == "abi",) + h["key"], t=float(rng.uniform(0.0, 2.0 ** -7)))
        _hold(s)
    if kind in ("abi", "slots", "dev"):
        ni = c["ni"]
        k = np.sort(rng.permutation(c["n"])[:ni]).astype(np.int32)
        s.update(slots=k)
        x, v = _predict(h, k, s["t"])
        if kind == "abi":
            s.update(x=x, v=v, ids=h["ids"][k].copy(),
                     out=dict(acc=np.zeros((ni, 3)), jerk=np.zeros((ni, 3)), pot=np.zeros(ni),
                              nn=np.zeros(ni, np.int32)))
        else:
            f = dict(dtype=torch.float64, device="cuda")
            s.update(x=_dev(x), v=_dev(v), dslots=_dev(k), acc=torch.zeros(ni, 3, **f),
                     jerk=torch.zeros(ni, 3, **f), pot=torch.zeros(ni, **f),
                     nn=torch.zeros(ni, dtype=torch.int32, device="cuda"))
    elif kind == "knn":
        n, ni = c["n"], c["ni"]
        s["slots"] = (np.arange(n) if ni == n else np.sort(rng.permutation(n)[:ni])).astype(np.int32)
    elif kind in ("all", "run"):
        m, x, v = _cluster(c["n"], c["imf"], seed)
        a, j = _mean_field(x, v)
        s.update(m=m, x=x, v=v, a=a, j=j, ids=np.arange(1, c["n"] + 1, dtype=np.int32))
        _library(s["prec"])
    elif kind in ("fixed", "adjoint"):
        m, x, v = _cluster(c["n"], "equal", seed)
        s.update(m=_dev(m), x=_dev(x), v=_dev(v), w=_dev(rng.uniform(0.5, 1.5, c["n"])),
                 a=_dev(np.zeros_like(x)), j=_dev(np.zeros_like(x)))
        _library(s["prec"])
    elif kind == "batch":
        ns, m, x, v, tcr = _uneven(c, seed)
        s.update(ns=ns, m=m, x=x, v=v, t_end=c["tcr"] * tcr)
        _reserve()
    else:
        ns, m, x, v = _encounters(c["nsys"], seed)
        s.update(ns=ns, m=m, x=x, v=v, t_end=c["t_end"])
        _reserve()
    return s


def _uneven(c, seed):
    """nsys equal-mass Plummer systems in virial equilibrium, virial radius
    1e-3.  The case sets how many bodies each has; the seed draws up to 64
    realisations, and the rest are turned and shuffled copies of them (the
    velocities turned the other way: other systems of the same energy)."""
    size = np.random.RandomState(c["nsys"] + 1009 * c["nmin"] + 9176 * c["nmax"])
    base = min(c["nsys"], 64)
    ns = size.randint(c["nmin"], c["nmax"] + 1, size=base)
    pick = np.concatenate([np.arange(base), size.randint(base, size=c["nsys"] - base)])
    r = np.random.RandomState((seed + 17) & 0x7FFFFFFF)
    made = [ic.plummer(int(n), do_scale=True, rng=r) for n in ns]
    ms, xs, vs = [], [], []
    for k, b in enumerate(pick):
        m, x, v = made[b]
        if k >= base:
            q = np.linalg.qr(r.normal(size=(3, 3)))[0]
            p = r.permutation(len(m))
            x, v = x[p] @ q, v[p] @ q.T
        ms.append(m)
        xs.append(x * 1e-3)
        vs.append(v / math.sqrt(1e-3))
    return (ns[pick].astype(np.int32), np.concatenate(ms), np.concatenate(xs), np.concatenate(vs),
            2 * math.sqrt(2) * 1e-3 ** 1.5)


# ------------------------------------------------------------------- run ---
def run(s):
    c, kind = s["case"], s["kind"]
    if kind == "abi":
        _hold(s)
        h, o = s["sys"], s["out"]
        # the block's particles as their last correction left them, then the
        # force on them at the block's time
        rc = ag.driver().drv_update(c["ni"], _i(s["slots"]), _i(h["ids"]), _d(h["t"]), _d(h["dt"]),
                                    _d(h["m"]), _d(h["x"]), _d(h["v"]), _d(h["a"]), _d(h["j"]))
        if rc:
            raise RuntimeError("drv_update: %d" % rc)
        ag.drive_force(c["n"], s["t"], c["eps2"], s["ids"], s["x"], s["v"], want_nn=c["nn"], out=o)
        return [o["acc"], o["jerk"], o["pot"]] + ([o["nn"]] if c["nn"] else [])
    if kind == "all":
        _library("split")
        _gpu["key"] = None
        ag.drive_load(s["m"], s["x"], s["v"], s["a"], s["j"], ids=s["ids"])
        o = ag.drive_force(c["n"], 0.0, c["eps2"], s["ids"], s["x"], s["v"], want_nn=c["nn"])
        return [o["acc"], o["jerk"], o["pot"]] + ([o["nn"]] if c["nn"] else [])
    if kind == "slots":
        g6 = _hold(s)
        g6.force_slots(s["t"], c["eps2"], c["n"], s["dslots"].data_ptr(), c["ni"],
                       s["acc"].data_ptr(), s["jerk"].data_ptr(), s["pot"].data_ptr(),
                       s["nn"].data_ptr() if c["nn"] else None)
        return [s["acc"], s["jerk"], s["pot"]] + ([s["nn"]] if c["nn"] else [])
    if kind == "dev":
        g6 = _hold(s)
        g6.force_dev(s["t"], c["eps2"], c["n"], c["ni"], s["x"].data_ptr(), s["v"].data_ptr(),
                     s["dslots"].data_ptr(), s["acc"].data_ptr(), s["jerk"].data_ptr(),
                     s["pot"].data_ptr(), s["nn"].data_ptr() if c["nn"] else None)
        return [s["acc"], s["jerk"], s["pot"]] + ([s["nn"]] if c["nn"] else [])
    if kind == "fixed":
        g6 = _library(s["prec"])
        g6.set_fixed_jerk(ag.JERK_HERMITE if c["jerk"] == "hermite" else ag.JERK_SOFTENED)
        g6.fixed_force(c["n"], c["eps2"], s["x"].data_ptr(), s["v"].data_ptr(), s["m"].data_ptr(),
                       s["a"].data_ptr(), s["j"].data_ptr())
        return [s["a"], s["j"]]
    if kind == "run":
        g6 = _library(s["prec"])
        _gpu["key"] = None
        g6.load_particles(s["m"], s["x"], s["v"], ids=s["ids"])
        g6.run_init(c["eps2"], c["eta"])
        g6.run(4.0, c["blocks"])
        o = g6.read_particles(c["n"])
        return [o["pos"], o["vel"], o["acc"], o["jerk"], o["pot"], o["time"], o["timestep"]]
    if kind == "knn":
        ids, d2 = _hold(s).knn(c["n"], c["k"], s["slots"], s["t"])
        return [ids, d2]
    if kind == "adjoint":
        x0, v0, m = (s[q].detach().requires_grad_() for q in "xvm")
        x, v = hermite_fixed(x0, v0, m, eps2=c["eps2"], dt=1.0 / 256, nsteps=c["nsteps"],
                             checkpoint=c["checkpoint"], precision=c["prec"], jerk=c["jerk"])
        (s["w"] * (x * x).sum(1)).sum().backward()
        return [x.detach(), v.detach(), x0.grad, v0.grad, m.grad]
    g6 = _library("split")
    g6.batch_unperturbed(c["unp"])
    o = g6.batch_run(s["ns"], s["t_end"], s["m"], s["x"], s["v"], max_steps=2000000,
                     mode=c["mode"])
    g6.batch_unperturbed(False)
    return [o["pos"], o["vel"], o["t_final"], o["steps"], o["status"]]


# ------------------------------------------------------------------ work ---
def work(case):
    c, kind = case, case["kind"]
    if kind in ("abi", "all", "slots", "dev", "fixed"):
        n = c["n"]
        ni = c.get("ni", n)
        # j: mass, position, velocity (and acceleration, jerk, time where
        # they are predicted); i: position, velocity in, 7 values out
        jb = 56 if kind == "fixed" else 112
        return dict(bytes=float(jb * n + (48 + 56) * ni), flops=60.0 * n * ni)
    if kind == "run":
        n = c["n"]
        ni = 0.011 * n + 1  # active particles of a mean block, near enough
        return dict(bytes=c["blocks"] * (112.0 * n + 210 * ni) + 60 * n,
                    flops=60.0 * n * (n + c["blocks"] * ni))
    if kind == "knn":
        return dict(bytes=c["n"] * 104.0 + c["ni"] * c["k"] * 12.0, flops=8.0 * c["n"] * c["ni"])
    if kind == "adjoint":
        n, k = c["n"], c["nsteps"]
        # the force forward and again backward (checkpoints), its transpose
        return dict(bytes=(3 * k + 2) * 24.0 * 12 * n, flops=(60.0 * (2 * k + 1) + 120.0 * (k + 1)) * n * n)
    if kind == "batch":
        nb = 0.5 * (c["nmin"] + c["nmax"])
        n2 = (nb * nb + (c["nmax"] - c["nmin"]) ** 2 / 12.0)
        return dict(bytes=c["nsys"] * nb * 104, flops=c["nsys"] * n2 * 60 * 3 * 2000 * c["tcr"])
    return dict(bytes=c["nsys"] * 3 * 104.0, flops=c["nsys"] * 9 * 60 * 3 * 25 * c["t_end"])


# ----------------------------------------------------------------- exact ---
def _pairs64(xi, vi, me, xj, vj, m, eps2, jerk="softened"):
    """acc, jerk, pot on i of all j (me: the j that is i itself, or None)."""
    d = xj[None] - xi[:, None]
    w = vj[None] - vi[:, None]
    q = (d * d).sum(-1)
    rinv = (q + (eps2 + TINY)).rsqrt()
    if me is not None:
        rinv = rinv.scatter(1, me[:, None], 0.0)
    rv = (d * w).sum(-1)
    if jerk == "hermite":
        if me is not None:
            q = q.scatter(1, me[:, None], 1.0)
        u = rv / q
    else:
        u = rv * rinv * rinv
    f = m[None] * rinv * rinv * rinv
    acc = torch.einsum("ij,ijk->ik", f, d)
    jk = torch.einsum("ij,ijk->ik", f, w) - 3 * torch.einsum("ij,ijk->ik", f * u, d)
    return acc, jk, -(m[None] * rinv).sum(1)


def _chunks(ni, nj):
    step = max(1, (1 << 25) // nj)
    return [(k, min(ni, k + step)) for k in range(0, ni, step)]


def _all64(xi, vi, me, xj, vj, m, eps2, jerk="softened"):
    got = [_pairs64(xi[a:b], vi[a:b], me[a:b], xj, vj, m, eps2, jerk)
           for a, b in _chunks(len(xi), len(xj))]
    return [torch.cat([g[k] for g in got]) for k in range(3)]


def _force_grad64(x, v, m, eps2, jerk):
    """acc and jerk on all, differentiable, recomputed chunk by chunk."""
    def part(a, b, x, v, m):
        me = torch.arange(a, b, device=x.device)
        return _pairs64(x[a:b], v[a:b], me, x, v, m, eps2, jerk)[:2]
    got = [torch.utils.checkpoint.checkpoint(part, a, b, x, v, m, use_reentrant=False)
           for a, b in _chunks(len(x), len(x))]
    return [torch.cat([g[k] for g in got]) for k in range(2)]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("run", "batch", "scatter"):
        return None
    s = prepare(case, seed)
    if kind in ("abi", "slots", "dev"):
        h = s["sys"]
        n = c["n"]
        xj, vj = (_dev(q) for q in _predict(h, np.arange(n), s["t"]))
        xi, vi = (_dev(q) if isinstance(q, np.ndarray) else q for q in (s["x"], s["v"]))
        o = _all64(xi, vi, _dev(s["slots"].astype(np.int64)), xj, vj, _dev(h["m"]), c["eps2"])
        return o + ([None] if c["nn"] else [])
    if kind == "all":
        x, v = _dev(s["x"]), _dev(s["v"])
        o = _all64(x, v, torch.arange(c["n"], device="cuda"), x, v, _dev(s["m"]), c["eps2"])
        return o + ([None] if c["nn"] else [])
    if kind == "fixed":
        return _all64(s["x"], s["v"], torch.arange(c["n"], device="cuda"), s["x"], s["v"], s["m"],
                      c["eps2"], c["jerk"])[:2]
    if kind == "knn":
        x = _dev(_predict(s["sys"], np.arange(c["n"]), s["t"])[0])
        me = _dev(s["slots"].astype(np.int64))
        got = []
        for a, b in _chunks(c["ni"], c["n"]):
            d = x[me[a:b]][:, None] - x[None]
            q = (d * d).sum(-1).scatter(1, me[a:b, None], math.inf)
            got.append(torch.topk(q, c["k"], dim=1, largest=False, sorted=True)[0])
        return [None, torch.cat(got)]
    # adjoint: the scheme of the hermite code, differentiated by torch
    x0, v0, m = (s[q].detach().requires_grad_() for q in "xvm")
    h = 1.0 / 256
    x, v = x0, v0
    a, j = _force_grad64(x, v, m, c["eps2"], c["jerk"])
    for _ in range(c["nsteps"]):
        xp = x + v * h + a * (h * h / 2) + j * (h ** 3 / 6)
        vp = v + a * h + j * (h * h / 2)
        a1, j1 = _force_grad64(xp, vp, m, c["eps2"], c["jerk"])
        v1 = v + (a + a1) * (h / 2) + (j - j1) * (h * h / 12)
        x = x + (v + v1) * (h / 2) + (a - a1) * (h * h / 12)
        v, a, j = v1, a1, j1
    (s["w"] * (x * x).sum(1)).sum().backward()
    return [x.detach(), v.detach(), x0.grad, v0.grad, m.grad]
