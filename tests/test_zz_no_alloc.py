"""g6x_force_dev_noalloc: the force entry point that allocates no device
memory (for callers whose device memory is owned by a host framework, or
whose step loop cannot absorb cudaMalloc's synchronisation).  Its split-j
partial sums live in a fixed 16 MiB array inside the library.

Checked through the C ABI against g6x_force_dev (the allocating entry point)
on the same inputs, twice in a row (the shared array keeps the previous
call's contents), in both precisions and with and without the nearest
neighbour: the launch shape and the fixed-order merge are the same, so the
results must be bit-identical.  This file is collected last so that a run
stopping at the first failure has already run every other test."""
import os
import subprocess
import sys

import numpy as np
import pytest

import amuse_gb300 as ag
from amuse_gb300 import ic

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("want_nn", [True, False], ids=["nn", "no-nn"])
@pytest.mark.parametrize("prec", [ag.SPLIT, ag.FP64], ids=["split", "fp64"])
def test_noalloc_matches_allocating_entry_point(g6, prec, want_nn):
    torch = pytest.importorskip("torch")
    g6.set_precision(prec)
    try:
        np.random.seed(31)
        nj = 20000
        m, x, v = ic.plummer(nj)
        g6.load_particles(m, x, v)
        outs = []
        for seed, ni in ((1, 1000), (2, 1000)):  # two calls in a row, new inputs each time
            rng = np.random.RandomState(seed)
            sel = np.sort(rng.choice(nj, ni, replace=False)).astype(np.int32)
            dx = torch.tensor(x[sel], device="cuda").contiguous()
            dv = torch.tensor(v[sel], device="cuda").contiguous()
            ds = torch.tensor(sel, device="cuda")
            res = {}
            for name in ("alloc", "noalloc"):
                da = torch.full((ni, 3), float("nan"), dtype=torch.float64, device="cuda")
                dj = torch.full_like(da, float("nan"))
                dp = torch.full((ni,), float("nan"), dtype=torch.float64, device="cuda")
                dn = torch.full((ni,), -7, dtype=torch.int32, device="cuda") if want_nn else None
                torch.cuda.synchronize()
                f = g6.force_dev if name == "alloc" else g6.force_dev_noalloc
                f(0.0, 1e-4, nj, ni, dx.data_ptr(), dv.data_ptr(), ds.data_ptr(), da.data_ptr(),
                  dj.data_ptr(), dp.data_ptr(), dn.data_ptr() if want_nn else None, sync=True)
                res[name] = dict(acc=da.cpu().numpy(), jerk=dj.cpu().numpy(),
                                 pot=dp.cpu().numpy())
                if want_nn:
                    res[name]["nn"] = dn.cpu().numpy()
            # the scratch array is actually used: this shape splits j across CTAs
            assert g6.stats()["nsplit"] > 1
            a, b = res["alloc"], res["noalloc"]
            assert np.all(np.isfinite(b["acc"])) and np.all(np.isfinite(b["pot"]))
            for k in a:
                assert np.array_equal(b[k], a[k]), k
            if want_nn:
                assert np.all(b["nn"] >= 0)
            outs.append(b)
        assert not np.array_equal(outs[0]["pot"], outs[1]["pot"])
    finally:
        g6.set_precision(ag.SPLIT)


def test_noalloc_refuses_oversized_scratch(g6):
    torch = pytest.importorskip("torch")
    g6.set_precision(ag.SPLIT)
    np.random.seed(32)
    n = 131072
    m, x, v = ic.plummer(n)
    g6.load_particles(m, x, v)
    dx = torch.tensor(x, device="cuda").contiguous()
    dv = torch.tensor(v, device="cuda").contiguous()
    da = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    dj = torch.empty_like(da)
    dp = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    # all 131072 i against 131072 j splits j 13 ways: ~100 MB of partials
    with pytest.raises(ag.G6Error, match="scratch"):
        g6.force_dev_noalloc(0.0, 1e-6, n, n, dx.data_ptr(), dv.data_ptr(), None, da.data_ptr(),
                             dj.data_ptr(), dp.data_ptr(), None, sync=True)


@pytest.mark.parametrize("ni,nj", [(226304, 226560), (225280, 262144)])
def test_noalloc_takes_unsplit_shapes(g6, ni, nj):
    """So many i that one split of j fills the GPU, and whose partial records
    would not fit the fixed array if j were split: no scratch, no refusal."""
    torch = pytest.importorskip("torch")
    g6.set_precision(ag.SPLIT)
    np.random.seed(34)
    m, x, v = ic.plummer(nj)
    g6.load_particles(m, x, v)
    new = lambda *s: torch.full(s, float("nan"), dtype=torch.float64, device="cuda")
    dx, dv = (torch.tensor(q[:ni], device="cuda").contiguous() for q in (x, v))
    ds = torch.arange(ni, dtype=torch.int32, device="cuda")
    out = []
    for f in (g6.force_dev_noalloc, g6.force_dev):
        o = new(ni, 3), new(ni, 3), new(ni)
        torch.cuda.synchronize()
        f(0.0, 1e-4, nj, ni, dx.data_ptr(), dv.data_ptr(), ds.data_ptr(),
          *(q.data_ptr() for q in o), None, sync=True)
        assert g6.stats()["nsplit"] == 1
        out.append(o)
    assert all(torch.equal(a, b) for a, b in zip(*out)) and torch.isfinite(out[0][0]).all()


# A process of its own: the library keeps an update buffer once it has one.
STAGED = """
import numpy as np, torch
import amuse_gb300 as ag
from amuse_gb300 import ic
n, first = {n}, 512
g6 = ag.G6X(0)
np.random.seed(33)
m, x, v = ic.plummer(n)
ids = np.arange(1, n + 1)
ag.drive_load(m[:first], x[:first], v[:first], ids=ids[:first])
ag.drive_force(first, 0.0, 1e-4, ids[:8], x[:8], v[:8])  # applies them: fewer than 1024
ag.drive_load(2 * m, x, v, ids=ids)                        # staged when the call comes
new = lambda *s: torch.full(s, float("nan"), dtype=torch.float64, device="cuda")
dx, dv = (torch.tensor(q[:64], device="cuda").contiguous() for q in (x, v))
ds = torch.arange(64, dtype=torch.int32, device="cuda")
out = []
for f in (g6.force_dev_noalloc, g6.force_dev):
    o = new(64, 3), new(64, 3), new(64)
    torch.cuda.synchronize()
    f(0.0, 1e-4, n, 64, dx.data_ptr(), dv.data_ptr(), ds.data_ptr(), *(q.data_ptr() for q in o),
      None, sync=True)
    out.append([q.cpu().numpy() for q in o])
assert all(np.array_equal(a, b) for a, b in zip(*out))
rel = x - x[0]
r = np.sqrt((rel[1:] ** 2).sum(1) + 1e-4)
assert abs(out[0][2][0] + (2 * m[1:] / r).sum()) < 1e-5 * abs(out[0][2][0])
"""


@pytest.mark.parametrize("n", [512, 2000], ids=["read-in-place", "by-copy"])
def test_noalloc_takes_staged_updates(lib_built, n):
    """Updates staged before the call are taken where every earlier flush was
    small enough to be read in place, as many as the staging ring held."""
    r = subprocess.run([sys.executable, "-c", STAGED.format(n=n)], cwd=ROOT, text=True,
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
