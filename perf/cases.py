"""The engine's performance cases: the calls that a user's program makes, over their real range.

listed() and draw() name the cases, prepare() makes what a program holds before
the call (a context with a state, pinned host buffers for what it reads back),
run() is one pass through the public entry points, work() what a pass cannot do
without and exact() the same results in plain 64-bit torch.

Kinds of cases:
  step     lj_gpu_step for `steps` steps with a record per step, then the state
           read back (lj_gpu_download_state); with `rdf` also one sample of the
           radial distribution per pass, accumulated on the device
  forces   new positions in, forces, energy and virial out (upload_state,
           compute_forces, download_state)
  batch    lj_batch_step over a sweep of systems of uneven size, records and
           every system's state read back
  adjoint  AdjointNVE.forward and .backward
  rdf      lj_gpu_rdf_noalloc on a caller's device buffers
States are FCC lattices (the engine's initial condition) with every atom moved
off its site by up to 6 % of the lattice constant per axis and Maxwell-Boltzmann
velocities, so that a system melts, diffuses and rebuilds its lists as it runs.
"""

import ctypes
import math
import pathlib
import random
import sys

import numpy as np
import torch

_PKG = str(pathlib.Path(__file__).resolve().parents[1] / "lennard-jonesium_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from lennardjonesium import AdjointNVE  # noqa: E402
from lennardjonesium import _native as nat  # noqa: E402

RC, DT = 2.5, 0.005


def listed():
    return [
        # a program that drives the integrator one step at a time (its own thermostat or
        # analysis between steps): the argon system of the tests, one step a call
        dict(name="step1_864_fp64", kind="step", N=864, rho=0.8442, T=0.722, precision="fp64", steps=1, rdf=False,
             slab=False),
        # a box of 2 cells per axis (the size of the Python package's own test runs), where
        # the list carries explicit images and is rebuilt every step; the single small
        # run of the example notebook; one run of a density/temperature sweep.  200 steps
        # between the control protocol's temperature checks
        dict(name="nve_256_smallbox", kind="step", N=256, rho=0.8, T=0.8, precision="fp64", steps=200, rdf=False,
             slab=False),
        dict(name="nve_500_fp64", kind="step", N=500, rho=0.8, T=0.8, precision="fp64", steps=200, rdf=False,
             slab=False),
        dict(name="nve_4000_fp64", kind="step", N=4000, rho=0.8, T=1.2, precision="fp64", steps=200, rdf=False,
             slab=False),
        # an ordinary liquid of a size that is no multiple of anything, mixed precision
        dict(name="nve_31987_mixed", kind="step", N=31987, rho=0.8442, T=1.0, precision="mixed", steps=200, rdf=False,
             slab=False),
        # the benchmark's system on both paths
        dict(name="nve_1m_fp64", kind="step", N=1048576, rho=0.8442, T=1.0, precision="fp64", steps=200, rdf=False,
             slab=False),
        dict(name="nve_1m_mixed", kind="step", N=1048576, rho=0.8442, T=1.0, precision="mixed", steps=200, rdf=False,
             slab=False),
        # the long run: 4 million atoms, a radial distribution sample every 100 steps
        dict(name="long_4m_mixed_rdf", kind="step", N=4000000, rho=0.8, T=0.9, precision="mixed", steps=100, rdf=True,
             slab=False),
        # 64 systems of 500 to 32 000 atoms over an 8 x 8 grid of (T, rho), advanced together
        dict(name="sweep_64", kind="batch", systems=64, n_min=5, n_max=20, pick=12345, steps=200),
        # gradients of time averages with respect to the start and the potential's parameters
        dict(name="adjoint_4000", kind="adjoint", N=4000, rho=0.8, T=1.2, steps=200, every=20),
        # forces of configurations that another program makes, in a flat box
        dict(name="forces_107k_slab", kind="forces", N=107001, rho=0.7, T=1.0, precision="fp64", slab=True),
        # an analysis hook on positions that are on the GPU already
        dict(name="rdf_100k", kind="rdf", N=100003, rho=0.8442, bins=200, rmax=4.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "batch", "adjoint", "forces", "rdf"])
    if kind == "step":
        precision = rng.choice(["fp64", "fp64", "mixed"])
        N = _log(rng, 200, 2000000)
        # steps between two looks at the system; at most the largest listed case's atom-steps
        steps = min(_log(rng, 1, 200), max(1, 160000000 // N))
        return dict(kind=kind, N=N, rho=round(rng.uniform(0.3, 1.0), 4), T=round(rng.uniform(0.5, 2.0), 3),
                    precision=precision, steps=steps, rdf=rng.random() < 0.2 and N > 4000, slab=rng.random() < 0.2 and N > 8000)
    if kind == "batch":
        return dict(kind=kind, systems=rng.randint(2, 64), n_min=5, n_max=rng.randint(7, 20), pick=rng.randrange(1 << 20),
                    steps=_log(rng, 10, 200))
    if kind == "adjoint":
        return dict(kind=kind, N=_log(rng, 700, 12000), rho=round(rng.uniform(0.5, 0.85), 4), T=round(rng.uniform(0.7, 1.5), 3),
                    steps=rng.randint(20, 200), every=rng.randint(5, 40))
    if kind == "forces":
        return dict(kind=kind, N=_log(rng, 500, 1000000), rho=round(rng.uniform(0.3, 1.0), 4), T=1.0,
                    precision=rng.choice(["fp64", "mixed"]), slab=rng.random() < 0.5)
    return dict(kind="rdf", N=_log(rng, 2000, 131072), rho=round(rng.uniform(0.3, 1.0), 4), bins=rng.randint(50, 600),
                rmax=round(rng.uniform(2.5, 4.5), 2))


# ---- states ---------------------------------------------------------------

def _cells(N, slab):
    """FCC cells per axis with at least N sites (a slab: a third as high as wide)."""
    m = math.ceil(N / 4)
    if not slab:
        n = max(1, round(m ** (1 / 3)))
        while n ** 3 < m:
            n += 1
        while n > 1 and (n - 1) ** 3 >= m:
            n -= 1
        return n, n, n
    h = max(1, round((m / 9) ** (1 / 3)))
    w = math.ceil(math.sqrt(m / h))
    return w, math.ceil(m / (h * w)), h


def _start(N, rho, T, seed, slab=False):
    """Positions and velocities (N x 4 on the GPU) and the box of N atoms at density rho."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz = _cells(N, slab)
    a = (N / (nx * ny * nz * rho)) ** (1 / 3)
    box = torch.tensor([nx * a, ny * a, nz * a], dtype=torch.float64, device="cuda")
    sites = 4 * nx * ny * nz
    # which sites are empty, when N is not 4 nx ny nz
    s = torch.arange(N, device="cuda") if sites == N else \
        torch.randperm(sites, generator=g, device="cuda")[:N].sort().values
    cell, b = s // 4, s % 4
    ijk = torch.stack([cell // (ny * nz), (cell // nz) % ny, cell % nz], 1).double()
    basis = torch.tensor([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]], dtype=torch.float64, device="cuda")
    x = torch.zeros(N, 4, dtype=torch.float64, device="cuda")
    v = torch.zeros(N, 4, dtype=torch.float64, device="cuda")
    jit = torch.rand(N, 3, dtype=torch.float64, device="cuda", generator=g) * 0.12 - 0.06
    p = (ijk + basis[b] + 0.25 + jit) * a
    x[:, :3] = p - torch.floor(p / box) * box
    u = torch.randn(N, 3, dtype=torch.float64, device="cuda", generator=g)
    v[:, :3] = (u - u.mean(0)) * math.sqrt(T)
    return x, v, [float(e) for e in box]


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


class _Context:
    """An engine context and the pinned buffers that its owner reads the state into."""

    def __init__(self, N, box, precision):
        self.lib, self.N, self.h = nat.lib(), N, ctypes.c_void_p()
        p = nat.Params()
        self.lib.lj_gpu_default_params(ctypes.byref(p))
        p.particle_count = N
        p.box[0], p.box[1], p.box[2] = box
        p.cutoff_distance, p.time_delta = RC, DT
        p.precision = nat.LJ_PRECISION_MIXED if precision == "mixed" else nat.LJ_PRECISION_FP64
        nat.check(self.lib.lj_gpu_create(ctypes.byref(p), ctypes.byref(self.h)))
        self.x, self.v, self.F = (torch.zeros(N, 4, dtype=torch.float64, pin_memory=True) for _ in range(3))

    def upload(self, x, v):
        nat.check(self.lib.lj_gpu_upload_state(self.h, _ptr(x), _ptr(v) if v is not None else None, None, None, 4,
                                               0.0, 0.0, 0.0), self.h)

    def download(self):
        nat.check(self.lib.lj_gpu_download_state(self.h, _ptr(self.x), _ptr(self.v), None, _ptr(self.F), 4, None, None,
                                                 None), self.h)

    def __del__(self):
        if self.h:
            self.lib.lj_gpu_destroy(self.h)
            self.h = ctypes.c_void_p()


class _Batch:
    """A batch of systems and the pinned buffers of their states."""

    def __init__(self, boxes, counts):
        self.lib, self.h, self.n = nat.lib(), ctypes.c_void_p(), len(counts)
        table = (nat.BatchSystem * self.n)()
        for q, box, N in zip(table, boxes, counts):
            q.particle_count, q.time_delta, q.skin = N, DT, -1.0
            q.box[0], q.box[1], q.box[2] = box
        nat.check(self.lib.lj_batch_create(table, self.n, RC, 0, ctypes.byref(self.h)))
        self.x, self.v, self.F = (torch.zeros(sum(counts), 4, dtype=torch.float64, pin_memory=True) for _ in range(3))
        self.at = np.concatenate([[0], np.cumsum(counts)]).tolist()

    def check(self, status):
        if status != nat.LJ_OK:
            raise nat.LJError(status, self.lib.lj_batch_last_error(self.h).decode())

    def __del__(self):
        if self.h:
            self.lib.lj_batch_destroy(self.h)
            self.h = ctypes.c_void_p()


def _sweep(case):
    """(N, rho, T) of a batch's systems: T outer, rho inner over a square grid."""
    r = random.Random(case["pick"])
    side = math.ceil(math.sqrt(case["systems"]))
    at = lambda lo, hi, k: lo + (hi - lo) * k / max(1, side - 1)  # noqa: E731
    return [(4 * r.randint(case["n_min"], case["n_max"]) ** 3, at(0.05, 1.0, k % side), at(0.5, 2.0, k // side))
            for k in range(case["systems"])]


# ---- one pass ---------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        starts = [_start(N, rho, T, seed * 1009 + k) for k, (N, rho, T) in enumerate(_sweep(case))]
        b = _Batch([s[2] for s in starts], [s[0].shape[0] for s in starts])
        for k, (x, v, _) in enumerate(starts):
            xh, vh = _pinned(x), _pinned(v)
            b.check(b.lib.lj_batch_upload_system(b.h, k, _ptr(xh), _ptr(vh), 4))
        return dict(kind=kind, b=b, steps=case["steps"])
    x, v, box = _start(case["N"], case["rho"], case.get("T", 1.0), seed, case.get("slab", False))
    if kind == "adjoint":
        e = AdjointNVE(case["N"], box, case["steps"], checkpoint_every=case["every"], time_delta=DT)
        return dict(kind=kind, e=e, x=x[:, :3].cpu().numpy().copy(), v=v[:, :3].cpu().numpy().copy())
    if kind == "rdf":
        edges = np.array(box)
        return dict(kind=kind, lib=nat.lib(), x=x, box=edges, bins=case["bins"], rmax=min(case["rmax"], 0.5 * edges.min()),
                    hist=torch.zeros(case["bins"], dtype=torch.int64, device="cuda"),
                    stream=torch.cuda.current_stream().cuda_stream)
    c = _Context(case["N"], box, case["precision"])
    xh, vh = _pinned(x), _pinned(v)
    if kind == "forces":
        return dict(kind=kind, c=c, x=xh)
    c.upload(xh, vh)
    return dict(kind=kind, c=c, steps=case["steps"], rdf=min(4.0, 0.5 * min(box)) if case["rdf"] else 0.0)


def run(state):
    kind = state["kind"]
    if kind == "step":
        c = state["c"]
        records = np.zeros((state["steps"], 7))
        nat.check(c.lib.lj_gpu_step(c.h, state["steps"], records.ctypes.data), c.h)
        out = dict(records=records, x=c.x, v=c.v, F=c.F)
        if state["rdf"]:
            hist = np.zeros(200, dtype=np.uint64)
            nat.check(c.lib.lj_gpu_rdf_accumulate(c.h, 200, state["rdf"]), c.h)
            nat.check(c.lib.lj_gpu_rdf_read(c.h, hist.ctypes.data, None), c.h)
            out["rdf"] = hist.astype(np.int64)
        c.download()
        return out
    if kind == "forces":
        c = state["c"]
        pe, virial = ctypes.c_double(), ctypes.c_double()
        c.upload(state["x"], None)
        nat.check(c.lib.lj_gpu_compute_forces(c.h, ctypes.byref(pe), ctypes.byref(virial)), c.h)
        nat.check(c.lib.lj_gpu_download_state(c.h, None, None, None, _ptr(c.F), 4, None, None, None), c.h)
        return dict(F=c.F, pe=pe.value, virial=virial.value)
    if kind == "batch":
        b = state["b"]
        records = np.zeros((state["steps"], b.n, 7))
        b.check(b.lib.lj_batch_step(b.h, state["steps"], records.ctypes.data))
        for k in range(b.n):
            at = b.at[k] * 32
            b.check(b.lib.lj_batch_download_system(b.h, k, ctypes.c_void_p(b.x.data_ptr() + at),
                                                   ctypes.c_void_p(b.v.data_ptr() + at),
                                                   ctypes.c_void_p(b.F.data_ptr() + at), 4))
        return dict(records=records, x=b.x, v=b.v, F=b.F)
    if kind == "adjoint":
        pe, p, series = state["e"].forward(state["x"], state["v"])
        g = state["e"].backward(1.0, 1.0)
        return dict(pe=pe, p=p, series=series, dx=g["x0"], dv=g["v0"], deps=g["epsilon"], dsigma=g["sigma"])
    s = state
    nat.check(s["lib"].lj_gpu_rdf_noalloc(_ptr(s["x"]), s["x"].shape[0], s["box"].ctypes.data, s["bins"], float(s["rmax"]),
                                          _ptr(s["hist"]), ctypes.c_void_p(s["stream"])))
    return s["hist"]


def work(case):
    """Half-shell pair arithmetic (30 flops a pair inside the cutoff) and the state's traffic: x, v, F and the
    displacement read and written once a step (216 bytes an atom)."""
    kind = case["kind"]
    pairs = lambda N, rho, r: 0.5 * N * rho * 4 / 3 * math.pi * r ** 3  # noqa: E731
    if kind == "batch":
        sys_ = _sweep(case)
        return {"bytes": case["steps"] * sum(216 * N for N, _, _ in sys_),
                "flops": case["steps"] * sum(30 * pairs(N, rho, RC) for N, rho, _ in sys_)}
    N, rho = case["N"], case["rho"]
    if kind == "step":
        n = case["steps"]
        flops = n * 30 * pairs(N, rho, RC) + (10 * pairs(N, rho, 4.0) if case["rdf"] else 0)
        return {"bytes": n * 216 * N + 96 * N, "flops": flops}
    if kind == "forces":
        return {"bytes": 64 * N, "flops": 30 * pairs(N, rho, RC)}
    if kind == "adjoint":
        # forward, the segments' second forward, and the Hessian-vector product with its parameter terms
        n = case["steps"]
        return {"bytes": n * N * (2 * 96 + 144), "flops": n * pairs(N, rho, RC) * (30 + 30 + 90)}
    return {"bytes": 32 * N + 8 * case["bins"], "flops": 10 * pairs(N, rho, case["rmax"])}


# ---- the same in plain 64-bit torch ------------------------------------------

def _neighbours(x, box, reach):
    """Padded neighbour table (N x K, -1 where empty) of all pairs within reach."""
    N, dev = x.shape[0], x.device
    n = [int(e // reach) for e in box]
    L = torch.tensor(box, dtype=torch.float64, device=dev)
    if min(n) < 3 or N < 3000:
        cand = torch.arange(N, device=dev).expand(N, N)
        rows = [(0, N, cand)]
    else:
        nn = torch.tensor(n, device=dev)
        c = torch.minimum((x / L * nn).long().clamp(min=0), nn - 1)
        flat = (c[:, 0] * n[1] + c[:, 1]) * n[2] + c[:, 2]
        order = flat.argsort(stable=True)
        count = torch.bincount(flat, minlength=n[0] * n[1] * n[2])
        first = count.cumsum(0) - count
        table = torch.full((len(count), int(count.max())), -1, dtype=torch.long, device=dev)
        table[flat[order], torch.arange(N, device=dev) - first[flat[order]]] = order
        off = torch.cartesian_prod(*[torch.tensor([-1, 0, 1], device=dev)] * 3)
        step = max(1, 200_000_000 // (27 * table.shape[1] * 32))
        rows = []
        for a in range(0, N, step):
            cc = (c[a:a + step, None, :] + off) % nn
            rows.append((a, min(N, a + step), table[(cc[..., 0] * n[1] + cc[..., 1]) * n[2] + cc[..., 2]].flatten(1)))
    out = []
    for a, b, cand in rows:
        d = x[a:b, None, :] - x[cand[a:b] if cand.shape[0] != b - a else cand]
        d = d - torch.round(d / L) * L
        ok = ((d * d).sum(-1) < reach * reach) & (cand >= 0) & (cand != torch.arange(a, b, device=dev)[:, None])
        k = int(ok.sum(1).max())
        out.append(torch.where(ok, cand, -1).topk(max(k, 1), dim=1).values)
    K = max(o.shape[1] for o in out)
    return torch.cat([torch.nn.functional.pad(o, (0, K - o.shape[1]), value=-1) for o in out])


def _lj(q, hit, eps=1.0, sigma=1.0):
    """Energy and virial of pairs at squared distance q (0 where not hit): the spline-truncated potential."""
    uc2 = RC * RC
    m6 = 1 / uc2 ** 3
    alpha, beta = -4 * m6 * (m6 - 1), 12 * m6 * (2 * m6 - 1)
    q = torch.where(hit, q, torch.ones_like(q))
    s6 = (sigma * sigma / q) ** 3
    z = q / (uc2 * sigma * sigma)
    zero = torch.zeros_like(q)
    V = torch.where(hit, eps * (4 * s6 * (s6 - 1) + alpha + beta * (z - 1)), zero)
    W = torch.where(hit, eps * (24 * s6 * (2 * s6 - 1) - 2 * beta * z), zero)
    return V, W, q


def _sep(x, nb, L):
    """Separations (periodic; in a box under 3 cutoffs, of the nearest image) and which are inside the cutoff."""
    d = x[:, None, :] - x[nb.clamp(min=0)]
    d = d - torch.round(d.detach() / L) * L
    q = (d * d).sum(-1)
    return d, q, (q < RC * RC) & (nb >= 0)


def _forces(x, nb, L):
    N, F, pe, w = x.shape[0], [], 0.0, 0.0
    step = max(1, 40_000_000 // nb.shape[1])
    for a in range(0, N, step):
        d = x[a:a + step, None, :] - x[nb[a:a + step].clamp(min=0)]
        d = d - torch.round(d / L) * L
        q = (d * d).sum(-1)
        V, W, q = _lj(q, (q < RC * RC) & (nb[a:a + step] >= 0))
        F.append(((W / q)[..., None] * d).sum(1))
        pe, w = pe + 0.5 * V.sum(), w + 0.5 * W.sum()
    return torch.cat(F), pe, w


def _trajectory(x, v, box, steps, F=None):
    """`steps` steps of velocity Verlet from (x, v) with no force on the first half kick, as the engine starts from an
    uploaded state without forces: records, x, v, F."""
    L = torch.tensor(box, dtype=torch.float64, device=x.device)
    x, v, disp = x[:, :3].clone(), v[:, :3].clone(), torch.zeros_like(x[:, :3])
    F, N, skin = torch.zeros_like(x), x.shape[0], 0.4
    nb, ref, t, rec = None, None, 0.0, []
    for _ in range(steps):
        v = v + 0.5 * F * DT
        x, disp, t = x + v * DT, disp + v * DT, t + DT
        x = x - torch.floor(x / L) * L
        if nb is None or float(((disp - ref) ** 2).sum(1).max()) > (skin / 2) ** 2:
            nb, ref = _neighbours(x, box, RC + skin), disp.clone()
        F, pe, w = _forces(x, nb, L)
        v = v + 0.5 * F * DT
        ke = 0.5 * (v * v).sum()
        rec.append(torch.stack([torch.tensor(t, dtype=torch.float64, device=x.device), ke, pe, pe + ke, w,
                                2 / 3 * ke / N, (disp * disp).sum() / N]))
    return torch.stack(rec), x, v, F


def _four(t):
    return torch.nn.functional.pad(t, (0, 1)).cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "rdf":
        return None  # counts
    if kind == "batch":
        got = []
        for k, (N, rho, T) in enumerate(_sweep(case)):
            x, v, box = _start(N, rho, T, seed * 1009 + k)
            if min(box) < 2 * (RC + 0.4) or case["steps"] * case["systems"] > 13000:
                return None
            got.append(_trajectory(x, v, box, case["steps"]))
        return dict(records=torch.stack([g[0] for g in got], 1).cpu().numpy(),
                    **{n: torch.cat([_four(g[q]) for g in got]) for n, q in (("x", 1), ("v", 2), ("F", 3))})
    x, v, box = _start(case["N"], case["rho"], case.get("T", 1.0), seed, case.get("slab", False))
    if kind == "adjoint":
        return _adjoint(x[:, :3].clone(), v[:, :3].clone(), box, case["steps"])
    if min(box) < 2 * (RC + 0.4) or case["N"] * case.get("steps", 1) > 220_000_000:
        return None  # the nearest image is not enough, or it takes too long
    if kind == "forces":
        L = torch.tensor(box, dtype=torch.float64, device=x.device)
        F, pe, w = _forces(x[:, :3], _neighbours(x[:, :3], box, RC), L)
        return dict(F=_four(F), pe=float(pe), virial=float(w))
    rec, x, v, F = _trajectory(x, v, box, case["steps"])
    out = dict(records=rec.cpu().numpy(), x=_four(x), v=_four(v), F=_four(F))
    return dict(out, rdf=None) if case["rdf"] else out


def _adjoint(x0, v0, box, steps):
    """Time averages of the energy and the pressure and their gradients, by differentiating through the steps."""
    N = x0.shape[0]
    if N * steps > 1_000_000:
        return None  # what autograd keeps does not fit beside everything else
    L = torch.tensor(box, dtype=torch.float64, device=x0.device)
    rho, skin = N / math.prod(box), 0.3
    one = torch.ones((), dtype=torch.float64, device=x0.device)
    x0, v0, eps, sigma = (t.clone().requires_grad_() for t in (x0, v0, one, one))

    def forces(x, nb):
        d, q, hit = _sep(x, nb, L)
        # the cutoff follows sigma; which pairs are inside does not
        V, W, q = _lj(q, hit, eps, sigma)
        return ((W / q)[..., None] * d).sum(1), 0.5 * V.sum(), 0.5 * W.sum()

    x, v, at, ref = x0, v0, x0.detach(), None
    nb, ref = _neighbours(at, box, RC + skin), at
    F, series, pe_sum, p_sum = forces(x, nb)[0], [], 0.0, 0.0
    for _ in range(steps):
        h = v + 0.5 * F * DT
        x = x + h * DT
        with torch.no_grad():
            moved = x - ref
        if float((moved ** 2).sum(1).max()) > (skin / 2) ** 2:
            ref = x.detach().clone()
            nb = _neighbours(ref - torch.floor(ref / L) * L, box, RC + skin)
        F, pe, w = forces(x, nb)
        v = h + 0.5 * F * DT
        ke = 0.5 * (v * v).sum()
        p = rho * (2 / 3 * ke / N + w / (3 * N))
        series.append(torch.stack([pe, w, ke, p]).detach())
        pe_sum, p_sum = pe_sum + pe, p_sum + p
    pe, p = pe_sum / steps, p_sum / steps
    (pe + p).backward()
    return dict(pe=float(pe), p=float(p), series=torch.stack(series).cpu().numpy(), dx=x0.grad.cpu().numpy(),
                dv=v0.grad.cpu().numpy(), deps=float(eps.grad), dsigma=float(sigma.grad))
