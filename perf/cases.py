"""Performance cases of the sweep: what a program that uses this framework has it do.

Every case is one call sequence through the public binding (a Sweeper on
device-resident state, the iteration loop on host buffers, or a batch of
independent problems), with the state drawn U[0, 1) and the transform matrices
of the random-input study (a_from_m ~ N(0, 1/nm), m_from_a its
pseudo-inverse); the boundary fluxes are the built-in ones.
"""
import math

import numpy as np
import torch

import minisweep_b200 as msb

NU = 4
NOCT = 8


def _sweep(name, nx, ny, nz, ne, na, nm, precision=0, norms=False):
    return dict(name=name, kind="sweep", nx=nx, ny=ny, nz=nz, ne=ne, na=na, nm=nm, precision=precision, norms=norms)


def listed():
    return [
        # the driver's default flags (5^3 cells, 30 groups, 33 angles): the smallest call a user makes, all latency
        _sweep("default_flags", 5, 5, 5, 30, 33, 16),
        # the headline configuration cut down to what the CPU build runs, with the driver's closing norms
        _sweep("cpu_headline_norms", 16, 16, 16, 16, 32, 4, norms=True),
        # an ordinary mid-size problem
        _sweep("mid", 32, 32, 32, 16, 32, 16),
        # odd everything: cells that no tile divides, an odd group count, a ragged second angle pass, 8 moments
        _sweep("ragged", 37, 29, 41, 23, 45, 8),
        # the headline benchmark configuration
        _sweep("headline", 64, 64, 64, 64, 32, 16),
        # the angle- and group-heavy geometry, four angle passes
        _sweep("dense", 32, 32, 96, 128, 128, 16),
        # mixed precision, FP16 halves, at the headline grid
        _sweep("mixed_fp16", 64, 64, 64, 16, 32, 16, precision=1),
        # mixed precision, BF16 halves, odd sizes and two angle passes
        _sweep("mixed_bf16_ragged", 45, 50, 39, 11, 64, 16, precision=2),
        # the driver's iteration loop from and to pinned host buffers, two iterations
        dict(name="host_iterations", kind="iterations", nx=32, ny=32, nz=32, ne=64, na=32, nm=16, niter=2),
        # many small problems in one launch (the batch API's serving workload)
        dict(name="batch_small", kind="batch", n=128, which="small", draw_seed=11),
        # fewer, larger problems of uneven sizes in one launch
        dict(name="batch_serving", kind="batch", n=12, which="serving", draw_seed=7),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _updates(c):
    return c["nx"] * c["ny"] * c["nz"] * c["ne"] * c["na"]


def draw(rng):
    """One more case of the ranges above; no larger than the largest listed one."""
    kind = rng.choice(["sweep"] * 5 + ["mixed"] * 2 + ["iterations", "batch"])
    if kind == "batch":
        which = rng.choice(["small", "serving"])
        n = _log_int(rng, 16, 160) if which == "small" else _log_int(rng, 2, 12)
        return dict(kind="batch", n=n, which=which, draw_seed=rng.randrange(1, 1 << 20))
    most = 64 ** 3 * 64 * 32 if kind == "sweep" else 64 ** 3 * 16 * 32 if kind == "mixed" else 32 ** 3 * 64 * 32
    while True:
        c = dict(kind="sweep" if kind == "mixed" else kind, nx=_log_int(rng, 3, 72), ny=_log_int(rng, 3, 72),
                 nz=_log_int(rng, 3, 96), ne=_log_int(rng, 1, 128), na=rng.choice([7, 16, 24, 32, 32, 33, 48, 64, 100, 128]),
                 nm=rng.choice([4, 8, 16, 16]))
        state = c["nx"] * c["ny"] * c["nz"] * c["ne"] * c["nm"] * NU * 8
        if 20000 <= _updates(c) <= most and state <= (9 << 30 if kind == "sweep" else 9 << 28):
            break
    if kind == "iterations":
        c["niter"] = rng.choice([1, 2])
    else:
        c["precision"] = rng.choice([1, 2]) if kind == "mixed" else 0
        c["norms"] = kind == "sweep" and rng.random() < 0.25
    return c


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _state(n, seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return torch.rand(n, generator=g, dtype=torch.float64, device=_device())


def _matrices(nm, na, seed):
    """a_from_m[oct][im][ia] ~ N(0, 1/nm), m_from_a[oct][ia][im] its pseudo-inverse."""
    rng = np.random.Generator(np.random.PCG64(seed))
    a, m = np.zeros((NOCT, nm, na)), np.zeros((NOCT, na, nm))
    for o in range(NOCT):
        w = rng.normal(0.0, 1.0 / np.sqrt(nm), size=(na, nm))
        a[o] = w.T
        m[o] = np.linalg.pinv(w).T
    return a, m


def _nstate(c):
    return c["nx"] * c["ny"] * c["nz"] * c["ne"] * c["nm"] * NU


def _flags(c):
    s = f"--ncell_x {c['nx']} --ncell_y {c['ny']} --ncell_z {c['nz']} --ne {c['ne']} --na {c['na']}"
    return s + (f" --precision {c['precision']}" if c.get("precision") else "")


def _batch_problems(c):
    """Sizes of a batch's problems, in the ranges of the two batch workloads."""
    rng = np.random.Generator(np.random.PCG64(c["draw_seed"]))
    out = []
    for _ in range(c["n"]):
        if c["which"] == "small":
            nx, ny, nz = (int(rng.integers(4, h)) for h in (13, 13, 17))
            ne, na = int(rng.choice([2, 4, 8])), int(rng.choice([16, 32]))
        else:
            nx, ny, nz = (int(rng.integers(8, h)) for h in (49, 49, 65))
            ne, na = int(rng.choice([8, 16, 32, 64])), int(rng.choice([16, 32, 64]))
        out.append(dict(nx=nx, ny=ny, nz=nz, ne=ne, na=na, nm=int(rng.choice([4, 16]))))
    return out


# ------------------------------------------------------- prepare, run, work
def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        problems = _batch_problems(c)
        total = sum(_nstate(p) for p in problems)  # all states in one array, one after another
        vi = _state(total, seed)
        vo = torch.empty_like(vi)
        mats, descs, at = [], [], 0
        for i, p in enumerate(problems):
            t = [torch.from_numpy(x.reshape(-1)).to(vi.device) for x in _matrices(p["nm"], p["na"], seed + 7 * i)]
            mats.append(t)
            descs.append(dict(ncell_x=p["nx"], ncell_y=p["ny"], ncell_z=p["nz"], ne=p["ne"], na=p["na"], nm=p["nm"],
                              vi=vi.data_ptr() + 8 * at, vo=vo.data_ptr() + 8 * at, a_from_m=t[0].data_ptr(),
                              m_from_a=t[1].data_ptr()))
            at += _nstate(p)
        torch.cuda.synchronize()
        return dict(case=c, vi=vi, vo=vo, mats=mats, batch=msb.Batch(descs))
    pb = msb.Problem(_flags(c), nm=c["nm"])
    a, m = _matrices(c["nm"], c["na"], seed)
    pb.set_matrices(a.reshape(-1), m.reshape(-1))
    vi = _state(_nstate(c), seed)
    if c["kind"] == "iterations":
        h_in = torch.empty(vi.numel(), dtype=torch.float64, pin_memory=True)
        h_in.copy_(vi)
        s = dict(case=c, pb=_Owner(pb), vi=h_in, vo=torch.empty(vi.numel(), dtype=torch.float64, pin_memory=True))
    else:
        s = dict(case=c, pb=_Owner(pb), vi=vi, vo=torch.empty_like(vi))
    torch.cuda.synchronize()  # the Sweeper works on its Env's own stream
    return s


class _Owner:
    """Closes the problem with the state that holds it."""

    def __init__(self, pb):
        self.pb = pb

    def __del__(self):
        self.pb.close()


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        state["batch"].sweep(0)
        return state["vo"]
    pb, vi, vo = state["pb"].pb, state["vi"], state["vo"]
    if c["kind"] == "iterations":
        pb.sweep_iterations_host(vo.data_ptr(), vi.data_ptr(), c["niter"])
        return vo
    pb.sweep_device(vo.data_ptr(), vi.data_ptr())
    if c["norms"]:
        normsq, normsqdiff = pb.norms_device(vi.data_ptr(), vo.data_ptr())
        return dict(vo=vo, normsq=normsq, normsqdiff=normsqdiff)
    return vo


def work(case):
    """vi read once and vo written once; two transforms (2 flops per moment, angle) and a 12-flop
    solve per (cell, group, unknown, octant)."""
    problems = _batch_problems(case) if case["kind"] == "batch" else [case]
    nbytes = flops = 0
    for p in problems:
        rows = p["nx"] * p["ny"] * p["nz"] * p["ne"] * NU
        nbytes += 2 * 8 * rows * p["nm"]
        flops += rows * NOCT * p["na"] * (4 * p["nm"] + 12)
    if case["kind"] == "iterations":
        flops *= case["niter"]
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------- exact value
def _space(x, y, z):
    return torch.pow(2.0, ((x + 3 * y + 7 * z + 2) & 3).double())


def _exact_sweep(c, vi, a, m):
    """The sweep of (nz, ne, ny, nx, NU, nm) state by diagonal planes, plain torch in FP64."""
    nx, ny, nz, ne, na, nm = (c[k] for k in ("nx", "ny", "nz", "ne", "na", "nm"))
    dev = vi.device
    vi = vi.view(nz, ne, ny, nx, NU, nm)
    vo = torch.zeros_like(vi)
    pad = (nz + 1) * (ny + 1) * (nx + 1)
    chunk = max(1, min(ne, int(1.5e9 / (8.0 * pad * NU * na))))
    ia = torch.arange(na, device=dev)
    ang = (1 + ia).double() * torch.pow(2.0, (ia & 7).double())
    wx = 0.25 - torch.pow(2.0, -(ia & 7).double())
    gz, gy, gx = torch.meshgrid(*(torch.arange(1, n + 1, device=dev) for n in (nz, ny, nx)), indexing="ij")
    diag = (gz + gy + gx).reshape(-1)
    order = torch.argsort(diag, stable=True)
    counts = torch.bincount(diag, minlength=nz + ny + nx + 1).tolist()
    cell = ((gz * (ny + 1) + gy) * (nx + 1) + gx).reshape(-1)
    for e0 in range(0, ne, chunk):
        e1 = min(ne, e0 + chunk)
        se = torch.tensor([float(1 << (((e * 1366 + 150889) % 714025) & 3)) for e in range(e0, e1)], device=dev).double()
        su = torch.tensor([float(1 << (((u * 741 + 66037) % 312500) & 3)) for u in range(NU)], device=dev).double()
        edge = (se.view(-1, 1, 1) * su.view(1, -1, 1) * ang.view(1, 1, -1)).reshape(1, -1)
        for o in range(NOCT):
            flip = [d for d, bit in ((0, 4), (2, 2), (3, 1)) if o & bit]
            # coordinates of the padded grid counted from the octant's upwind corner; 0 is the ghost layer
            cz, cy, cx = (torch.arange(n + 1, device=dev) - 1 if not o & bit else n - torch.arange(n + 1, device=dev)
                          for n, bit in ((nz, 4), (ny, 2), (nx, 1)))
            sp = _space(cx.view(1, 1, -1), cy.view(1, -1, 1), cz.view(-1, 1, 1)).reshape(-1, 1)
            am = torch.from_numpy(a[o]).to(dev)
            ma = torch.from_numpy(m[o]).to(dev)
            src = vi[:, e0:e1].flip(flip) if flip else vi[:, e0:e1]
            q = src.permute(0, 2, 3, 1, 4, 5).reshape(-1, nm) @ am
            # psi / s_space: the ghost layer holds the boundary flux, the rest the source
            psi = edge.repeat(pad, 1)
            psi[cell] = q.view(nz * ny * nx, -1) / sp[cell]
            del q, src
            w = wx.repeat(edge.numel() // na).view(1, -1)
            sx, sy, sz = 1, nx + 1, (nx + 1) * (ny + 1)
            at = 0
            for d in range(len(counts)):
                k = counts[d]
                if not k:
                    continue
                i = cell[order[at:at + k]]
                at += k
                psi[i] += 0.5 * psi[i - sz] + 0.25 * psi[i - sy] + w * psi[i - sx]
            out = (psi[cell] * sp[cell]).view(-1, na) @ ma
            out = out.view(nz, ny, nx, e1 - e0, NU, nm).permute(0, 3, 1, 2, 4, 5)
            vo[:, e0:e1] += out.flip(flip) if flip else out
            del psi, out
    return vo.reshape(-1)


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        problems = _batch_problems(c)
        vi = _state(sum(_nstate(p) for p in problems), seed).split([_nstate(p) for p in problems])
        return torch.cat([_exact_sweep(p, vi[i], *_matrices(p["nm"], p["na"], seed + 7 * i))
                          for i, p in enumerate(problems)])
    a, m = _matrices(c["nm"], c["na"], seed)
    vi = _state(_nstate(c), seed)
    vo = _exact_sweep(c, vi, a, m)
    if c["kind"] == "iterations":
        for _ in range(1, c["niter"]):
            vo = _exact_sweep(c, vo, a, m)
        return vo
    if c["norms"]:
        d = vi - vo
        return dict(vo=vo, normsq=float((vo * vo).sum()), normsqdiff=float((d * d).sum()))
    return vo
