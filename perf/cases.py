"""What the solver's users run, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a program has in hand
before the call (decks on disk, initialized solves, device tensors), `run` is
one pass through the public interface (the `rism3d` module, its C-ABI and
`slabs`), and `exact` computes what `run` returns in plain FP64 torch, without
the library.  Kinds of pass:

  solve      a started solve: t goes to the device, the closures of the ladder
             (KH, then PSE-2 ... PSE-n) run `steps` iterations each, and the
             excess chemical potentials, the partial molar volume and g(r) of
             every site come back to the host
  batch      the same for many solutes iterated together (the screen)
  setup      a new solve from its deck: parsing, shells, grid potentials,
             long-range terms; beta u, beta phi_L(r) and phi_L(k) come back
  integrals  forces, site energies and the lambda derivative per solute atom,
             over the g(r) of a solve
  split      iterations of a solve split over ranks, one rank's work
             (slabs.DistSolve on device tensors)

Solves run a fixed number of iterations (a tolerance that is never reached):
a pass does the same work on every build.  Mixed solves run fewer of them: from
about 20 on the mixing amplifies any rounding of their FP32 transforms, and two
correct builds differ by what a longer pass made of it.  Mixed-precision
results are returned as float32, the precision of their transforms.
"""
import ctypes
import gzip
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "3d-rism-cuda-mpi_b200"))
import rism3d  # noqa: E402
import slabs  # noqa: E402
import synthetic  # noqa: E402

DEV = "cuda:0"
SPACING = 0.5  # A, every configuration's grid
TOL = 1e-12    # never reached: a solve runs its `steps`
SITES = {"h2o_vv": 2, "naclaq_vv": 4}


def listed():
    return [
        # the smallest configuration: 20 atoms in a 64^3 water cell, FP64 as the
        # command line runs it (latency and launches count)
        dict(name="water64_fp64", kind="solve", nx=64, ny=64, nz=64, solvent="h2o_vv", atoms=20,
             closure="KH", mixer="an2", precision="fp64", steps=48),
        # one drug-like solute of a screen: 96^3 water, the PSE-3 closure ladder
        dict(name="ladder96_mixed", kind="solve", nx=96, ny=96, nz=96, solvent="h2o_vv", atoms=40,
             closure="PSE3", mixer="an2", precision="mixed", steps=16),
        # the screen itself: solutes of 8..60 atoms on 64^3 and 96^3, iterated together
        dict(name="screen12_mixed", kind="batch", solvent="h2o_vv", solves=12, closure="KH",
             mixer="an2", precision="mixed", steps=24),
        # a served request: a peptide-sized solute in salt water
        dict(name="salt144_mixed", kind="solve", nx=144, ny=144, nz=144, solvent="naclaq_vv",
             atoms=200, closure="KH", mixer="an2", precision="mixed", steps=16),
        # a cell that fits its solute: three different, unround sizes
        dict(name="ragged120x100x84_mixed", kind="solve", nx=120, ny=100, nz=84,
             solvent="naclaq_vv", atoms=60, closure="KH", mixer="an2", precision="mixed", steps=16),
        dict(name="ragged80x72x96_fp64", kind="solve", nx=80, ny=72, nz=96, solvent="naclaq_vv",
             atoms=30, closure="KH", mixer="an2", precision="fp64", steps=32),
        # the headline: a 2000-atom globule in 256^3 salt water, mixed and FP64
        dict(name="globule256_mixed", kind="solve", nx=256, ny=256, nz=256, solvent="naclaq_vv",
             atoms=2000, closure="KH", mixer="an2", precision="mixed", steps=16),
        dict(name="globule256_fp64", kind="solve", nx=256, ny=256, nz=256, solvent="naclaq_vv",
             atoms=2000, closure="KH", mixer="an2", precision="fp64", steps=32),
        # the largest configuration's mixer (history-10 Anderson) on the headline grid
        dict(name="globule256_anm10", kind="solve", nx=256, ny=256, nz=256, solvent="naclaq_vv",
             atoms=2000, closure="KH", mixer="anm10", precision="mixed", steps=16),
        # what a new solute costs before its first iteration
        dict(name="setup160_mixed", kind="setup", nx=160, ny=160, nz=160, solvent="naclaq_vv",
             atoms=500, precision="mixed"),
        # forces and energies per atom after a solve
        dict(name="integrals128", kind="integrals", nx=128, ny=128, nz=128, solvent="naclaq_vv",
             atoms=300, closure="KH", precision="fp64", steps=8),
        # one rank of the solve split over GPUs
        dict(name="split192", kind="split", nx=192, ny=192, nz=192, solvent="naclaq_vv", atoms=100,
             steps=4),
    ]


# even sizes whose halves and wholes factor into the engine's primes
def _even_sizes(lo, hi):
    def smooth(n):
        for p in (2, 3, 5, 7, 11, 13):
            while n % p == 0:
                n //= p
        return n == 1
    return [n for n in range(lo + lo % 2, hi + 1, 2) if smooth(n)]


def _draw_dims(rng, lo, hi):
    n = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    sizes = _even_sizes(lo, hi)

    def near(v):
        return min(sizes, key=lambda s: (abs(s - v), s))
    if rng.random() < 0.5:
        return (near(n),) * 3
    return tuple(near(n * rng.uniform(0.75, 1.3)) for _ in range(3))


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["batch", "setup", "integrals", "split"])
    solvent = rng.choice(["h2o_vv", "naclaq_vv"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    atoms = round(math.exp(rng.uniform(math.log(8), math.log(500))))
    if kind == "batch":
        return dict(kind="batch", solvent=solvent, solves=rng.randint(3, 16), closure="KH",
                    mixer="an2", precision=precision,
                    steps=rng.choice([8, 16, 24] if precision == "mixed" else [16, 24, 32]))
    hi = {"solve": 224, "setup": 160, "integrals": 112, "split": 176}[kind]
    nx, ny, nz = _draw_dims(rng, 48, hi)
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, solvent=solvent, atoms=atoms)
    if kind == "solve":
        mixer = rng.choice(["an2", "an2", "anm10"])
        closure = rng.choice(["KH", "PSE2"]) if solvent == "h2o_vv" else "KH"
        c.update(closure=closure, mixer=mixer, precision=precision,
                 steps=rng.choice([8, 12, 16] if precision == "mixed" else [16, 24, 32]))
    elif kind == "setup":
        c.update(precision=precision)
    elif kind == "integrals":
        c.update(closure="KH", precision=precision, steps=8)
        c["atoms"] = min(atoms, 200)
    else:
        c.update(steps=rng.choice([3, 4]))
        c["atoms"] = min(atoms, 100)
    return c


# ------------------------------------------------------------------ inputs
def _solvent_text(name):
    with gzip.open(os.path.join(ROOT, "tests", "golden", name + ".xvk.gz"), "rt") as f:
        return f.read()


def _solute(case, seed, k=0, atoms=None):
    """The seeded solute: drug-like below 64 atoms, else a compact globule.
    Rounded to the digits of a deck."""
    nu = atoms or case["atoms"]
    s = seed * 1009 + k
    if nu <= 64:
        sol = synthetic.make_solute(nu, s, radius=6.0 * (nu / 20.0) ** (1.0 / 3.0), dmin=1.1,
                                    sig=(2.5, 3.8), qsd=0.35)
    else:
        sol = synthetic.make_solute(nu, s)
    return sol


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _box(dims):
    return tuple(SPACING * d for d in dims)


def _closure(case):
    return case.get("closure", "KH")


def _ladder(case):
    """[(library closure, order)]: KH, then PSE-2 ... PSE-n."""
    c = _closure(case)
    st = [(rism3d.KH, 1)]
    if c.startswith("PSE"):
        st += [(rism3d.PSE, k) for k in range(2, int(c[3:]) + 1)]
    return st


class _Work:
    """The files of one prepared case; removed with it."""

    def __init__(self, solvent):
        self.dir = tempfile.TemporaryDirectory(prefix="r3dcase_")
        self.xvk = os.path.join(self.dir.name, solvent + ".xvk")
        with open(self.xvk, "w") as f:
            f.write(_solvent_text(solvent))

    def deck(self, name, sol, dims, steps):
        return synthetic.write_inp(os.path.join(self.dir.name, name + ".inp"), sol, _box(dims),
                                   dims, self.xvk, closure="KH", tol=TOL, maxstep=steps)


def _started(work, case, sol, dims, name="case"):
    """An initialized solve, its start t in page-locked host memory and a
    host buffer for g(r)."""
    steps = case.get("steps", 1)
    s = rism3d.RISM3D(precision=case["precision"])
    s.load(work.deck(name, sol, dims, steps), xvk=work.xvk)
    if case.get("mixer") == "anm10":
        s.set_mixer(rism3d.MIX_ANM, 10, 0.3)
    s.initialize()
    t0 = torch.from_numpy(s.get("t")).pin_memory()
    g = torch.empty(t0.shape, dtype=torch.float64).pin_memory()
    g32 = torch.empty(t0.shape, dtype=torch.float32) if case["precision"] == "mixed" else None
    return dict(s=s, t0=t0.numpy(), g=g, g32=g32, keep=t0)


def _grid(s, which, buf):
    rc = rism3d.lib.r3d_get_grid(s.h, rism3d.GRID[which],
                                 ctypes.cast(buf.data_ptr(), ctypes.POINTER(ctypes.c_double)))
    if rc:
        raise rism3d.R3DError(rc, rism3d.lib.r3d_last_error(s.h).decode())


def _results(e, mixed):
    """The numbers of a .xmu and g(r) of a finished solve."""
    xmu, xmu2, pmv, _ = e["s"].thermo()
    _grid(e["s"], "g", e["g"])
    if not mixed:
        return {"xmu": xmu, "xmu2": xmu2, "pmv": np.array([pmv * 1e6]), "g": e["g"]}
    e["g32"].copy_(e["g"])
    return {"xmu": xmu.astype(np.float32), "xmu2": xmu2.astype(np.float32),
            "pmv": np.array([pmv * 1e6], dtype=np.float32), "g": e["g32"]}


def _batch_solutes(case, seed):
    """(solute, cell) of the screen: the smaller half of the solutes (8..24
    atoms) in 64^3 cells, the others (25..60) in 96^3 cells."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["solves"]):
        small = 2 * k < case["solves"]
        sol = _solute(case, seed, k, atoms=int(rng.integers(8, 25) if small else rng.integers(25, 61)))
        out.append((sol, (64, 64, 64) if small else (96, 96, 96)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "split":
        return _prepare_split(case, seed)
    work = _Work(case["solvent"])
    if kind == "batch":
        es = [_started(work, case, sol, dims, "b%d" % k)
              for k, (sol, dims) in enumerate(_batch_solutes(case, seed))]
        b = rism3d.Batch()
        for e in es:
            b.add(e["s"])
        return dict(kind=kind, es=es, batch=b, mixed=case["precision"] == "mixed", work=work)
    dims = _dims(case)
    sol = _solute(case, seed)
    if kind == "setup":
        n = SITES[case["solvent"]]
        N = dims[0] * dims[1] * dims[2]
        return dict(kind=kind, work=work, inp=work.deck("setup", sol, dims, 100),
                    precision=case["precision"], mixed=case["precision"] == "mixed",
                    u=torch.empty(n * N, dtype=torch.float64).pin_memory(),
                    fr=torch.empty(N, dtype=torch.float64).pin_memory(),
                    fk=torch.empty(N, dtype=torch.float64).pin_memory())
    e = _started(work, case, sol, dims)
    st = dict(kind=kind, e=e, ladder=_ladder(case), mixed=case["precision"] == "mixed", work=work)
    if kind == "integrals":  # the solve whose g(r) the integrals are taken over
        e["s"].iterate()
    return st


def run(state):
    kind, mixed = state["kind"], state.get("mixed", False)
    if kind == "solve":
        e = state["e"]
        s = e["s"]
        s.set_t(e["t0"])
        for clos, order in state["ladder"]:
            s.set_closure(clos, order)
            s.iterate()
        return _results(e, mixed)
    if kind == "batch":
        for e in state["es"]:
            e["s"].set_t(e["t0"])
        state["batch"].iterate()
        return [_results(e, mixed) for e in state["es"]]
    if kind == "setup":
        with rism3d.RISM3D(precision=state["precision"]) as s:
            s.load(state["inp"], xvk=state["work"].xvk)
            s.initialize()
            _grid(s, "u", state["u"])
            _grid(s, "fr", state["fr"])
            _grid(s, "fk", state["fk"])
        u, fr, fk = state["u"], state["fr"], state["fk"]
        return {"u": u.float() if mixed else u, "fr": fr.float() if mixed else fr, "fk": fk}
    if kind == "integrals":
        grad, euv, ad = state["e"]["s"].atom_integrals()
        f = np.float32 if mixed else np.float64
        return {"grad": grad.astype(f), "euv": euv.astype(f), "ad": ad.astype(f)}
    ds = state["ds"]
    ds.t = state["t0"].clone()
    ds.iterate()
    return {"t": ds.t, "r": ds.r, "g": ds.g}


def _prepare_split(case, seed):
    """One rank holding the whole grid: u, phi_L(r), phi_L(k) and chi on
    device, and a t some steps into its solve."""
    m = _Model(case, _solute(case, seed))
    nx, ny, nz = _dims(case)
    plan = slabs.SlabPlan(nz, ny, nx, 1)
    half = m.chi[:, :, :, :, 0::2].contiguous()
    fkt = (m.fk / (m.dv * m.phase_c()))[:, :, 0::2]
    ts, _, _ = m.solve(0, 1, 8, "an2")
    t0 = (ts + m.qfr).contiguous()
    ds = slabs.DistSolve(plan, 0, m.u.contiguous(), t0.clone(), m.fr.contiguous(), half,
                         torch.view_as_real(fkt.resolve_conj().contiguous()).contiguous(),
                         m.qv.cpu().numpy(), m.rhov.cpu().numpy(), tol=TOL, maxstep=case["steps"],
                         stages=slabs.CudaStages(rism3d.lib, 0), ops=slabs.CudaOps(rism3d.lib, 0))
    return dict(kind="split", ds=ds, t0=t0)


# ------------------------------------------------------------- work of a pass
def _iteration_work(case, N, n):
    """Bytes and operations of one iteration: state and grids read and written
    once per stage (closure, transform slabs, OZ, residual, mixing history),
    real transforms both ways, the closure and the n x n OZ product."""
    b = 4 if case.get("precision", "fp64") == "mixed" else 8
    m = 10 if case.get("mixer") == "anm10" else 2
    lg = math.log2(N)
    return N * b * (n * (14 + 3 * m) + 2), n * N * (2 * 2.5 * lg + 2 * n + 30 + 10 * m)


def work(case):
    kind = case["kind"]
    n = SITES[case["solvent"]]
    if kind == "batch":
        w = [_iteration_work(case, N, n) for N in (64 ** 3, 96 ** 3)]
        k = [case["steps"] * ((case["solves"] + 1) // 2), case["steps"] * (case["solves"] // 2)]
        return {"bytes": float(k[0] * w[0][0] + k[1] * w[1][0]), "flops": k[0] * w[0][1] + k[1] * w[1][1]}
    N = case["nx"] * case["ny"] * case["nz"]
    if kind == "setup":
        b = 4 if case["precision"] == "mixed" else 8
        return {"bytes": float(N * (n * b * 3 + b + 8)),
                "flops": float(N) * case["atoms"] * (6 * n + 20) + 4.0 * N * case["atoms"]}
    if kind == "integrals":
        return {"bytes": 8.0 * n * N, "flops": float(N) * case["atoms"] * (22 * n + 12)}
    by, fl = _iteration_work(case, N, n)
    k = case["steps"] * len(_ladder(case))
    io = 16.0 * n * N if kind == "solve" else 0.0
    return {"bytes": k * by + io, "flops": k * float(fl)}


# ------------------------------------------------------- FP64 torch reference
AVOGADRO, BOLTZMANN = 6.02214076e23, 1.380649e-23
HARTREE, BOHR = 4.359744722207185e-18, 0.5291771500001


def _read_xvk(name):
    lines = _solvent_text(name).splitlines()
    h = lines[1].split()
    num, natv, ntab, dr = int(h[1]), int(h[2]), int(h[3]), float(h[4])
    h2 = lines[2].split()
    sig, eps, q, rho = (np.zeros(natv) for _ in range(4))
    for a in lines[4:4 + num]:
        c = a.split()
        i = abs(int(c[3])) - 1
        sig[i], eps[i], q[i] = float(c[4]), float(c[5]), float(c[6])
        rho[i] += float(c[10])
    vals = np.array(" ".join(lines[num + 5:]).split()[:natv * natv * ntab], dtype=np.float64)
    return dict(natv=natv, ntab=ntab, dr=dr, temper=float(h2[2]), xt=float(h2[3]), sig=sig, eps=eps,
                q=q, rho=rho * AVOGADRO * 1e-27, tab=vals.reshape(ntab, natv * natv))


def _natural_spline(x, y):
    """Second derivatives of the natural cubic spline through y [np, columns]
    at the uniform abscissae x."""
    h = x[1] - x[0]
    n = len(x)
    d2 = 6.0 * (y[2:] - 2 * y[1:-1] + y[:-2]) / (h * h)
    c = np.zeros(n - 2)
    d = np.zeros_like(d2)
    c[0], d[0] = 0.25, d2[0] / 4.0
    for i in range(1, n - 2):
        w = 1.0 / (4.0 - c[i - 1])
        c[i] = w
        d[i] = (d2[i] - d[i - 1]) * w
    m = np.zeros_like(y)
    m[n - 2] = d[n - 3]
    for i in range(n - 4, -1, -1):
        m[i + 1] = d[i] - c[i] * m[i + 2]
    return m


class _Model:
    """3D-RISM of one solute in FP64 torch: full complex k grid, shifted
    transforms F(k) = dv sum f e^{-ikr}, r = (i - n/2) dr, k = 2 pi (j - n/2 +
    1/2) / L, on the short-range parts u_s, t_s with phi_L added in k space."""

    def __init__(self, case, sol, dims=None):
        self.case = case
        nx, ny, nz = dims or _dims(case)
        self.dims = (nz, ny, nx)
        self.N = nx * ny * nz
        box = _box((nx, ny, nz))
        self.dv = box[0] * box[1] * box[2] / self.N
        v = _read_xvk(case["solvent"])
        self.v, self.n = v, v["natv"]
        f64 = dict(dtype=torch.float64, device=DEV)
        self.qv = torch.tensor(v["q"], **f64)
        self.rhov = torch.tensor(v["rho"], **f64)
        # the solute as its deck says it, centred by whole angstroms
        sig = np.array([float("%.6f" % x) for x in sol["sig"]])
        eps = np.array([float("%.6f" % x) for x in sol["eps"]])
        q = np.array([float("%.8f" % x) for x in sol["q"]])
        r = np.array([[float("%.6f" % x) for x in p] for p in sol["r"]])
        for d in range(3):
            s = -(r[:, d].max() - r[:, d].min()) / 2 - r[:, d].min()
            r[:, d] += math.copysign(math.floor(abs(s) + 0.5), s)
        self.sol = (sig, eps, q, r)
        ikt = 1.0 / (AVOGADRO * BOLTZMANN * v["temper"])
        ub = HARTREE * BOHR / (BOLTZMANN * v["temper"])
        self.ikt, self.ub = ikt, ub
        ax = [((torch.arange(m, **f64)) - m // 2) * (b / m)
              for m, b in zip((nx, ny, nz), box)]
        self.ax = ax
        # pair sums
        n, shp = self.n, self.dims
        lj = torch.zeros((n,) + shp, **f64)
        e, f = torch.zeros(shp, **f64), torch.zeros(shp, **f64)
        s6max = (2.0e-3) ** -6
        for k in range(len(q)):
            r2 = ((ax[2] - r[k, 2]) ** 2)[:, None, None] + ((ax[1] - r[k, 1]) ** 2)[None, :, None] \
                + ((ax[0] - r[k, 0]) ** 2)[None, None, :]
            r1 = torch.sqrt(r2)
            ir6 = r2.reciprocal().pow_(3)
            for s in range(n):
                sg = (sig[k] + v["sig"][s]) * 0.5
                s6 = (sg ** 6 * ir6).clamp_(max=s6max)
                lj[s] += 4.0 * math.sqrt(eps[k] * v["eps"][s]) * (s6 * s6 - s6)
            near = r1 < 1e-5
            ir = r1.reciprocal()
            e += torch.where(near, 0.0, q[k] * ir)
            f += torch.where(near, q[k], q[k] * ir * (-torch.expm1(-r1)))
        self.fr = f * ub
        self.qfr = self.qv[:, None, None, None] * self.fr
        self.u = lj * ikt + self.qv[:, None, None, None] * (e * ub)
        del lj
        self.us = self.u - self.qfr
        # k space
        kk = [2.0 * math.pi * (torch.arange(m, **f64) - m / 2 + 0.5) / b
              for m, b in zip((nx, ny, nz), box)]
        k2 = (kk[2] ** 2)[:, None, None] + (kk[1] ** 2)[None, :, None] + (kk[0] ** 2)[None, None, :]
        ph = [torch.exp(-1j * kk[d][None, :] * torch.tensor(r[:, d], **f64)[:, None])
              for d in range(3)]
        S = torch.zeros(shp, dtype=torch.complex128, device=DEV)
        qt = torch.tensor(q, **f64)
        for z in range(nz):
            S[z] = (ph[1] * (qt[:, None] * ph[2][:, z:z + 1])).T @ ph[0]
        self.fk = S * (4.0 * math.pi * ub) / (k2 * (k2 + 1.0))
        del S
        # chi_ab(|k|): natural splines of the table over the grid's |k| range
        dk = math.pi / (v["dr"] * v["ntab"])
        ks = torch.sqrt(k2)
        kmin, kmax = float(ks.min()), float(ks.max())
        tt = dk * (np.arange(v["ntab"]) + 1)
        below, above = np.nonzero(tt < kmin)[0], np.nonzero(tt[1:] > kmax)[0] + 1
        i1 = int(below[-1]) if len(below) else 0
        i2 = int(above[0]) if len(above) else v["ntab"] - 1
        x, y = tt[i1:i2 + 1], v["tab"][i1:i2 + 1]
        m2 = torch.tensor(_natural_spline(x, y), **f64)
        yt, xt = torch.tensor(y, **f64), torch.tensor(x, **f64)
        lo = (torch.searchsorted(xt, ks.reshape(-1), right=True) - 1).clamp_(0, len(x) - 2)
        t = ks.reshape(-1) - xt[lo]
        self.chi = torch.empty((n, n) + shp, **f64)
        for a in range(n):
            for b in range(n):
                col = a * n + b
                y0, y1, s0, s1 = yt[lo, col], yt[lo + 1, col], m2[lo, col], m2[lo + 1, col]
                c1 = s0 / 2
                c2 = (s1 - s0) / (6 * dk)
                c0 = (y1 - y0) / dk - dk * (2 * s0 + s1) / 6
                self.chi[a, b] = (((c2 * t + c1) * t + c0) * t + y0).reshape(shp)
        del lo, t, ks, k2
        # transform phases: F = dv post fftn(f pre)
        pre, post = [], []
        for m in (nz, ny, nx):
            i = torch.arange(m, **f64)
            sgn = 1.0 - 2.0 * (torch.arange(m, device=DEV) % 2)
            pre.append(sgn * torch.exp(-1j * math.pi * i / m))
            ang = math.pi * (0.5 - m / 2)
            post.append(sgn * complex(math.cos(ang), math.sin(ang)))
        self.pre, self.post = ([p[0][:, None, None], p[1][None, :, None], p[2][None, None, :]]
                               for p in (pre, post))

    def fwd(self, f):
        x = f * self.pre[0] * self.pre[1] * self.pre[2]
        return torch.fft.fftn(x) * (self.dv * self.post[0]) * self.post[1] * self.post[2]

    def inv(self, F):
        x = F * self.post[0].conj() * self.post[1].conj() * self.post[2].conj()
        x = torch.fft.ifftn(x) * self.pre[0].conj() * self.pre[1].conj() * self.pre[2].conj()
        return x.real / self.dv

    def phase_c(self):
        """C(k) = -i (-1)^{jx+jy+jz+(nx+ny+nz)/2} of the unphased transform."""
        nz, ny, nx = self.dims
        s = [1.0 - 2.0 * (torch.arange(m, device=DEV, dtype=torch.float64) % 2)
             for m in (nz, ny, nx)]
        sg = s[0][:, None, None] * s[1][None, :, None] * s[2][None, None, :]
        return -1j * sg * (-1.0) ** ((nx + ny + nz) // 2)

    def closure(self, clos, order, x):
        if clos == rism3d.KH:
            up = 1.0 + x
        else:
            up, term = torch.ones_like(x), torch.ones_like(x)
            for i in range(1, order + 1):
                term = term * x / i
                up = up + term
        return torch.where(x >= 0, up, torch.exp(x.clamp(max=0.0)))

    def evaluate(self, clos, order, ts):
        g = self.closure(clos, order, ts - self.us)
        C = []
        for b in range(self.n):
            C.append(self.fwd(g[b] - 1.0 - ts[b]) - self.qv[b] * self.fk)
        r = torch.empty_like(ts)
        for a in range(self.n):
            H = self.chi[a, 0] * C[0]
            for b in range(1, self.n):
                H += self.chi[a, b] * C[b]
            r[a] = self.inv(H) + 1.0 - g[a]
        return g, r

    def solve(self, clos, order, steps, mixer, ts=None, mix_last=False):
        """`steps` evaluations with a mix between them: (t_s, g, R) of the
        last; mix_last: t_s after one more mix."""
        ts = torch.zeros_like(self.us) if ts is None else ts
        irho = 1.0 / self.rhov
        w = irho[:, None, None, None]

        def dot(a, b):
            return float((a * b * w).sum())
        tp, rp, binary, left = [None, None], [None, None], 0, 2
        hist, H = [], 10
        for step in range(steps):
            g, r = self.evaluate(clos, order, ts)
            if step == steps - 1 and not mix_last:
                break
            if mixer == "an2":
                if left > 0:
                    left -= 1
                    tn = ts + r
                else:
                    d0, d1 = r - rp[0], r - rp[1]
                    a00, a01, a11 = dot(d0, d0), dot(d0, d1), dot(d1, d1)
                    c0, c1 = dot(r, d0), dot(r, d1)
                    x1 = (c1 - a01 * c0 / a00) / (a11 - a01 * a01 / a00)
                    x0 = c0 / a00 - a01 / a00 * x1
                    s0 = x0 + 0.2 * (0 if binary == 0 else 1)
                    s1 = x1 + 0.2 * (1 if binary == 0 else 0)
                    uu = ts + s0 * (tp[0] - ts) + s1 * (tp[1] - ts)
                    vv = ts + r + s0 * (tp[0] + rp[0] - ts - r) + s1 * (tp[1] + rp[1] - ts - r)
                    tn = uu + 0.6 * (vv - uu)
                tp[binary], rp[binary] = ts, r
                binary = 1 - binary
            else:
                beta = 0.3
                z = ts + beta * r
                m = len(hist)
                tn = z
                if m:
                    d = [r - h[0] for h in hist]
                    A = np.array([[dot(p, q) for q in d] for p in d])
                    y = np.linalg.solve(A, np.array([dot(p, r) for p in d]))
                    tn = (1.0 - y.sum()) * z
                    for c, h in zip(y, hist):
                        tn = tn + float(c) * h[1]
                hist = ([(r, z)] + hist)[:H]
            ts = tn
        return ts, g, r

    def ladder(self):
        ts = None
        for clos, order in _ladder(self.case):
            ts, g, r = self.solve(clos, order, self.case["steps"], self.case.get("mixer", "an2"), ts)
            last = (clos, order)
        return ts, g, r, last

    def results(self):
        ts, g, r, (clos, order) = self.ladder()
        h = r - 1.0 + g
        t = ts + self.qfr
        c = h - t
        hnc = 0.5 * h * t - c
        gf = -(0.5 * h + 1.0) * c
        if clos == rism3d.KH:
            up = gf
        else:
            x = ts - self.us
            term = torch.ones_like(x)
            for k in range(1, order + 2):
                term = term * x / k
            up = 0.5 * h * h - c - 0.5 * h * c - term
        sc = torch.where(h > 0, up, hnc)

        def site(q):
            return (q.sum(dim=(1, 2, 3)) * self.rhov * self.dv).cpu().numpy()
        xmu = np.concatenate([site(sc), site(gf)])
        ibeta = AVOGADRO * BOLTZMANN * self.v["temper"]
        pmv = self.v["xt"] * (1.0 - site(c).sum()) * ibeta
        return {"xmu": xmu, "xmu2": site(hnc), "pmv": np.array([pmv * 1e6]), "g": g}

    def integrals(self):
        _, g, _, _ = self.ladder()
        sig, eps, q, r = self.sol
        v, cc, kcal = self.v, HARTREE * BOHR * AVOGADRO, 4184.0
        grad, euv, ad = np.zeros((len(q), 3)), np.zeros((len(q), self.n)), np.zeros(len(q))
        for k in range(len(q)):
            dx, dy, dz = (self.ax[d] - r[k, d] for d in range(3))
            r2 = (dz ** 2)[:, None, None] + (dy ** 2)[None, :, None] + (dx ** 2)[None, None, :]
            r1 = torch.sqrt(r2)
            fm = torch.zeros_like(r2)
            for s in range(self.n):
                sg = (sig[k] + v["sig"][s]) * 0.5
                ep = math.sqrt(eps[k] * v["eps"][s])
                qq = q[k] * v["q"][s] * cc
                s6 = (sg * sg / r2) ** 3
                w = torch.where(r1 >= sg * 0.5, v["rho"][s] * g[s], 0.0)
                on = w != 0
                zero = torch.zeros_like(w)
                fm += torch.where(on, (24 * ep * s6 / r2 * (2 * s6 - 1) + qq / (r2 * r1)) * w, zero)
                euv[k, s] = float(torch.where(on, (4 * ep * s6 * (s6 - 1) + qq / r1) * w, zero).sum())
                ad[k] += float(torch.where(on, qq / r1 * w, zero).sum())
            grad[k] = [float((fm * dx[None, None, :]).sum()), float((fm * dy[None, :, None]).sum()),
                       float((fm * dz[:, None, None]).sum())]
        return {"grad": grad * self.dv / kcal, "euv": euv * self.dv, "ad": ad * self.dv / kcal}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for sol, dims in _batch_solutes(case, seed):
            r = _Model(case, sol, dims).results()
            r["g"] = r["g"].cpu()
            out.append(r)
        return out
    m = _Model(case, _solute(case, seed))
    if kind == "solve":
        return m.results()
    if kind == "setup":
        fk = torch.view_as_real(m.fk[:, :, 0::2].contiguous()).reshape(-1)
        return {"u": m.u.reshape(-1), "fr": m.fr.reshape(-1), "fk": fk}
    if kind == "integrals":
        return m.integrals()
    t8, _, _ = m.solve(0, 1, 8, "an2")
    ts, g, r = m.solve(0, 1, case["steps"], "an2", t8, mix_last=True)
    return {"t": ts + m.qfr, "r": r, "g": g}
