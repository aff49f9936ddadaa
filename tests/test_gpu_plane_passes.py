"""The iteration on the plane passes (whole z-planes per CTA, or row tiles with
y passes of their own, on the run-time-planned transform engine) against the
general run-time-length passes at the sizes where they can go wrong: prime
factors 7, 11 and 13, odd half rows (single-element loads), rows that end in a
partial tile, columns that end in a partial tile, compile-time and run-time
sizes, one to four sites.  Also the slab stages on that engine, the per-atom
integrals for atom counts around a warp, and grid copies to page-locked memory.

Tolerances: three evaluations and mixes in FP64 differ by roundings of order
1e-15, and each mix multiplies a difference of R by less than 30 at contact
peaks: 1e-10 of t's largest value.  In mixed precision the general passes'
transforms, and those of the plane passes in FP32 arithmetic, round to about
3e-7 of c: 1e-4 of t's largest value after the same three steps.  The plane
passes in FP64 arithmetic on FP32 grids (most grids below 3.5 million voxels)
are also held to the FP64 solve, see test_fp64_arithmetic_on_fp32_grids."""
import gzip
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def _subset_xvk(path, sites):
    """The shipped salt-water table reduced to its first `sites` sites."""
    lines = gzip.open(os.path.join(GOLD, "naclaq_vv.xvk.gz"), "rt").read().splitlines()
    h = lines[1].split()
    num, natv, ntab = int(h[1]), int(h[2]), int(h[3])
    atoms = [a for a in lines[4:4 + num] if abs(int(a.split()[3])) <= sites]
    vals = np.array(" ".join(lines[num + 5:]).split()[:natv * natv * ntab], float)
    tab = vals.reshape(ntab, natv, natv)[:, :sites, :sites].reshape(ntab, -1)
    with open(path, "w") as f:
        f.write(lines[0] + "\n## %d %d %d %s %s\n" % (len(atoms), sites, ntab, h[4], h[5]))
        f.write("\n".join([lines[2], lines[3]] + atoms + ["##"]) + "\n")
        for row in tab:
            f.write(" ".join("%.15e" % v for v in row) + "\n")
    return path


def _three_steps(R, inp, xvk, prec):
    s = R.RISM3D(precision=prec)
    s.initialize(inp, xvk=xvk)
    for _ in range(3):
        rms = s.calculate()
        s.anderson()
    t = s.get("t")
    s.close()
    return rms, t


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("grid,sites", [
    ((48, 48, 48), 2),      # compile-time planes
    ((96, 32, 36), 4),       # a run-time plane
    ((90, 22, 26), 3),      # odd half rows, primes 11 and 13
    ((44, 52, 28), 1),      # primes 11, 13 and 7; columns end in a partial tile
    ((256, 10, 18), 4),     # row tiles, the last of them partial
    ((200, 126, 12), 2),    # run-time sizes, 7 x 18 columns
    ((8, 6, 4), 2),         # the smallest
    # mixed: FP32 arithmetic (lengths all listed, an FP64 plan of a pass more)
    ((48, 48, 128), 2),     # a run-time plane, a compile-time z of radices 16 and 8
    ((128, 128, 32), 2),    # mixed: FP64 arithmetic in tiles (32 is not listed)
    ((128, 128, 128), 1),   # compile-time planes
    # and above 3.5 million voxels: run-time tiles, several per inverse CTA, the
    # last partial; odd half rows of 7 x 11 and 7 x 13
    ((154, 150, 156), 2),
    ((182, 144, 150), 1),
])
def test_plane_passes_match_general_passes(tmp_path, monkeypatch, grid, sites, prec):
    import rism3d as R
    import synthetic as S
    xvk = _subset_xvk(str(tmp_path / "s.xvk"), sites)
    box = tuple(0.5 * n for n in grid)
    sol = S.make_solute(4, 3, radius=0.9, dmin=0.5, sig=(2.5, 3.0), qsd=0.2)
    inp = S.write_inp(str(tmp_path / "p.inp"), sol, box, grid, xvk)
    got = {}
    for variant in ("0", "5"):
        monkeypatch.setenv("R3D_X_VARIANT", variant)
        monkeypatch.setenv("R3D_YZ_VARIANT", "0")
        got[variant] = _three_steps(R, inp, xvk, prec)
    (r0, t0), (r5, t5) = got["0"], got["5"]
    tol = 1e-10 if prec == "fp64" else 1e-4
    scale = np.abs(t0).max()
    assert np.isfinite(t0).all() and scale > 0
    assert np.abs(t5 - t0).max() <= tol * scale
    assert abs(r5 - r0) <= tol * max(r0, 1.0)


@pytest.mark.parametrize("n", [2, 5])
def test_fp64_step_leaves_the_mixed_t(tmp_path, monkeypatch, solvents, n):
    """r3d_step ends with t mixed (the plane passes mix at the start of the
    next iteration; step applies the one still pending): t as on the general
    path, and further steps continue from it."""
    import rism3d as R
    import synthetic as S
    xvk = solvents["h2o_vv"]
    inp = S.small(str(tmp_path), nu=6, grid=(32, 24, 28), box=(16.0, 12.0, 14.0), solvent=xvk)
    out = {}
    for variant in ("0", "5"):
        monkeypatch.setenv("R3D_X_VARIANT", variant)
        s = R.RISM3D(precision="fp64")
        s.initialize(inp, xvk=xvk)
        s.step(n)
        a = s.get("t")
        s.step(2)
        out[variant] = (a, s.get("t"), s.status()[0])
        s.close()
    for k in (0, 1):
        d = np.abs(out["5"][k] - out["0"][k]).max()
        assert d <= 1e-10 * np.abs(out["0"][k]).max()
    assert out["5"][2] == out["0"][2] == n + 2


@pytest.mark.parametrize("grid,sites", [((48, 48, 48), 2), ((90, 22, 26), 3), ((44, 52, 28), 1),
                                        ((200, 126, 12), 2), ((96, 32, 36), 4)])
def test_fp64_arithmetic_on_fp32_grids(tmp_path, monkeypatch, grid, sites):
    """Three mixed steps against three FP64 ones on the plane passes.  What the
    mixed path stores in FP32: u, up to 4 where g is large (half an ulp, 1.2e-7,
    times g < 30: 4e-6 of g) and R and the long-range term, up to 30 (1e-6); the
    spectra's roundings average out in the transforms.  5e-6 per evaluation:
    2e-5 of t's largest value after three."""
    import rism3d as R
    import synthetic as S
    xvk = _subset_xvk(str(tmp_path / "s.xvk"), sites)
    sol = S.make_solute(4, 3, radius=0.9, dmin=0.5, sig=(2.5, 3.0), qsd=0.2)
    inp = S.write_inp(str(tmp_path / "p.inp"), sol, tuple(0.5 * n for n in grid), grid, xvk)
    monkeypatch.setenv("R3D_X_VARIANT", "5")
    t = {p: _three_steps(R, inp, xvk, p)[1] for p in ("fp64", "mixed")}
    assert np.abs(t["mixed"] - t["fp64"]).max() <= 2e-5 * np.abs(t["fp64"]).max()


# the paths whose next forward pass mixes (a listed and an unlisted row length
# on the plane passes, the mix-fused x pass of the per-axis ones)
DEFERRED = {"plane_listed": ((64, 24, 28), {"R3D_X_VARIANT": "5"}),
            "plane_unlisted": ((60, 24, 28), {"R3D_X_VARIANT": "5"}),
            "fused_per_axis": ((64, 24, 28), {"R3D_X_VARIANT": "1", "R3D_MFX": "1"})}
GENERAL = {"R3D_X_VARIANT": "0", "R3D_YZ_VARIANT": "0"}


def _sequence(R, monkeypatch, inp, xvk, prec, env, ops):
    """t after every mixing operation of ops (a number: step(n)), and the
    evaluations counted."""
    for k in ("R3D_X_VARIANT", "R3D_YZ_VARIANT", "R3D_MFX"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    s = R.RISM3D(precision=prec)
    s.initialize(inp, xvk=xvk)
    out = []
    for op in ops:
        if op == "calculate":
            s.calculate()
            continue
        s.anderson() if op == "anderson" else s.step(op)
        out.append(s.get("t"))
    out.append(s.status()[0])
    s.close()
    return out


def _same_sequence(R, monkeypatch, tmp_path, xvk, prec, path, ops):
    import synthetic as S
    grid, env = DEFERRED[path]
    inp = S.small(str(tmp_path), nu=6, grid=grid, box=tuple(0.5 * k for k in grid), solvent=xvk)
    got = _sequence(R, monkeypatch, inp, xvk, prec, env, ops)
    ref = _sequence(R, monkeypatch, inp, xvk, prec, GENERAL, ops)
    assert got[-1] == ref[-1]
    for g, r in zip(got[:-1], ref[:-1]):  # (a mix left out or made twice: 4e-2 and more)
        assert np.abs(g - r).max() <= (1e-10 if prec == "fp64" else 1e-4) * np.abs(r).max()


@pytest.mark.parametrize("ops", [(3, 1), (3, "calculate", "anderson")])
@pytest.mark.parametrize("path", sorted(DEFERRED))
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_step_applies_the_pending_mix(tmp_path, monkeypatch, solvents, prec, path, ops):
    """r3d_step(n) leaves t mixed n times, and calculate and anderson go on from
    it, whichever pass would have mixed next."""
    import rism3d as R
    _same_sequence(R, monkeypatch, tmp_path, solvents["h2o_vv"], prec, path, ops)


@pytest.mark.parametrize("path", sorted(DEFERRED))
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_step_after_anderson_mixes_once(tmp_path, monkeypatch, solvents, prec, path):
    """The mix that r3d_anderson has applied is not pending any more."""
    import rism3d as R
    _same_sequence(R, monkeypatch, tmp_path, solvents["h2o_vv"], prec, path,
                   ("calculate", "anderson", 1, 1))


@pytest.mark.parametrize("path,prec", [("plane_listed", "fp64"), ("plane_listed", "mixed"),
                                       ("fused_per_axis", "mixed")])
def test_profiled_forward_pass_mixes(tmp_path, monkeypatch, solvents, path, prec):
    """After r3d_step nothing is pending, but the mixing forward pass is profiled
    with its mix: bytes of t, u, (c_ref,) R and four history rows in, t, two
    history rows, g and the spectrum out; and the next steps start from the
    same t."""
    import rism3d as R
    import synthetic as S
    grid, env = DEFERRED[path]
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    inp = S.small(str(tmp_path), nu=6, grid=grid, box=tuple(0.5 * k for k in grid), solvent=solvents["h2o_vv"])
    s = R.RISM3D(precision=prec)
    s.initialize(inp, xvk=solvents["h2o_vv"])
    s.step(3)
    t = s.get("t")
    by = {name: b for name, _, b in s.profile_kernels(2)}
    assert by["mix_fx"] == (96 if prec == "fp64" else 64) * 2 * np.prod(grid)
    assert np.array_equal(s.get("t"), t)
    s.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_ksave_file_holds_the_mixed_t(tmp_path, monkeypatch, solvents, prec):
    """The .tuv that iterate saves after step 3 is the t of the start of step 4."""
    import rism3d as R
    import synthetic as S
    xvk = solvents["h2o_vv"]
    grid = (60, 24, 28)
    inp = S.small(str(tmp_path), nu=6, grid=grid, box=(30.0, 12.0, 14.0), solvent=xvk, tol=1e-12, maxstep=4)
    lines = open(inp).read().split("\n")
    lines[0] = " m  3  20220301"
    open(inp, "w").write("\n".join(lines))
    s = R.RISM3D(precision=prec)
    s.initialize(inp, xvk=xvk)
    s.iterate()
    s.close()
    # (saved with six significant digits)
    t = np.array(open(inp[:-4] + ".tuv").read().split()[4:], dtype=float)
    ref = _sequence(R, monkeypatch, inp, xvk, prec, GENERAL, (3,))[0].ravel()
    assert np.abs(t - ref).max() <= 1e-4 * np.abs(ref).max()


class _ReducedPhases:
    """The dense stages' matrices with every phase reduced to one turn in whole
    numbers first: unreduced, phases of up to 2 pi 9000 are 7e-12 off."""

    @staticmethod
    def _mx(nx):
        x, p = np.arange(nx), np.arange(nx // 2)
        return ((-1.0) ** x)[None, :] * np.exp(-1j * np.pi * (np.outer(4 * p + 1, x) % (2 * nx)) / nx)

    @staticmethod
    def _mk(n):
        j = np.arange(n)
        return np.exp(-1j * np.pi * (np.outer(2 * j + 1, j) % (2 * n)) / n)


# (4 and 9000: the shortest and about the longest row; 3125: five passes)
@pytest.mark.parametrize("n,nz,ny,nx", [(1, 6, 10, 22), (3, 4, 1, 6), (2, 1, 13, 8), (2, 14, 35, 52),
                                        (1, 4, 6, 4), (1, 2, 3125, 4), (1, 2, 2, 9000)])
def test_slab_stages_match_numpy(n, nz, ny, nx):
    import torch
    import rism3d as R
    import slabs
    rng = np.random.default_rng(nx)
    real = rng.standard_normal((n, nz, ny, nx))
    class Stages(_ReducedPhases, slabs.NumpyStages):
        pass

    np_st, cu = Stages(), slabs.CudaStages(R.lib, 0)
    ref = np.stack([np_st.forward_z(np_st.forward_xy(real[v])) for v in range(n)])
    spec = cu.forward_z_all(cu.forward_xy_all(torch.from_numpy(real).cuda()))
    got = torch.view_as_complex(spec.contiguous()).cpu().numpy()
    scale = np.abs(ref).max()
    assert np.abs(got - ref).max() <= 1e-12 * scale
    back = cu.inverse_xy_all(cu.inverse_z_all(spec)).cpu().numpy()
    N = nx * ny * nz
    assert np.abs(back - real * (N / 2)).max() <= 1e-12 * N * np.abs(real).max()


@pytest.mark.parametrize("nu", [1, 31, 33])
def test_atom_integrals_match_direct_sums(tmp_path, solvents, nu):
    import rism3d as R
    import synthetic as S
    xvk = solvents["naclaq_vv"]
    grid, box = (24, 20, 18), (12.0, 10.0, 9.0)
    inp = S.small(str(tmp_path), nu=nu, grid=grid, box=box, solvent=xvk, seed=nu) if nu < 20 else \
        S.write_inp(str(tmp_path / "a.inp"), S.make_solute(nu, nu, radius=4.0, dmin=0.8, qsd=0.2),
                    box, grid, xvk)
    s = R.RISM3D(precision="fp64")
    s.load(inp, xvk=xvk)
    qv, rhov = s.solvent_sites()
    s.set_control(maxstep=3)
    s.initialize()
    s.iterate()
    g = s.get("g")
    grad, euv, ad = s.atom_integrals()
    s.close()
    lines = gzip.open(os.path.join(GOLD, "naclaq_vv.xvk.gz"), "rt").read().splitlines()
    sv, ev = np.zeros(4), np.zeros(4)
    for a in lines[4:9]:
        c = a.split()
        i = abs(int(c[3])) - 1
        sv[i], ev[i] = float(c[4]), float(c[5])
    rows = np.array([[float(x) for x in l.split()] for l in open(inp).read().splitlines()[-nu:]])
    r = rows[:, 3:6].copy()
    for d in range(3):
        sh = -(r[:, d].max() - r[:, d].min()) / 2 - r[:, d].min()
        r[:, d] += np.copysign(np.floor(abs(sh) + 0.5), sh)
    ax = [(np.arange(m) - m // 2) * (b / m) for m, b in zip(grid, box)]
    Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    dv, cc, kcal = np.prod(box) / np.prod(grid), 4.359744722207185e-18 * 0.5291771500001 * 6.02214076e23, 4184.0
    with np.errstate(divide="ignore", invalid="ignore"):
        for a in range(nu):
            dx, dy, dz = X - r[a, 0], Y - r[a, 1], Z - r[a, 2]
            r2 = dx * dx + dy * dy + dz * dz
            r1 = np.sqrt(r2)
            F, A = np.zeros(3), 0.0
            for v in range(4):
                sg, ep = (rows[a, 0] + sv[v]) / 2, np.sqrt(rows[a, 1] * ev[v])
                on, s6, qq = r1 >= sg / 2, (sg * sg / r2) ** 3, rows[a, 2] * qv[v] * cc
                w = rhov[v] * g[v]
                fm = np.where(on, (24 * ep * s6 / r2 * (2 * s6 - 1) + qq / (r2 * r1)) * w, 0)
                F += [(fm * q).sum() for q in (dx, dy, dz)]
                e = np.where(on, (4 * ep * s6 * (s6 - 1) + qq / r1) * w, 0)
                A += np.where(on, qq / r1 * w, 0).sum()
                # sums of some 8000 terms in another order
                assert abs(euv[a, v] - e.sum() * dv) <= 1e-11 * np.abs(e).sum() * dv
            big = np.abs(grad).max() + 1e-30
            assert np.abs(grad[a] - F * dv / kcal).max() <= 1e-10 * big
            assert abs(ad[a] - A * dv / kcal) <= 1e-10 * (np.abs(ad).max() + 1e-30)


def test_atom_integrals_of_two_million_atoms(tmp_path, solvents):
    """More groups of 32 atoms than a grid has rows (65535): the first and the
    last atom, alike, get the same numbers; those between have no charge and no
    depth."""
    import rism3d as R
    nu = 65536 * 32 + 1
    real, ghost = "3.0 0.2 0.3 1.0 1.0 1.0\n", "3.0 0.0 0.0 0.0 0.0 0.0\n"
    inp = str(tmp_path / "many.inp")
    with open(inp, "w") as f:
        f.write(" m 0 20220301\n KH\n %s\n 1.0e-6 1\n 2 0.6 0.2\n 8.0 8.0 4.0\n 16 16 8\n %d\n"
                % (solvents["h2o_vv"], nu))
        f.write(real + ghost * (nu - 2) + real)
    s = R.RISM3D(precision="fp64")
    s.initialize(inp, xvk=solvents["h2o_vv"])
    s.iterate()
    grad, euv, ad = s.atom_integrals()
    s.close()
    assert np.isfinite(grad).all() and np.abs(grad[0]).min() > 0 and np.abs(euv[0]).min() > 0
    for a in (grad, euv, ad):
        assert np.array_equal(a[0], a[-1]) and not a[1:-1].any()


def test_grid_copy_to_page_locked_memory(tmp_path, solvents):
    import ctypes
    import torch
    import rism3d as R
    import synthetic as S
    xvk = solvents["h2o_vv"]
    inp = S.small(str(tmp_path), nu=4, grid=(80, 72, 64), box=(40.0, 36.0, 32.0), solvent=xvk)
    s = R.RISM3D(precision="mixed")
    s.initialize(inp, xvk=xvk)
    for which in ("u", "fk"):
        ref = s.get(which)  # pageable
        n = ref.size * (2 if np.iscomplexobj(ref) else 1)
        buf = torch.empty(n, dtype=torch.float64).pin_memory()
        rc = R.lib.r3d_get_grid(s.h, R.GRID[which],
                                ctypes.cast(buf.data_ptr(), ctypes.POINTER(ctypes.c_double)))
        assert rc == 0
        assert np.array_equal(buf.numpy(), np.ascontiguousarray(ref).view(np.float64).reshape(-1))
    s.close()


# the rule that leaves a geometry to the per-axis passes: a default solve is
# the pinned plane-pass solve where it does not apply, and close to it where it
# does (more than one round of planes; tiles; the shortest rows)
@pytest.mark.parametrize("precision,n,dims,plane", [
    ("mixed", 4, (64, 72, 80), False), ("mixed", 4, (80, 64, 64), True),
    ("mixed", 2, (128, 128, 40), False), ("mixed", 2, (32, 32, 32), False),
    ("mixed", 2, (48, 48, 40), True), ("fp64", 4, (80, 72, 80), False),
    ("fp64", 4, (64, 72, 80), True),
    # few planes; row tiles; a round that the planes fill, with other rows and z
    ("fp64", 2, (64, 144, 24), False), ("mixed", 2, (64, 72, 48), False),
    ("fp64", 2, (96, 96, 32), False), ("mixed", 2, (256, 128, 80), False),
    ("mixed", 2, (288, 128, 24), False), ("mixed", 2, (128, 72, 128), False),
    ("fp64", 4, (96, 80, 80), True), ("mixed", 4, (144, 72, 40), True)])
def test_default_passes_by_geometry(tmp_path, monkeypatch, solvents, precision, n, dims, plane):
    import rism3d as R
    import synthetic as S
    xvk = solvents["h2o_vv" if n == 2 else "naclaq_vv"]
    inp = S.small(str(tmp_path), nu=12, grid=dims, box=tuple(0.5 * k for k in dims), solvent=xvk, seed=3)
    out = []
    for variant in (None, "5"):
        if variant:
            monkeypatch.setenv("R3D_X_VARIANT", variant)
        s = R.RISM3D(precision=precision)
        s.load(inp, xvk=xvk)
        s.initialize()
        s.step(4)
        out.append(s.get("g"))
        s.close()
    same = np.array_equal(out[0], out[1])
    assert same == plane
    # four iterations' roundings: FP32 spectra 1e-5 of the largest g, FP64 1e-10
    assert np.abs(out[0] - out[1]).max() <= (1e-5 if precision == "mixed" else 1e-10) * np.abs(out[1]).max()
