"""Edges of the kernels' tiles and batches: grids that are no multiple of a
tile, the smallest grids, z chunks of every size, against the oracle or
bit for bit against another split of the same work."""
import numpy as np
import pytest

from ps3d_b200 import abi
from ps3d_b200 import configs as cf
from ps3d_b200.model import Model
from oracle.binding import Oracle
from tests.test_zz_no_alloc import _noalloc
from tests.helpers import (FIELDS, compare_state, load_oracle, random_state, small_params, smooth_state,
                           upload_from_oracle)

pytestmark = pytest.mark.gpu
TOL_KERNEL = 1e-12   # one FP64 pressure solve
TOL64 = 1e-11   # several FP64 steps: the suite's bound for rounding in another order

FRICTION = {"none": dict(Ah=0.0, Av=0.0), "uvw": {}, "uvwb": dict(Kh=2e-2, Kv=1e-2)}


def _pair(p, f):
    o, m = Oracle(p), Model(p)
    load_oracle(o, f)
    upload_from_oracle(m, o)
    return o, m


@pytest.mark.parametrize("friction", sorted(FRICTION))
@pytest.mark.parametrize("n", [(4, 4, 2), (36, 10, 3), (64, 8, 5), (30, 18, 7)])
@pytest.mark.parametrize("rigid", [True, False])
def test_step_at_tile_edges(n, friction, rigid):
    """Four AB3 steps (cold, one and two history levels, a pending
    correction) on grids narrower and wider than the 32 x 8 column tile."""
    nz = n[2] if rigid else max(2, 2 * (n[2] // 2))
    p = small_params(n[0], n[1], nz, rigid=rigid, **FRICTION[friction])
    o, m = _pair(p, smooth_state(p, seed=31))
    o.integrate(4)
    m.run(4)
    err = compare_state(m, o)
    assert max(err.values()) < TOL64, err


@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("precision", [abi.PS3D_FP64, abi.PS3D_MIXED])
def test_step_z_chunks_give_the_same_bits(precision, forced, monkeypatch):
    """Any z chunk of the step kernel (a block's carried fluxes start anew at
    every chunk) gives the same bits."""
    ref = None
    for kc in (13, 1, 2, 3, 5):
        monkeypatch.setenv("PS3D_TUNE", f"im0,C1,rc4,tj8,ly8,pol1,kc{kc}")
        p = small_params(36, 20, 13, rigid=True, precision=precision)
        if forced:
            p.Ah = p.Av = 0.0
        m = Model(p)
        f = smooth_state(p, seed=32)
        m.upload(**{k: f[k] for k in FIELDS})
        if forced:
            rng = np.random.default_rng(33)
            g = {k: cf.halo_fill(a * rng.standard_normal(m.shape)) for k, a in
                 (("w_r", 1e-6), ("b_i", 1e-8), ("u_back", 0.1), ("b_back", 1e-4))}
            m.set_forcing(abi.PS3D_FORCE_WAVEMAKER | abi.PS3D_FORCE_BACKGROUND, omega=5e-4, **g)
        m.run(5)
        got = m.download()
        assert f"kchunk={kc}" in m.describe()
        if ref is None:
            ref = got
        for k in FIELDS + ("p", "du", "dv", "dw", "db"):
            assert np.array_equal(got[k], ref[k]), (kc, k)


@pytest.mark.parametrize("n", [(2, 2, 2), (4, 2, 3), (30, 18, 7), (270, 4, 5)])
def test_halo_layout_round_trip(n):
    """Upload takes the interior, download fills the halos periodically (p
    under a rigid lid: the nearest level), exactly."""
    p = small_params(*n, rigid=True, precision=abi.PS3D_FP64)
    m = Model(p)
    rng = np.random.default_rng(34)
    up = {k: rng.standard_normal(m.shape) for k in FIELDS + ("p",)}
    up["du"] = rng.standard_normal((3,) + m.shape)
    m.upload(**up)
    got = m.download()
    for k in FIELDS:
        assert np.array_equal(got[k], cf.halo_fill(up[k].copy())), k
    want = cf.halo_fill(up["p"].copy())
    for z, s in ((0, 2), (1, 2), (-1, -3), (-2, -3)):
        want[z] = want[s]
    assert np.array_equal(got["p"], want)
    for s in range(3):
        assert np.array_equal(got["du"][s], cf.halo_fill(up["du"][s].copy()))


@pytest.mark.parametrize("n", [(18, 10, 32), (18, 10, 64), (20, 6, 128), (16, 4, 256), (20, 6, 50)])
def test_periodic_z_solve_in_registers(n, monkeypatch):
    """Triply periodic solve on columns in registers (nz = 32 .. 256, a last
    block that is not full) and staged (nz = 50): FP64 against the oracle,
    FP32 spectra bit for bit against the staged form."""
    p = small_params(*n, rigid=False)
    o, m = _pair(p, random_state(p, seed=35))
    o.pressure_solver()
    m.pressure_solver()
    err = compare_state(m, o)
    # w - dt dp/dz: the two p of a difference agree to all but a few digits
    # at small dz, so w carries p's rounding times dt/dz
    norm = {k: np.linalg.norm(cf.interior(o.field(k))) for k in ("p", "w")}
    err["w"] -= 8 * np.finfo(float).eps * p.dt / p.dz * norm["p"] / norm["w"]
    assert max(err.values()) < TOL_KERNEL, err
    got = []
    for form in ("1", "0"):
        monkeypatch.setenv("PS3D_ZSOLVE", form)
        q = small_params(*n, rigid=False, precision=abi.PS3D_MIXED)
        mm = Model(q)
        f = random_state(q, seed=36)
        mm.upload(**{k: f[k] for k in FIELDS})
        mm.run(3)
        got.append(mm.download(tendencies=False))
    for k in FIELDS + ("p",):
        assert np.array_equal(got[0][k], got[1][k]), k


BIHARMONIC = {"all": dict(Ahbi=1e7, Avbi=1e1, Khbi=1e7, Kvbi=1e1), "horizontal": dict(Ahbi=1e7),
              "vertical": dict(Avbi=1e1, Kvbi=1e1)}


@pytest.mark.parametrize("mix", sorted(BIHARMONIC))
@pytest.mark.parametrize("harmonic", [False, True])
@pytest.mark.parametrize("n", [(4, 4, 2), (36, 10, 3), (64, 8, 5), (30, 18, 23)])
@pytest.mark.parametrize("rigid", [True, False])
def test_biharmonic_in_one_pass(n, harmonic, mix, rigid):
    """Biharmonic friction, wavemaker and Adams-Bashforth in one kernel: four
    AB3 steps, the state's correction pending (no harmonic friction) or
    applied, grids narrower and wider than the tile, odd z chunks."""
    nz = n[2] if rigid else {2: 2, 3: 4, 5: 6, 23: 24}[n[2]]
    p = small_params(n[0], n[1], nz, rigid=rigid, **({} if harmonic else FRICTION["none"]), **BIHARMONIC[mix])
    f = smooth_state(p, seed=37)
    o, m = _pair(p, f)
    rng = np.random.default_rng(38)
    g = {k: cf.halo_fill(a * rng.standard_normal(m.shape)) for k, a in (("u_r", 1e-6), ("u_i", 1e-6), ("b_i", 1e-9))}
    F = abi.Forcing()
    F.kind, F.omega = abi.PS3D_FORCE_WAVEMAKER, 5e-4
    F.u_r, F.u_i, F.b_i = (abi.dptr(g[k]) for k in ("u_r", "u_i", "b_i"))
    o.set_forcing(F, g)
    m.set_forcing(abi.PS3D_FORCE_WAVEMAKER, omega=5e-4, **g)
    o.integrate(4)
    m.run(4)
    err = compare_state(m, o)
    assert max(err.values()) < TOL64, err


@pytest.mark.parametrize("n", [(16, 4, 2), (16, 10, 3), (36, 20, 17), (32, 64, 32), (24, 80, 50), (16, 150, 65)])
def test_fused_y_transforms_and_vertical_solve(n, monkeypatch):
    """The FP64 y transforms and rigid-lid vertical solve in one block per kx
    (odd and even nz, more columns than threads) against the oracle, and
    against the separate kernels."""
    p = small_params(*n, rigid=True)
    f = random_state(p, seed=39)
    o = Oracle(p)
    load_oracle(o, f)
    o.pressure_solver()
    monkeypatch.setenv("PS3D_AUTOTUNE", "0")
    for form in ("1", "0"):
        monkeypatch.setenv("PS3D_YFUSED", form)
        m = Model(p)
        m.upload(**{k: f[k] for k in FIELDS})
        m.pressure_solver()
        assert f"yfused={form}" in m.describe()
        err = compare_state(m, o)
        assert max(err.values()) < TOL_KERNEL, (form, err)


@pytest.mark.parametrize("rigid", [True, False])
def test_noalloc_projection_shapes(rigid):
    """ps3d_pressure_solve_noalloc on grids of each route (y transforms with
    the vertical solve; y lines of their own where there are more kx than SMs;
    rows passes of 2 to 16 rows), one after the other and back again, so that
    each call finds another grid's tables."""
    grids = [(48, 40, 24), (6, 10, 4), (300, 16, 8), (32, 54, 20), (48, 40, 24), (8, 250, 16), (200, 2, 30)]
    for seed, n in enumerate(grids):
        p = small_params(*n, rigid=rigid)
        f = random_state(p, seed=40 + seed)
        o = Oracle(p)
        load_oracle(o, f)
        o.pressure_solver()
        got = _noalloc(p, f)
        pn = np.linalg.norm(cf.interior(o.field("p")))
        for k, d in (("p", None), ("u", p.dx), ("v", p.dy), ("w", p.dz)):
            want = cf.interior(o.field(k))
            # a velocity carries p's rounding times dt over its grid distance
            tol = TOL_KERNEL + (8 * np.finfo(float).eps * p.dt / d * pn / np.linalg.norm(want) if d else 0.0)
            assert np.linalg.norm(got[k] - want) <= tol * np.linalg.norm(want), (n, k)


@pytest.mark.parametrize("rigid", [True, False])
@pytest.mark.parametrize("n", [(18, 10, 6), (36, 30, 20), (128, 128, 70), (256, 128, 36)])
def test_projection_columns(n, rigid):
    """The eigenvector projection by columns: fewer columns than a block, a
    last block that is not full, chunks of 2, 4 and 8 levels with a remainder."""
    nz = n[2] if rigid else {6: 6, 20: 20, 70: 72, 36: 36}[n[2]]
    p = small_params(n[0], n[1], nz, rigid=rigid, Lz=1000.0 * nz / 16)
    o, m = _pair(p, smooth_state(p, seed=47))
    o.project(abi.PS3D_PROJ_NORMAL_MODE)
    m.project(abi.PS3D_PROJ_NORMAL_MODE)
    err = compare_state(m, o, names=FIELDS)
    assert max(err.values()) < TOL_KERNEL, err
