"""The rules that choose between kernels: what a rule lets in gets the result
it gets by any other route."""
import numpy as np
import pytest

from ps3d_b200 import abi
from ps3d_b200 import configs as cf
from ps3d_b200.model import Model, PS3DError
from ps3d_b200.serve import Server, request
from ps3d_b200.slab import Slab, SlabGroup
from oracle.binding import Oracle
from tests.helpers import (FIELDS, compare_state, load_oracle, random_state, small_params, smooth_state,
                           upload_from_oracle)

pytestmark = pytest.mark.gpu
TOL_KERNEL = 1e-12   # one FP64 pressure solve or projection
TOL64 = 1e-11        # several FP64 steps: the suite's bound for rounding in another order
TOL_MIXED = 1e-5     # the mixed path


def _pair(p, f):
    o, m = Oracle(p), Model(p)
    load_oracle(o, f)
    upload_from_oracle(m, o)
    return o, m


def _projected(o, m, p, tol):
    """One pressure solve against the oracle; a velocity carries p's rounding
    times dt over its grid distance."""
    o.pressure_solver()
    m.pressure_solver()
    got = m.download(tendencies=False)
    pn = np.linalg.norm(cf.interior(o.field("p")))
    for k, d in (("p", None), ("u", p.dx), ("v", p.dy), ("w", p.dz)):
        want = cf.interior(o.field(k))
        t = tol * np.linalg.norm(want) + (8 * np.finfo(float).eps * p.dt / d * pn if d else 0.0)
        assert np.linalg.norm(cf.interior(got[k]) - want) <= t, (k, np.linalg.norm(cf.interior(got[k]) - want), t)


@pytest.mark.parametrize("n", [(128, 16, 8), (96, 20, 10)])
def test_batched_requests_match_alone_on_wide_grids(n, monkeypatch):
    """FP64 requests whose nx/2+1 fits the SMs alone but not times the group:
    each gets bit for bit its result alone, in a group and afterwards alone
    in the group's pooled context."""
    monkeypatch.setenv("PS3D_AUTOTUNE", "0")
    p, opt, f = request(*n, precision=abi.PS3D_FP64, ramp_steps=6, iters=2)
    states = [{k: v * a for k, v in f.items()} for a in (1.0, 1.7, 0.6, 2.5)]
    s = Server(max_active=1)
    alone = [s.wait(s.submit(p, opt, st)) for st in states]
    s.close()
    s = Server(max_active=1, max_batch=4)
    blocker = s.submit(*request(64, 32, 16, precision=abi.PS3D_FP64, ramp_steps=60, iters=4))
    tks = [s.submit(p, opt, st) for st in states]   # queue up behind the blocker
    assert s.wait(blocker).status == 0
    got = [s.wait(t) for t in tks]
    assert abs(got[3].queue_ms - got[0].queue_ms) < got[0].run_ms   # one group
    last = s.wait(s.submit(p, opt, states[3]))
    s.close()
    for a, g in list(zip(alone, got)) + [(alone[3], last)]:
        assert a.status == g.status == 0 and g.iters == a.iters and g.norm == a.norm
        for k in ("u", "v", "w", "b"):
            assert np.array_equal(g.fields[k], a.fields[k]), k


@pytest.mark.parametrize("pin,fused", [("im0,C1,rc4,tj8,ly8,pol1,kc4", 0), ("im1,C1,rc8,tj16,ly16,pol1,kc4", 1),
                                       ("im2,C1,rc8,tj8,ly16,pol2,kc4", 1)])
def test_pinned_fused_solve(pin, fused, monkeypatch):
    """A pin's suffix yf1 takes the fused y transforms and vertical solve where
    the pinned plane form feeds them, and is without effect on the cluster
    form, which transforms along y itself."""
    monkeypatch.setenv("PS3D_TUNE", pin + ",yf1")
    p = small_params(32, 32, 10, rigid=True)
    f = random_state(p, seed=51)
    o, m = Oracle(p), Model(p)
    load_oracle(o, f)
    m.upload(**{k: f[k] for k in FIELDS})
    o.pressure_solver()
    m.pressure_solver()
    assert f"yfused={fused}" in m.describe() and "tuned=pinned" in m.describe()
    err = compare_state(m, o)
    assert max(err.values()) < TOL_KERNEL, err


@pytest.mark.parametrize("form", ["fused", "0", "2", "3"])
@pytest.mark.parametrize("impl", ["0", "1"])
@pytest.mark.parametrize("nz", [3, 16, 41])
def test_columns_without_a_wavenumber(nz, impl, form, monkeypatch):
    """Lx = nx dx / 2 and Ly = ny dy / 2: besides (0,0), the columns at kx =
    nx/2, at ky = ny/2 and at both have no horizontal wavenumber, and the
    vertical solve takes them by the (0,0) recurrence, part by part."""
    if form == "fused" and impl == "0":
        pytest.skip("the cluster kernels transform along y themselves")
    monkeypatch.setenv("PS3D_AUTOTUNE", "0")
    monkeypatch.setenv("PS3D_PLANE_IMPL", impl)
    monkeypatch.setenv("PS3D_YFUSED", "1" if form == "fused" else "0")
    if form != "fused":
        monkeypatch.setenv("PS3D_THOMAS_FORM", form)
    p = small_params(16, 12, nz, rigid=True, dx=2 * 32e3 / 16, dy=2 * 32e3 / 12)
    o, m = _pair(p, random_state(p, seed=52))
    assert f"yfused={int(form == 'fused')}" in m.describe()
    _projected(o, m, p, TOL_KERNEL)


@pytest.mark.parametrize("n", [(18, 10, 64), (20, 6, 128), (20, 6, 50)])
def test_periodic_solve_mixed(n):
    """The periodic solve on FP32 spectra, in registers and staged."""
    p = small_params(*n, rigid=False)
    f = random_state(p, seed=54)
    o = Oracle(p)
    load_oracle(o, f)
    p.precision = abi.PS3D_MIXED
    m = Model(p)
    m.upload(**{k: f[k] for k in FIELDS})
    _projected(o, m, p, TOL_MIXED)


@pytest.mark.parametrize("mode", [abi.PS3D_PROJ_NORMAL_MODE, abi.PS3D_PROJ_EXCHANGE])
@pytest.mark.parametrize("n", [(18, 10, 32), (12, 10, 64), (10, 6, 128), (8, 6, 256)])
def test_periodic_projection_in_registers(n, mode):
    """The forward-only and inverse-only z transforms on columns in registers,
    with a last block that is not full."""
    p = small_params(*n, rigid=False, Lz=1000.0 * n[2] / 16)
    o, m = _pair(p, smooth_state(p, seed=55))
    if mode == abi.PS3D_PROJ_EXCHANGE:
        o.project(abi.PS3D_PROJ_BASE_POINT)
        m.project(abi.PS3D_PROJ_BASE_POINT)
    o.project(mode)
    m.project(mode)
    err = compare_state(m, o, names=FIELDS)
    assert max(err.values()) < TOL_KERNEL, err


@pytest.mark.parametrize("harmonic", [False, True])
@pytest.mark.parametrize("n", [(64, 64, 23), (64, 128, 23), (64, 180, 23), (256, 256, 5), (64, 128, 20)])
def test_biharmonic_friction_marches(n, harmonic):
    """Biharmonic friction on grids where a block of its kernel (two an SM)
    marches over chunks of 2, 3, 4 and 5 levels, the last one shorter or
    with the lid in it; nz = 20: triply periodic."""
    p = small_params(*n, rigid=n[2] != 20, Ahbi=1e7, Avbi=1e1, Khbi=1e7, Kvbi=1e1,
                     **({} if harmonic else dict(Ah=0.0, Av=0.0)))
    o, m = _pair(p, smooth_state(p, seed=56))
    o.integrate(3)
    m.run(3)
    err = compare_state(m, o)
    assert max(err.values()) < TOL64, err


@pytest.mark.parametrize("ny,taken", [(2, False), (4, False), (10, False), (36, False), (8, True), (24, True)])
@pytest.mark.parametrize("precision", [abi.PS3D_FP64, abi.PS3D_MIXED])
def test_slabs_take_rows_in_eights(ny, taken, precision):
    """z-slabs exist for grids whose ny is a multiple of 8 and are refused for
    others, which whole grids take in shorter runs of rows."""
    p = small_params(16, ny, 8, rigid=True, precision=precision)
    Model(p).close()
    if taken:
        Slab(p, 2, 0).close()
    else:
        with pytest.raises(PS3DError) as e:
            Slab(p, 2, 0)
        assert e.value.status == abi.PS3D_ERR_UNSUPPORTED


@pytest.mark.parametrize("rigid", [True, False])
def test_slab_download_in_mid_run(rigid, monkeypatch):
    """Every level of a slab run, w at the top one included, is the single
    grid's, at a download between steps and after further steps."""
    monkeypatch.setenv("PS3D_PLANE_IMPL", "1")
    p = small_params(16, 8, 20, rigid=rigid, Lz=1250.0)
    f = random_state(p, seed=58)
    m, s = Model(p), SlabGroup(p, 2)
    m.upload(**{k: f[k] for k in FIELDS})
    s.upload(*[np.ascontiguousarray(cf.interior(f[k])) for k in FIELDS])
    for n in (2, 3):
        m.run(n)
        s.step(n)
        ref, got = m.download(tendencies=False), s.download()
        for k in FIELDS + ("p",):
            want = cf.interior(ref[k])
            assert np.linalg.norm(got[k] - want) < TOL64 * np.linalg.norm(want), (n, k)
    s.close()


@pytest.mark.parametrize("rigid", [True, False])
def test_slabs_without_columns(rigid, monkeypatch):
    """More ranks than spectral columns: some slabs hold none and solve none."""
    monkeypatch.setenv("PS3D_PLANE_IMPL", "1")
    p = small_params(2, 8, 40, rigid=rigid, Lz=2500.0)   # 16 columns
    f = random_state(p, seed=57)
    m = Model(p)
    m.upload(**{k: f[k] for k in FIELDS})
    m.run(3)
    ref = m.download(tendencies=False)
    s = SlabGroup(p, 20)
    s.upload(*[np.ascontiguousarray(cf.interior(f[k])) for k in FIELDS])
    s.step(3)
    got = s.download()
    s.close()
    for k in FIELDS + ("p",):
        want = cf.interior(ref[k])
        assert np.linalg.norm(got[k] - want) < TOL64 * np.linalg.norm(want), k
