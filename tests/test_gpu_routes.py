"""The rules that choose between kernels: what a rule lets in gets the result
it gets by any other route."""
import numpy as np
import pytest

from ps3d_b200 import abi
from ps3d_b200.model import Model
from ps3d_b200.serve import Server, request
from oracle.binding import Oracle
from tests.helpers import FIELDS, compare_state, load_oracle, random_state, small_params

pytestmark = pytest.mark.gpu
TOL_KERNEL = 1e-12   # one FP64 pressure solve


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
