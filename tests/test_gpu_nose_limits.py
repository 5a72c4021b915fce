"""FP64 Nose-Hoover at the limits of its implicit velocity step
(int-verlet-nh-mav.f:105-180): a PSI or a thermostat mass at which a step turns
velocities round (1 + dt PSI / 2 <= 0, or the closed form leaves that domain
from a cold start), and a NaN, which the reference carries on.  The engine's
FP64 step kernels against the oracle's sweeps: the same status, and PSI and the
velocities within 1e-8 (the sweeps settle to 1e-10 per component; inputs moved
by 1e-13 move neither by more than that)."""
import ctypes as C

import numpy as np
import pytest

import clmd
import orc
from conftest import random_state

pytestmark = pytest.mark.gpu

# thermostat mass (of N T), PSI, velocities (of thermal)
LIMITS = {"psi-600": (0.25, -600.0, 1.0), "psi-1500": (0.25, -1500.0, 1.0),
          "mass1e-5": (1e-5, 0.0, 0.1), "mass1.8e-5": (1.8e-5, 0.0, 0.1),
          "mass2.2e-5": (2.2e-5, 0.0, 0.1), "ordinary": (0.25, 0.0, 1.0)}


def start(n, mass, psi, scale, nan=False):
    cfg = clmd.lj_config(n, 0.04, 0.8, ethst="N", integrator=clmd.INT_NOSE, q=n * 0.8 * mass)
    o = orc.Oracle(cfg, neighbor_mode=1 if n > 64 else 0)
    o.set_state(random_state(cfg, 3 + n), scalars=orc.scalars_init(cfg))
    o.stopdead(-1)
    o.neighbor(0)
    o.zero_acc()
    o.accatom()
    s, q = o.get_state(), o.scalars()
    for k in ("vx", "vy", "vz"):
        setattr(s, k, getattr(s, k) * scale)
    if nan:
        s.vx[n // 2] = np.nan
    q.psi = psi
    o.set_state(s, scalars=q)
    g = clmd.System(cfg)
    g.set_state(s, scalars=q)
    g.neighbor(0)
    g.set_scalars(q)
    return g, o


@pytest.mark.parametrize("n", [33, 8192, 8193])  # one cluster, the grid
@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("steps", [1, 2])
def test_nose_limits(gpu, n, limit, steps):
    g, o = start(n, *LIMITS[limit])
    g.steps(1, steps)
    for i in range(1, steps + 1):
        o.integrator(i)
    sg, so = g.scalars(), o.scalars()
    assert so.status == 0 and sg.status == 0
    assert abs(sg.psi - so.psi) <= 1e-8 * max(abs(so.psi), 1.0)
    assert abs(sg.nh_iters - so.nh_iters) <= 1
    a, b = g.get_state(), o.get_state()
    scale = np.abs(b.vx).max()
    for k in ("vx", "vy", "vz"):
        np.testing.assert_allclose(getattr(a, k), getattr(b, k), rtol=0, atol=1e-8 * scale)


@pytest.mark.parametrize("n", [33, 8193])
def test_nose_nan(gpu, n):
    g, o = start(n, 0.25, 0.0, 1.0, nan=True)
    g.steps(1, 2)
    for i in (1, 2):
        o.integrator(i)
    sg, so = g.scalars(), o.scalars()
    assert so.status == 0 and sg.status == 0 and np.isnan(so.psi) and np.isnan(sg.psi)
    assert (sg.nh_iters, so.nh_iters) == (1, 1)
    assert np.isnan(g.get_state().vx).all()


@pytest.mark.parametrize("n", [33, 8193])
@pytest.mark.parametrize("apart", [0.5, 0.1, 0.02])
@pytest.mark.parametrize("precision,tol", [(clmd.PREC_FP64, 1e-8), (clmd.PREC_MIXED, 1e-5)])
def test_nose_overlap(gpu, n, apart, precision, tol):
    """Two atoms that nearly coincide, their first forces met inside the step:
    the velocity solve's sum is up to 1e50 times the thermal one.  (Mixed: PSI
    goes with the 2/3 power of the force, whose FP32 terms hold to 1e-6.)"""
    cfg = clmd.lj_config(n, 0.04, 0.8, ethst="N", integrator=clmd.INT_NOSE)
    st = random_state(cfg, 3 + n)
    st.x[1], st.y[1], st.z[1] = st.x[0] + apart, st.y[0], st.z[0]
    st.vx[1], st.vy[1], st.vz[1] = st.vx[0], st.vy[0], st.vz[0]
    o = orc.Oracle(cfg, neighbor_mode=1 if n > 64 else 0)
    o.set_state(st, scalars=orc.scalars_init(cfg))
    o.neighbor(0)
    cfg.precision = precision
    g = clmd.System(cfg)
    g.set_state(st, scalars=clmd.scalars_init(cfg))
    g.neighbor(0)
    o.integrator(1)
    g.integrator(1)
    sg, so = g.scalars(), o.scalars()
    assert so.status == 0 and sg.status == 0
    assert abs(sg.psi - so.psi) <= tol * abs(so.psi)
    a, b = g.get_state(), o.get_state()
    np.testing.assert_allclose(a.vx, b.vx, rtol=0, atol=10 * tol * np.abs(b.vx).max())


@pytest.mark.parametrize("n", [400, 10000])  # one CTA, a cluster
@pytest.mark.parametrize("limit", ["mass1e-5", "mass1.8e-5", "mass2.2e-5", "nan"])
def test_nose_limits_ensemble(gpu, n, limit):
    """The same for a replica of the FP64 ensemble whose velocities the caller
    cools (or sets a NaN among) between two of its steps."""
    mass, _, scale = LIMITS.get(limit, LIMITS["ordinary"])
    cfg = clmd.lj_config(n, 0.04, 0.8, ethst="N", integrator=clmd.INT_NOSE, q=n * 0.8 * mass)
    st = random_state(cfg, n)
    e = clmd.Ensemble(clmd.ens_config(n, 1, ftcsi=1, precision=clmd.PREC_FP64))
    slot = e.add(n, cfg.boxx, 0.8, st.x, st.y, st.z, st.vx, st.vy, st.vz, csover=10**6, q=cfg.Q)
    e.step(1)
    st, _ = e.state(slot)
    for k in ("vx", "vy", "vz"):
        setattr(st, k, getattr(st, k) * scale)
    if limit == "nan":
        st.vx[n // 2] = np.nan
    v = [np.ascontiguousarray(a) for a in (st.vx, st.vy, st.vz)]
    assert e.lib.clmd_ens_upload(e.h, None, None, None,
                                 *[clmd.ptr(a, C.c_double) for a in v]) == 0
    o = orc.Oracle(cfg, neighbor_mode=1)
    q = orc.scalars_init(cfg)
    q.psi, q.s = e.results()[slot].psi, e.results()[slot].s
    o.set_state(st, scalars=q)
    o.neighbor(0)
    for i in (1, 2):
        o.integrator(i)
        e.step(1)
        r, s = e.results()[slot], o.scalars()
        assert s.status == 0 and r.status == 0 and r.step == i + 1
        a, b = e.state(slot)[0], o.get_state()
        if limit == "nan":
            assert np.isnan(s.psi) and np.isnan(r.psi)
            assert np.isnan(a.vx).all() and np.isnan(b.vx).all()
            continue
        assert abs(r.psi - s.psi) <= 1e-8 * abs(s.psi)
        for k in ("vx", "vy", "vz"):
            np.testing.assert_allclose(getattr(a, k), getattr(b, k), rtol=0,
                                       atol=1e-8 * np.abs(b.vx).max())
