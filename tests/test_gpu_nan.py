"""Atoms at a NaN through a list rebuild: their cell is a valid one (a NaN
converts to the smallest integer, which must not become a cell number), they
are nobody's neighbours, and the others' lists and forces are complete."""
import numpy as np
import pytest

import clmd

pytestmark = pytest.mark.gpu

RSKIN = 2.8


def positions(n, rho, seed):
    """Random positions with three atoms at a NaN in one or all coordinates,
    and the others' indices."""
    box = (n / rho) ** (1.0 / 3.0)
    x = list(np.random.default_rng(seed).uniform(0, box, (3, n)))
    x[0][5] = x[1][7] = np.nan
    for a in x:
        a[9] = np.nan
    return box, x, np.delete(np.arange(n), [5, 7, 9])


def ordered_pairs(x, ok, box, r):
    from scipy.spatial import cKDTree

    t = cKDTree(np.stack([a[ok] for a in x], 1), boxsize=box)
    return t.count_neighbors(t, r) - len(ok)


@pytest.mark.parametrize("n,rho", [(40, 0.3), (300, 0.05), (2049, 0.05), (8192, 0.02),
                                   (8193, 0.02), (60000, 0.02)])
@pytest.mark.parametrize("precision", [clmd.PREC_FP64, clmd.PREC_MIXED])
def test_system_rebuild(gpu, n, rho, precision):
    cfg = clmd.lj_config(n, rho, 0.7, precision=precision, rskin=min(RSKIN, 2.51) if n < 100
                         else RSKIN)
    box, x, ok = positions(n, rho, n)
    z = np.zeros(n)
    g = clmd.System(cfg)
    g.set_state(clmd.State(*x, *np.zeros((3, n)), z, z, z), scalars=clmd.scalars_init(cfg))
    g.neighbor(0)
    g.zero_acc()
    g.accatom()
    s = g.scalars()
    assert s.status == 0
    assert 2 * s.npairs_half == ordered_pairs(x, ok, box, cfg.atrskin)
    st = g.get_state()
    assert np.isfinite(np.stack([st.ax, st.ay, st.az])[:, ok]).all()


@pytest.mark.parametrize("n,rho", [(60, 0.35), (300, 0.05), (8200, 0.05), (12000, 0.03)])
def test_replica_rebuild(gpu, n, rho):
    """Candidates in and outside shared memory, and a cluster; some atoms near
    the origin, where the cell of the NaNs is."""
    box, x, ok = positions(n, rho, n)
    for a in x:
        a[20:28] = np.random.default_rng(1).uniform(0, 0.4, 8)
    v = np.random.default_rng(n).normal(size=(3, n)) * 1e-9
    e = clmd.Ensemble(clmd.ens_config(n, 1, ftcsi=1, rskin=RSKIN, integrator=clmd.INT_VERLET,
                                      precision=clmd.PREC_FP64, dt=1e-30, list_stride=512))
    assert e.add(n, box, 0.7, *x, *v, ethst="-") is not None
    e.step(1)
    r = e.results()[0]
    assert r.status == 0 and r.nrebuild == 1
    assert e.pair_terms() == ordered_pairs(x, ok, box, RSKIN)
    st, _ = e.state(0)
    assert np.isfinite(np.stack([st.ax, st.ay, st.az])[:, ok]).all()
