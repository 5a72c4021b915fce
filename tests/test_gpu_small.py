"""The step kernel of small systems (one thread-block cluster, one atom per
thread) at the edges of its range: one and several CTAs, partial warps, the
largest size and the first beyond it, rows longer than the search's buffer.
FP64 velocity Verlet is bit-identical to the oracle; Nose-Hoover and the
energy sums agree within the rounding of the sums, mixed precision within
the FP32 rounding of the pair terms over a few steps."""
import ctypes as C

import numpy as np
import pytest

import clmd
import orc
from conftest import droplet_state, random_state, start_pair

pytestmark = pytest.mark.gpu

SIZES = [3, 32, 33, 128, 129, 1000, 2048, 2049, 4097, 8192, 8193]


def rel(a, b):
    return abs(a - b) / max(abs(b), 1e-300)


@pytest.mark.parametrize("n", SIZES)
def test_small_verlet_bit_exact(gpu, n):
    cfg = clmd.lj_config(n, 0.01 if n < 10 else 0.04, 0.8)
    g, o = clmd.System(cfg), orc.Oracle(cfg, neighbor_mode=1 if n > 64 else 0)
    start_pair(g, o, cfg, random_state(cfg, 5 + n))
    g.steps(1, 25)
    for i in range(1, 26):
        o.integrator(i)
    a, b = g.get_state(), o.get_state()
    for k in ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    for u, v in zip(g.halflist(), o.halflist()):
        assert np.array_equal(u, v)
    sg, so = g.scalars(), o.scalars()
    assert (sg.nrebuild, sg.dmmst, sg.atrskin) == (so.nrebuild, so.dmmst, so.atrskin)
    # sums of n terms in another order: n ulps at most of the terms' scale
    assert abs(sg.ekin - so.ekin) <= 1e-12 * so.ekin
    assert abs(sg.epot - so.epot) <= 1e-12 * max(abs(so.epot), 1.0)


@pytest.mark.parametrize("n", [33, 129, 2049, 8192, 8193])
@pytest.mark.parametrize("ethst", ["N", "X"])
def test_small_thermostats(gpu, n, ethst):
    cfg = clmd.lj_config(n, 0.04, 0.8, ethst=ethst,
                         integrator=clmd.INT_NOSE if ethst == "N" else clmd.INT_VERLET)
    if ethst == "X":
        cfg.apth = b"X" + b"-" * (clmd.MXSORTS - 1)
    g, o = clmd.System(cfg), orc.Oracle(cfg, neighbor_mode=1 if n > 64 else 0)
    start_pair(g, o, cfg, random_state(cfg, 9 + n))
    g.run(1, 20)
    o.run(1, 20)
    a, b = g.get_state(), o.get_state()
    # 20 steps amplify the sums' rounding (1e-15) by far less than 1e4
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        np.testing.assert_allclose(getattr(a, k), getattr(b, k), rtol=1e-9, atol=1e-10)
    sg, so = g.scalars(), o.scalars()
    assert rel(sg.ekin, so.ekin) < 1e-11
    if ethst == "N":
        assert abs(sg.psi - so.psi) < 1e-11
        assert abs(sg.nh_iters - so.nh_iters) <= 1


@pytest.mark.parametrize("drops,radius", [(2, 3.4), (1, 7.0)])
def test_small_long_rows_bit_exact(gpu, drops, radius):
    """Rows of ~100 entries (liquid droplets) and, at the largest list radius
    in the denser blob, of more."""
    cfg = clmd.lj_config(4000, 0.03, 0.7, rskin=3.4)
    g, o = clmd.System(cfg), orc.Oracle(cfg, neighbor_mode=1)
    start_pair(g, o, cfg, droplet_state(cfg, 3, drops, radius))
    for u, v in zip(g.halflist(), o.halflist()):
        assert np.array_equal(u, v)
    g.steps(1, 12)
    for i in range(1, 13):
        o.integrator(i)
    a, b = g.get_state(), o.get_state()
    for k in ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k


@pytest.mark.parametrize("n", [129, 4097])
def test_small_mixed_forces(gpu, n):
    cfg = clmd.lj_config(n, 0.05, 0.75, precision=clmd.PREC_MIXED, integrator=clmd.INT_NOSE,
                         ethst="N")
    g, o = clmd.System(cfg), orc.Oracle(cfg, neighbor_mode=1)
    start_pair(g, o, cfg, random_state(cfg, 77))
    g.integrator(1)
    o.integrator(1)
    a, b = g.get_state(), o.get_state()
    ga = np.stack([a.ax, a.ay, a.az])
    oa = np.stack([b.ax, b.ay, b.az])
    assert np.linalg.norm(ga - oa) <= 1e-5 * np.linalg.norm(oa)
    assert g.scalars().status == 0


def block_tree(e):
    """The sum of e over blocks of 256 as a block reduces it: xor butterflies
    over 32 lanes, over a block's 8 warps, then over the blocks."""
    def butterfly(v):
        for o in (16, 8, 4, 2, 1):
            v = v + v[..., np.arange(32) ^ o]
        return v[..., 0]
    nb = -(-len(e) // 256)
    v = np.zeros(256 * nb)
    v[:len(e)] = e
    warps = np.zeros((nb, 32))
    warps[:, :8] = butterfly(v.reshape(nb, 8, 32))
    blocks = np.zeros(32)
    blocks[:nb] = butterfly(warps)
    return butterfly(blocks)


@pytest.mark.parametrize("n", [3, 33, 256, 257, 2011, 5000, 8191, 8192])
@pytest.mark.parametrize("two", [False, True])
def test_velocity_scaling_bits(gpu, n, two):
    """Velocity scaling of small systems (one launch): the factor of each
    species, and with it every velocity, to the last bit of the tree of sums
    that larger systems use (all atoms in input order, no list yet)."""
    n2 = n // 3 if two else 0
    cfg = clmd.lj_config(n, 0.02, 0.8, species=dict(n=n2, mass=1.7) if two else None)
    cfg.apth = b"XX" + b"-" * (clmd.MXSORTS - 2)
    rng = np.random.default_rng(n)
    st = random_state(cfg, n) if n > 3 else clmd.State(*rng.uniform(0, cfg.boxx, (3, n)),
                                                       *rng.normal(size=(3, n)),
                                                       *np.zeros((3, n)))
    api = np.r_[np.full(n - n2, 1), np.full(n2, 2)].astype(np.int32) if two else None
    g = clmd.System(cfg)
    g.set_state(st, api=api, scalars=clmd.scalars_init(cfg))
    v = np.stack([st.vx, st.vy, st.vz])
    sp = np.r_[np.zeros(n - n2, int), np.ones(n2, int)]
    mass = np.array([1.0, 1.7])
    e = 0.5 * mass[sp] * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
    g.thermostat(1)
    out = g.get_state()
    for s in range(2 if two else 1):
        m = sp == s
        kf = np.sqrt(1.5 * clmd.CIKB * cfg.att * m.sum() / block_tree(np.where(m, e, 0.0)))
        for got, was in zip((out.vx, out.vy, out.vz), v):
            assert np.array_equal(got[m], was[m] * kf), s


@pytest.mark.parametrize("n", [64, 2049, 9000])  # one cluster, the grid
def test_bad_species_leaves_positions(gpu, n):
    """A pair of species without coefficients stops a run in its first force
    pass: the positions are those of that step, whether the launch would have
    gone on with the next step's drift or not."""
    cfg = clmd.lj_config(n, 0.05, 0.8)
    cfg.atsorts = 3
    for s, (k, m) in enumerate(((n // 2, 1.0), (n // 4, 1.0), (n - n // 2 - n // 4, 1.0))):
        cfg.apnum[s], cfg.apmas[s], cfg.apsig[s], cfg.apeps[s] = k, m, 1.0, 1.0
    st = random_state(cfg, n)
    out = []
    for steps in (1, 3):
        g = clmd.System(cfg)
        g.set_state(st, scalars=clmd.scalars_init(cfg))
        g.neighbor(0)
        assert g.lib.clmd_steps(g.h, 1, steps) == clmd.ERR_BAD_SPECIES
        x = [np.zeros(n) for _ in range(3)]
        g.lib.clmd_get_state(g.h, *[clmd.ptr(a, C.c_double) for a in x], *([None] * 7))
        out.append(x)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
