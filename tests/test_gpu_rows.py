"""The list search's FP32 test with its FP64 decision near the list radius,
and the rows' warp-wide sort, against the oracle's list, bit for bit: boxes
with fewer than three cells per dimension (alone or all), thin and long
boxes, a large sparse one, rows longer than the buffer and than a warp's
registers, atoms left outside the box by one length and by several, pairs
placed on the list radius."""
import numpy as np
import pytest

import clmd
import orc

pytestmark = pytest.mark.gpu


def lists(cfg, pos):
    n = cfg.natom
    z = np.zeros(n)
    st = clmd.State(*[np.ascontiguousarray(pos[:, k]) for k in range(3)], z, z, z, z, z, z)
    out = []
    for s in (clmd.System(cfg), orc.Oracle(cfg, neighbor_mode=0 if n < 12000 else 1)):
        s.set_state(st, scalars=(clmd if isinstance(s, clmd.System) else orc).scalars_init(cfg))
        s.neighbor(0)
        out.append((*s.halflist(), s.get_state()))
    return out


def same(cfg, pos):
    (gl, gi, gs), (ol, oi, os_) = lists(cfg, pos)
    assert np.array_equal(gi, oi) and np.array_equal(gl, ol)
    for k in ("x", "y", "z"):
        assert np.array_equal(getattr(gs, k), getattr(os_, k)), k


def boxed(n, box, **kw):
    cfg = clmd.lj_config(n, 0.05, 0.7, **kw)
    cfg.boxx, cfg.boxy, cfg.boxz = box
    return cfg


@pytest.mark.parametrize("n,box,kw", [
    (40, (6.0, 6.0, 6.0), {}),            # two cells per dimension
    (30, (5.7, 9.0, 30.0), {}),           # two, three and many
    (300, (5.6, 5.6, 90.0), {}),          # the list radius is half the box
    (9001, (8.5, 60.0, 80.0), {}),        # three cells in one dimension, grid kernel
    (9001, (6.0, 75.0, 90.0), {}),        # two in one dimension, grid kernel
    (3000, (1500.0, 1400.0, 1600.0), {}),  # sparse, coarse FP32 coordinates
    (60000, (1500.0, 1400.0, 1600.0), {}),
    (9000, (21.0, 22.0, 23.0), {}),       # liquid density, rows of ~80
    (4000, (15.0, 15.0, 15.0), dict(rskin=5.0, nlist_cap=4000000)),  # rows above 256
    (9000, (20.0, 20.0, 20.0), dict(rskin=5.0, nlist_cap=4000000)),
])
def test_rows_match_oracle(gpu, n, box, kw):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.3, 1.3, (n, 3)) * np.array(box)
    pos[: n // 50] += 5 * np.array(box)  # dmod proper
    same(boxed(n, box, **kw), pos)


@pytest.mark.parametrize("n", [400, 20000])
def test_pairs_on_the_list_radius(gpu, n):
    """Partners at the list radius times 1 +- a few ulps up to 1e-6, across the
    box's faces too."""
    box = np.array([60.0, 70.0, 80.0])
    rng = np.random.default_rng(3)
    a = rng.uniform(0, 1, (n // 2, 3)) * box
    d = rng.normal(size=(n // 2, 3))
    d[: n // 8] = np.eye(3)[rng.integers(0, 3, n // 8)]
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = 2.8 * (1 + rng.choice([0, 1, -1], n // 2) * 10.0 ** rng.uniform(-16, -6, n // 2))
    same(boxed(n, box), np.concatenate([a, a + d * r[:, None]]))
