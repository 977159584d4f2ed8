"""Worlds of many bodies with few contacts, against the oracle bit for bit: up to 65,536 bodies the solve of small substeps keeps
all velocities in shared memory, above that it reads them in memory, alone or on a cluster; with contact reduction and a large
body among more bodies than the one-block build counts in shared memory. Such steps take as many launches as those of a small
world."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT, IT = 1.0 / 60.0, 4


def loose(n, seed, lo, hi):
    f, x, m, p = S.loose_debris(n, seed, box_lo=lo, box_hi=hi)
    return S.Scene(body_first=f, body_brick_xyz=x, body_brick_mat=m, body_pose=p).contiguous()


def merged(a, b):
    return S.Scene(a.static_xyz, a.static_mat, a.static_sid, a.static_infill,
                   np.concatenate([a.body_first, a.body_first[-1] + b.body_first[1:]]).astype(np.uint32),
                   np.concatenate([a.body_brick_xyz, b.body_brick_xyz]), np.concatenate([a.body_brick_mat, b.body_brick_mat]),
                   np.concatenate([a.body_pose, b.body_pose])).contiguous()


def world(bodies, pile, slab):
    """`pile` bricks in a heap, on a slab of slab x slab bricks if any, the other bodies high above them and far apart."""
    sc = loose(pile, 4, (0.0, 0.3 + (slab > 0), 0.0), (1.5 + pile ** 0.5 / 6, 4.0, 1.5 + pile ** 0.5 / 6))
    if slab:
        sc = merged(S.body_blocks(1, slab, slab, 1), sc)
    k = bodies - sc.n_bodies
    return merged(loose(k // 2, 6, (60.0, 200.0, -500.0), (500.0, 400.0, 500.0)),
                  merged(sc, loose(k - k // 2, 7, (-500.0, 200.0, -500.0), (-60.0, 400.0, 500.0))))


@pytest.mark.parametrize("bodies,pile,slab,reduce,warm", [(65536, 300, 0, 0, 0), (65537, 300, 0, 0, 0), (70001, 300, 0, 0, 1),
                                                          (70000, 2500, 0, 0, 0), (70000, 700, 12, 0, 0), (70000, 700, 30, 1, 1),
                                                          (9000, 700, 30, 1, 0), (131073, 900, 0, 0, 0)])
def test_few_contacts_equal_oracle(sf, oracle, bodies, pile, slab, reduce, warm):
    sc = world(bodies, pile, slab)
    assert sc.n_bodies == bodies
    w = sf.World(sc, iterations=IT, max_colors=256, reduce=reduce, warm_start=warm)
    ow = oracle.OracleWorld(sc)
    for _ in range(4):
        st = w.step(DT)
        assert 50 < st.contacts <= 8192
        ow.step(DT, iterations=IT, order=oracle.ORDER_COLOR, reduce=reduce, warm=warm)
    for x, y in zip(w.bodies(), ow.bodies()):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(w.manifolds(0), ow.manifolds())
    w.close()


def test_launches_do_not_grow_with_the_bodies(sf):
    counts = []
    for bodies in (5000, 60000, 80000):
        w = sf.World(world(bodies, 300, 0), iterations=IT)
        for _ in range(3):
            w.step(DT)
        before = w.stats().launches
        w.step(DT)
        counts.append(w.stats().launches - before)
        w.close()
    assert max(counts) - min(counts) <= 8, counts      # (the scans of more bricks take a level more)
