"""Substeps of few contacts (at most 8,192) against the oracle, bit for bit: one block or one cluster, contacts and bodies in
shared memory or not, few colours or more than the kernels keep tables for, with and without a warm start."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT, IT = 1.0 / 60.0, 8


def merged(a, b, dx):
    """Scene a with scene b's bodies moved dx metres along x."""
    pose = b.body_pose.copy()
    pose[:, 0] += dx
    return S.Scene(a.static_xyz, a.static_mat, a.static_sid, a.static_infill,
                   np.concatenate([a.body_first, a.body_first[-1] + b.body_first[1:]]).astype(np.uint32),
                   np.concatenate([a.body_brick_xyz, b.body_brick_xyz]), np.concatenate([a.body_brick_mat, b.body_brick_mat]),
                   np.concatenate([a.body_pose, pose])).contiguous()


def loose(n, seed, lo, hi):
    f, x, m, p = S.loose_debris(n, seed, box_lo=lo, box_hi=hi)
    return S.Scene(body_first=f, body_brick_xyz=x, body_brick_mat=m, body_pose=p).contiguous()


SCENES = {
    "one_body": lambda: S.body_blocks(1, 2, 2, 1),
    "pile_alone": lambda: loose(300, 3, (0.0, 0.3, 0.0), (4.0, 4.0, 4.0)),
    "pile_cluster": lambda: loose(1500, 4, (0.0, 0.3, 0.0), (7.0, 4.0, 7.0)),
    "compound": lambda: S.debris_scene(900, seed=6, obstacles=(2, 4), spacing=1.0, p_geom=0.15, kmax=40),
    "hub_157_colours": lambda: S.body_blocks(1, 25, 25, 4),
    "hub_beside_many": lambda: merged(S.body_blocks(1, 20, 20, 3), loose(40000, 5, (40.0, 30.0, -60.0), (120.0, 90.0, 60.0)), 0.0),
    "hub_and_pile": lambda: merged(S.body_blocks(1, 12, 12, 3), loose(700, 8, (-1.0, 2.0, -1.0), (6.0, 5.0, 6.0)), 0.0),
}


@pytest.mark.parametrize("name,steps,warm", [("one_body", 30, 0), ("pile_alone", 25, 0), ("pile_alone", 25, 1), ("pile_cluster", 20, 0),
                                             ("pile_cluster", 12, 1), ("compound", 45, 0), ("hub_157_colours", 6, 0),
                                             ("hub_157_colours", 4, 1), ("hub_beside_many", 3, 0), ("hub_and_pile", 30, 0)])
def test_small_substeps_equal_oracle(sf, oracle, name, steps, warm):
    sc = SCENES[name]()
    w = sf.World(sc, iterations=IT, warm_start=warm, max_colors=256)
    ow = oracle.OracleWorld(sc)
    most = 0
    for k in range(steps):
        st = w.step(DT)
        most = max(most, st.contacts)
        ow.step(DT, iterations=IT, order=oracle.ORDER_COLOR, warm=warm)
        if k % 4 and k + 1 < steps:
            continue
        for x, y in zip(w.bodies(), ow.bodies()):
            np.testing.assert_array_equal(x, y)
        for x, y in zip(w.contacts(0), ow.contacts()):
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(w.manifolds(0), ow.manifolds())
    assert 0 < most <= 8192
    w.close()
