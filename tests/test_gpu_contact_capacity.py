"""Worlds with more contacts than bricks, against the oracle bit for bit: with a fixed contact capacity, whose steps then
allocate nothing, and with one that grows in the step; the manifolds' records in the room of the contact slots (up to six
manifolds a brick of capacity) and in their own; the one-block build and the large form of it."""
import numpy as np
import pytest
import torch

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT, IT = 1.0 / 60.0, 4


def loose(n, seed, lo, hi):
    f, x, m, p = S.loose_debris(n, seed, box_lo=lo, box_hi=hi)
    return S.Scene(body_first=f, body_brick_xyz=x, body_brick_mat=m, body_pose=p).contiguous()


def crowds(k, n, seed):
    """k crowds of n bricks that all touch one another."""
    sc = loose(k * n, seed, (0.0, 5.0, 0.0), (0.3, 5.3, 0.3))
    sc.body_pose[:, 0] += 4.0 * (np.arange(k * n) // n).astype(np.float32)
    return sc


SCENES = {
    "crowd": lambda: crowds(1, 60, 2),                                        # 29 contacts a brick, one block
    "crowds": lambda: crowds(40, 100, 3),                                     # 49 contacts a brick
    "dense_small": lambda: loose(1500, 4, (0.0, 0.3, 0.0), (7.0, 4.0, 7.0)),  # some 2.7 contacts a brick, one cluster
    "dense": lambda: loose(6000, 5, (0.0, 0.3, 0.0), (14.0, 4.0, 14.0)),
}


@pytest.mark.parametrize("name,per_brick", [("crowd", 64), ("crowd", 0), ("crowds", 64), ("crowds", 0), ("dense_small", 4),
                                            ("dense", 4), ("dense", 5), ("dense", 0)])
def test_more_contacts_than_bricks(sf, oracle, name, per_brick):
    sc = SCENES[name]()
    n = sc.n_body_bricks
    make = lambda: sf.World(sc, iterations=IT, max_colors=256, contact_capacity=per_brick * n)
    first = make()                        # (the kernels' code is loaded with their first launch)
    for _ in range(3):
        first.step(DT)
    w, ow = make(), oracle.OracleWorld(sc)
    most = 0
    for _ in range(3):
        free = torch.cuda.mem_get_info()[0]   # (before the step: reading the bodies stages them)
        most = max(most, w.step(DT).contacts)
        if per_brick:
            assert torch.cuda.mem_get_info()[0] == free
        ow.step(DT, iterations=IT, order=oracle.ORDER_COLOR)
        for x, y in zip(w.bodies(), ow.bodies()):
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(w.manifolds(0), ow.manifolds())
    assert most > n
    w.close()
    first.close()
