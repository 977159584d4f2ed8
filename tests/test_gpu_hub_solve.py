"""The solve of substeps with many colours, against the oracle bit for bit: a slab on the ground under a layer of single
bricks, with chunks of 1, 16 and 32 contacts (the last has more rows of places than are kept in shared memory), alone and on a
cluster, with and without a warm start."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT, IT = 1.0 / 60.0, 3


def laden_slab(w, every=1):
    """A slab of w x w bricks on the ground and a single brick on every `every`-th of its bricks."""
    a = S.body_blocks(1, w, w, 1)
    k = np.arange(0, w * w, every)
    n = len(k)
    f, x, m, p = S.loose_debris(n, 1)
    p[:, 0:3] = np.stack([0.5 * (k % w), np.full(n, 0.52), 0.5 * (k // w)], 1)
    return S.Scene(a.static_xyz, a.static_mat, a.static_sid, a.static_infill,
                   np.concatenate([a.body_first, a.body_first[-1] + f[1:]]).astype(np.uint32),
                   np.concatenate([a.body_brick_xyz, x]), np.concatenate([a.body_brick_mat, m]),
                   np.concatenate([a.body_pose, p])).contiguous()


@pytest.mark.parametrize("w,chunk,warm,colours", [(8, 1, 0, 320), (8, 1, 1, 320), (8, 16, 0, 80), (8, 32, 1, 72), (16, 16, 0, 320),
                                                  (26, 16, 0, 845), (26, 16, 1, 845), (26, 32, 0, 761), (26, 32, 1, 761)])
def test_many_colours_equal_oracle(sf, oracle, w, chunk, warm, colours):
    sc = laden_slab(w)
    g = sf.World(sc, iterations=IT, max_colors=1024, manifold_chunk=chunk, warm_start=warm)
    ow = oracle.OracleWorld(sc)
    most = 0
    for _ in range(3):
        st = g.step(DT)
        most = max(most, st.colors)
        assert st.contacts <= 8192
        ow.step(DT, iterations=IT, order=oracle.ORDER_COLOR, warm=warm, chunk=chunk)
        for x, y in zip(g.bodies(), ow.bodies()):
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(g.manifolds(0), ow.manifolds())
    assert most >= colours
    g.close()


@pytest.mark.parametrize("warm", [0, 1])
def test_a_large_substep_of_many_colours_equals_oracle(sf, oracle, warm):
    """8,464 contacts of the slab with the ground and some of its bricks' with single ones: warps of k_solve with and without
    second bodies."""
    sc = laden_slab(46, 13)
    g = sf.World(sc, iterations=IT, max_colors=1024, warm_start=warm)
    ow = oracle.OracleWorld(sc)
    most = 0
    for _ in range(2):
        most = max(most, g.step(DT).contacts)
        ow.step(DT, iterations=IT, order=oracle.ORDER_COLOR, warm=warm)
        for x, y in zip(g.bodies(), ow.bodies()):
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(g.manifolds(0), ow.manifolds())
    assert most > 8192
    g.close()


def solve_ms_a_contact(sf, wx, wz, h):
    w = sf.World(S.body_blocks(1, wx, wz, h), iterations=8, max_colors=256)
    for _ in range(2):
        w.step(DT)
    w.set_profiling(True)
    w.reset_profile()
    for _ in range(3):
        w.step(DT)
    p = w.profile()
    w.close()
    return p["ms"]["solve"] / p["contacts_sum"]


def test_a_contact_of_many_colours_takes_what_one_of_few_does(sf):
    """Chunks of one body, one after another: 157 colours against 36."""
    assert solve_ms_a_contact(sf, 25, 25, 4) < 1.15 * solve_ms_a_contact(sf, 12, 12, 3)
