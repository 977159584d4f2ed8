"""Colouring of small substeps with many manifolds at one body, against the oracle bit for bit: bodies of 32 to 34 manifolds (up
to 32 their colours are read from their list, above that kept as a mask), of a few hundred, hubs in a pile with the masks in
shared memory and in memory (3,152 manifolds and more at 1,024 colours), and several hubs of different scenes at once."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT, IT = 1.0 / 60.0, 2


def loose(n, seed, lo, hi):
    f, x, m, p = S.loose_debris(n, seed, box_lo=lo, box_hi=hi)
    return S.Scene(body_first=f, body_brick_xyz=x, body_brick_mat=m, body_pose=p).contiguous()


def merged(a, b):
    return S.Scene(a.static_xyz, a.static_mat, a.static_sid, a.static_infill,
                   np.concatenate([a.body_first, a.body_first[-1] + b.body_first[1:]]).astype(np.uint32),
                   np.concatenate([a.body_brick_xyz, b.body_brick_xyz]), np.concatenate([a.body_brick_mat, b.body_brick_mat]),
                   np.concatenate([a.body_pose, b.body_pose])).contiguous()


def slab(wx, wz):
    return S.body_blocks(1, wx, wz, 1)                 # wx * wz / 4 manifolds of 16 contacts with the ground


CASES = {                                              # scenes, max_colors, steps, least manifolds at the last step
    "32": (lambda: [slab(16, 8)], 256, 3, 32),
    "33": (lambda: [slab(12, 11)], 256, 3, 33),
    "34": (lambda: [slab(17, 8)], 256, 3, 34),
    "512": (lambda: [slab(64, 32)], 1024, 2, 512),
    "three hubs": (lambda: [slab(20, 12), slab(4, 4), slab(40, 8)], 128, 3, 144),
    "hub under a pile": (lambda: [merged(slab(12, 12), loose(500, 8, (-1.0, 2.0, -1.0), (6.0, 5.0, 6.0)))], 256, 25, 100),
    "masks in memory": (lambda: [merged(slab(20, 20), loose(3200, 3, (0.0, 1.2, 0.0), (11.0, 5.0, 11.0)))], 1024, 12, 3152),
    "the same, fewer colours": (lambda: [merged(slab(20, 20), loose(3200, 3, (0.0, 1.2, 0.0), (11.0, 5.0, 11.0)))], 256, 12, 3152),
}


@pytest.mark.parametrize("name", list(CASES))
def test_hub_colours_equal_oracle(sf, oracle, name):
    make, colors, steps, least = CASES[name]
    scenes = make()
    w = sf.World(scenes, iterations=IT, max_colors=colors, verify=1)
    ows = [oracle.OracleWorld(s) for s in scenes]
    for _ in range(steps):
        st = w.step(DT)
        assert st.contacts <= 8192
        for ow in ows:
            ow.step(DT, iterations=IT, order=oracle.ORDER_COLOR)
    assert st.manifolds >= least
    body = w.bodies()
    for k, ow in enumerate(ows):
        a, b = int(w.body_off[k]), int(w.body_off[k + 1])
        for x, y in zip(body, ow.bodies()):
            np.testing.assert_array_equal(x[a:b], y)
        np.testing.assert_array_equal(w.manifolds(k), ow.manifolds())
    w.close()


def test_a_hub_colours_in_a_fraction_of_its_solve(sf):
    """450 manifolds at one body, each a colour of its own: the colouring's rounds cost less than a tenth of the solve's."""
    w = sf.World(S.body_blocks(1, 60, 30, 2), iterations=8, max_colors=512)
    w.step(DT)
    w.set_profiling(True)
    w.reset_profile()
    assert w.step(DT).colors == 450
    ms = w.profile()["ms"]
    assert ms["colour"] < 0.1 * ms["solve"], ms
    w.close()
