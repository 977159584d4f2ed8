"""Contact generation from bucket tables in shared memory (worlds of many bricks) against the form that small worlds take:
scenes stepped together equal each scene stepped alone, bit for bit, while they fall, pile up, and with most bodies asleep
(then only the buckets around awake bricks are hashed)."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


@pytest.mark.parametrize("asleep", [0.0, 0.3, 0.9])
def test_table_form_equals_small_worlds(sf, asleep):
    lib = S.ClusterLibrary(11)
    scenes = [S.debris_scene(n, 100 + n, lib=lib, spacing=1.6) for n in (11000, 40, 9000, 1, 7000)]
    assert sum(s.n_body_bricks for s in scenes) > 70000 and max(s.n_body_bricks for s in scenes) < 65536
    both = sf.World(scenes, iterations=8)
    alone = [sf.World(s, iterations=8) for s in scenes]
    rng = np.random.default_rng(3)
    for k, steps in enumerate((3, 30, 25, 10, 2)):
        if k == 3 and asleep:
            st, sl, fl = both.bodies()
            fl = fl.copy()
            fl[rng.random(len(fl)) < asleep] |= 2
            both.set_bodies(st, sl, fl)
            for i, w in enumerate(alone):
                a, b = int(both.body_off[i]), int(both.body_off[i + 1])
                w.set_bodies(st[a:b], sl[a:b], fl[a:b])
            both.step(DT, 1)                       # (the form by the awake bodies is chosen from the last step's count)
            for w in alone:
                w.step(DT, 1)
        both.step(DT, steps)
        st, sl, fl = both.bodies()
        for i, w in enumerate(alone):
            w.step(DT, steps)
            a, b = int(both.body_off[i]), int(both.body_off[i + 1])
            x = w.bodies()
            assert np.array_equal(x[0], st[a:b]) and np.array_equal(x[1], sl[a:b]) and np.array_equal(x[2], fl[a:b]), (k, i)
            for u, v in zip(w.contacts(0), both.contacts(i)):
                assert np.array_equal(u, v), (k, i)
    for w in [both, *alone]:
        w.close()
