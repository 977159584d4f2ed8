"""The rule between the two forms of contact generation, and its table form at the sizes that take it: scenes stepped together
against each scene alone (which takes the other form), bit for bit, all awake and with most bodies asleep, when the list of
awake bricks has its own places for the scenes: some awake whole, some but for one body asleep."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def table(n, k):
    """The rule (gen_table of sf_step.cu)."""
    return n * n >= 12500000000 * k or (n >= 1250000 and n >= 4096 * k)


@pytest.mark.parametrize("asleep", [False, True])
def test_table_form_equals_scenes_alone(sf, asleep):
    lib = S.ClusterLibrary(11)
    scenes = [S.debris_scene(n, 100 + n, lib=lib, spacing=1.6) for n in (32000, 29000, 31000, 30000, 31500, 28000)]
    bricks = [s.n_body_bricks for s in scenes]
    assert not any(table(n, 1) for n in bricks)
    both = sf.World(scenes, iterations=4)
    alone = [sf.World(s, iterations=4) for s in scenes]
    both.step(DT, 20)
    if asleep:
        st, sl, fl = both.bodies()
        fl = fl.copy()
        for i in (0, 2, 5):                               # all asleep but for a body in the middle, the first, the last
            a, b = int(both.body_off[i]), int(both.body_off[i + 1])
            fl[a:b] |= 2
            fl[{0: (a + b) // 2, 2: a, 5: b - 1}[i]] &= 253
        both.set_bodies(st, sl, fl)
    for i, w in enumerate(alone):
        w.step(DT, 20)
        a, b = int(both.body_off[i]), int(both.body_off[i + 1])
        if asleep:
            w.set_bodies(st[a:b], sl[a:b], fl[a:b])
    for k, steps in enumerate((1, 1, 4, 10)):             # (the sparse form is chosen from the last step's count of awake bodies)
        both.step(DT, steps)
        st, sl, fl = both.bodies()
        awake = (fl & 3) == 1
        if asleep:
            assert awake.sum() * 2 <= len(fl)
        per_body = np.concatenate([np.diff(s.body_first) for s in scenes])
        assert table(int(per_body[awake].sum()), len(scenes))
        for i, w in enumerate(alone):
            w.step(DT, steps)
            a, b = int(both.body_off[i]), int(both.body_off[i + 1])
            x = w.bodies()
            assert np.array_equal(x[0], st[a:b]) and np.array_equal(x[1], sl[a:b]) and np.array_equal(x[2], fl[a:b]), (k, i)
            for u, v in zip(w.contacts(0), both.contacts(i)):
                assert np.array_equal(u, v), (k, i)
    for w in [both, *alone]:
        w.close()


def gen_us(sf, n_scenes):
    lib = S.ClusterLibrary(11)
    w = sf.World([S.debris_scene(150, 100 + q, lib=lib, spacing=2.5) for q in range(n_scenes)], iterations=2)
    for _ in range(20):
        w.step(DT)
    w.set_profiling(True)
    w.reset_profile()
    for _ in range(10):
        w.step(DT)
    p = w.profile()
    w.close()
    return 1e3 * p["gen_ms"] / p["substeps"], p["gen_bricks"] // p["substeps"]


def test_small_scenes_take_no_longer_for_being_many(sf):
    """150 scenes of 500 bricks against 120 of them."""
    (few, a), (many, b) = gen_us(sf, 120), gen_us(sf, 150)
    assert a < 65536 < b and many < 1.8 * few, (few, many)
