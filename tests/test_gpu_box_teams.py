"""The box world's teams at their edges, against the oracle bit for bit: one box, sizes around a warp, a block and the
largest one-block scene, worlds of more scenes than SMs (two blocks of 256 threads an SM) and of fewer (one of 512).
"""
import numpy as np
import pytest

from shatterforge_b200 import boxes as X

pytestmark = pytest.mark.gpu

DT = np.float32(1.0 / 60.0)


def check(oracle, scenes, params, steps):
    w = X.BoxWorld(scenes, params)
    ows = [oracle.OracleBoxWorld(s, params, oracle.ORDER_COLOR) for s in scenes]
    for _ in range(steps):
        w.step(DT)
    for i, ow in enumerate(ows):
        for _ in range(steps):
            ow.step(DT)
        st = w.stats(i)
        assert st.status == 0
        assert (st.awake, st.pairs, st.manifolds, st.points, st.colours) == ow.stats(), i
        np.testing.assert_array_equal(w.state(i), ow.state())
        np.testing.assert_array_equal(w.manifolds(i), ow.manifolds())


@pytest.mark.parametrize("sizes", [
    [1], [33, 1, 32, 31], [255, 256, 257], [511, 512, 513], [1023, 1025], [4096, 40], [4097, 255],
    [20 + k % 23 for k in range(170)], [300 + k % 7 for k in range(150)],
], ids=lambda s: f"{len(s)}x{max(s)}")
def test_scene_sizes(sf, oracle, sizes):
    steps = 6 if max(sizes) > 2000 else 12 if len(sizes) > 100 else 30
    check(oracle, [X.pile(n) for n in sizes], X.box_params(allow_sleep=0, substeps=4), steps)


@pytest.mark.parametrize("sizes", [[1024], [1025], [1025] * 7, [1025] * 9, [1025, 4097], [1024, 4097]],
                         ids=lambda s: "-".join(map(str, s)))
def test_scenes_on_clusters_side_by_side(sf, oracle, sizes):
    """Middling scenes take a cluster each where the whole world fits as clusters, else a block each."""
    check(oracle, [X.pile(n) for n in sizes], X.box_params(allow_sleep=0, substeps=4), 8)


@pytest.mark.parametrize("under", [30, 34, 400, 1100])
def test_pairs_of_one_body(sf, oracle, under):
    """A static slab under `under` boxes: its list of pairs is sorted by its thread (up to 32), by the team, or (past the
    980 that one walk keeps) walked for again."""
    side = int(np.ceil(np.sqrt(under)))
    k = np.arange(under)
    recs = np.zeros((under + 1, 11), np.float32)
    half = np.float32(0.14 * side)
    recs[0] = [0, 0.5, 0, 0, 0, 0, 1, half, 0.5, half, 0.0]
    recs[1:, 0] = (k % side - 0.5 * (side - 1)) * 0.28
    recs[1:, 1] = 1.13
    recs[1:, 2] = (k // side - 0.5 * (side - 1)) * 0.28
    recs[1:, 6] = 1
    recs[1:, 7:10] = 0.125
    recs[1:, 10] = 1.0
    recs[1:, :3] += np.random.default_rng(under).uniform(-0.004, 0.004, (under, 3)).astype(np.float32)
    check(oracle, [recs, X.pile(40)], X.box_params(substeps=4), 20)


@pytest.mark.parametrize("under", [1, 63, 70, 140])
def test_colours_of_one_body(sf, oracle, under):
    """A moving plate on `under` boxes: as many colours as it has manifolds, in one or two mask words, and past the 128
    that there are the step is refused and the scene left as it was, while the other scene steps as its oracle."""
    side = int(np.ceil(np.sqrt(under)))
    k = np.arange(under)
    recs = np.zeros((under + 1, 11), np.float32)
    half = np.float32(0.14 * side)
    recs[:under, 0] = (k % side - 0.5 * (side - 1)) * 0.28
    recs[:under, 1] = 0.125
    recs[:under, 2] = (k // side - 0.5 * (side - 1)) * 0.28
    recs[:under, 7:10] = 0.125
    recs[under, 1] = 0.255
    recs[under, :3] += [0, 0.1, 0]
    recs[under, 7:10] = [half, 0.1, half]
    recs[:, 6] = 1
    recs[:, 10] = 1.0
    other = X.pile(40)
    p = X.box_params(allow_sleep=0, substeps=4)
    if under <= 128:
        check(oracle, [recs, other], p, 20)
        return
    w = X.BoxWorld([recs, other], p)
    before = w.state(0).copy()
    ow = oracle.OracleBoxWorld(other, p, oracle.ORDER_COLOR)
    for _ in range(3):
        with pytest.raises(sf.SfError) as e:
            w.step(DT)
        assert e.value.status == sf.SF_ERR_CAPACITY
        ow.step(DT)
    assert w.stats(0).status == 8
    np.testing.assert_array_equal(w.state(0), before)
    np.testing.assert_array_equal(w.state(1), ow.state())


def test_state_words(sf, oracle):
    """The 22 floats of a box, for boxes asleep and awake, against the oracle's records; the state of a world that has not
    stepped is its records."""
    recs = X.pile(100)
    w = X.BoxWorld([recs, X.stack(20)], X.box_params())
    s = w.state(0)
    np.testing.assert_array_equal(s[:, :7], recs[:, :7])
    np.testing.assert_array_equal(s[:, 7:14], np.zeros((100, 7), np.float32))
    ow = oracle.OracleBoxWorld(X.stack(20), X.box_params(), oracle.ORDER_COLOR)
    for _ in range(90):
        w.step(DT)
        ow.step(DT)
        np.testing.assert_array_equal(w.state(1), ow.state())
    assert w.state(1)[:, 21].sum() in (0, 20) and w.state(1)[:, 13].max() >= 0.5
