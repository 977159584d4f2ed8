"""Boxes whose grid spans are out of the ordinary beside a pile, on a block and on a cluster: negative half extents (such a box
covers no cell but counts for entries when two of them are negative) and a centre past the range of the cells' integers."""
import numpy as np
import pytest

from shatterforge_b200 import boxes as X

pytestmark = pytest.mark.gpu

DT = np.float32(1.0 / 60.0)
STEPS = 8


def beside(n, centre, half, times):
    """pile(n) and `times` boxes of these half extents, the first at `centre`, 40 m apart in y."""
    odd = np.zeros((times, 11), np.float32)
    odd[:, :3] = centre
    odd[:, 1] += 40.0 * np.arange(times)
    odd[:, 6] = 1.0
    odd[:, 7:10] = half
    odd[:, 10] = 1.0
    return np.concatenate([X.pile(n), odd])


@pytest.mark.parametrize("n", [60, 1100])
@pytest.mark.parametrize("half", [(-3, -3, 0.2), (0.2, -3, -2), (-2.5, 0.3, -4)])
def test_two_negative_extents_equal_oracle(sf, oracle, n, half):
    recs = beside(n, (1.0, 60.0, 1.0), half, 9)
    p = X.box_params(allow_sleep=0, substeps=4)
    w, ow = X.BoxWorld(recs, p), oracle.OracleBoxWorld(recs, p, oracle.ORDER_COLOR)
    for k in range(STEPS):
        w.step(DT)
        ow.step(DT)
        st = w.stats()
        assert (st.awake, st.pairs, st.manifolds, st.points, st.colours) == ow.stats(), k
    np.testing.assert_array_equal(w.state(), ow.state())
    np.testing.assert_array_equal(w.manifolds(), ow.manifolds())
    w.close()


def test_one_negative_extent_stays_refused(sf):
    recs = beside(40, (1.0, 60.0, 1.0), (-3, 0.2, 0.2), 1)
    w = X.BoxWorld(recs, X.box_params(allow_sleep=0, substeps=4))
    before = w.state()
    with pytest.raises(sf.SfError) as e:
        w.step(DT)
    assert e.value.status == sf.SF_ERR_CAPACITY and w.stats().status == 1
    np.testing.assert_array_equal(w.state(), before)
    w.close()


@pytest.mark.parametrize("n", [60, 1100])
@pytest.mark.parametrize("centre", [(3e9, 60.0, 1.0), (1.0, 60.0, -4e9), (5e9, 60.0, 5e9)])
def test_far_box_leaves_the_pile_as_it_is(sf, oracle, n, centre):
    """The pile's boxes come first, so their pairs, priorities and colours are those of the pile alone."""
    p = X.box_params(allow_sleep=0, substeps=4)
    w, ow = X.BoxWorld(beside(n, centre, 0.2, 1), p), oracle.OracleBoxWorld(X.pile(n), p, oracle.ORDER_COLOR)
    for _ in range(STEPS):
        w.step(DT)
        ow.step(DT)
    np.testing.assert_array_equal(w.state()[:n], ow.state())
    np.testing.assert_array_equal(w.manifolds(), ow.manifolds())
    w.close()


def test_box_over_the_whole_range_is_refused(sf):
    """A box that covers more cells along one axis than an int counts."""
    recs = beside(40, (1.0, 60.0, 1.0), (4e9, 0.2, 0.2), 1)
    recs[-1, 10] = 0.0
    w = X.BoxWorld(recs, X.box_params(allow_sleep=0, substeps=4))
    with pytest.raises(sf.SfError) as e:
        w.step(DT)
    assert e.value.status == sf.SF_ERR_CAPACITY
    w.close()
