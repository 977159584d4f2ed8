"""The profile's contact-iterations are those of the contacts that the solve takes, with and without a contact reduction, of small
substeps and large ones."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu
DT, IT = 1.0 / 60.0, 4


@pytest.mark.parametrize("reduce", [0, 1])
@pytest.mark.parametrize("wx,wz", [(12, 12), (30, 40), (60, 60)])
def test_contact_iterations_are_the_solved_ones(sf, wx, wz, reduce):
    """A slab on the ground, at rest: four contacts a brick, of which a reduction keeps at most 27."""
    w = sf.World(S.body_blocks(1, wx, wz, 1), iterations=IT, max_colors=1024, reduce=reduce)
    w.step(DT)
    w.set_profiling(True)
    w.reset_profile()
    w.step(DT, 2)
    p = w.profile()
    manifolds = w.manifolds(0)
    assert p["substeps"] == 4 and p["contacts_sum"] == 4 * 4 * wx * wz
    solved = p["solve_contact_iters"] / IT
    if reduce:
        assert 4 * 4 <= solved <= 4 * 27
        assert len(manifolds) <= 2
    else:
        assert solved == p["contacts_sum"]
    w.reset_profile()
    assert w.profile()["solve_contact_iters"] == 0
    w.close()
