"""The one-cluster-per-structure solve against the grid kernel, bit for bit: potentials, sweep counts and residuals, at
sizes that reach every form of the cluster kernel, with bricks removed (cells that no longer update, halo cells without
links) and with the sweep limit or the tolerance ending the solve."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu


def building(wx, wz, storeys, spacing=6, seed=0, mats=(S.CONC, S.MASON, S.STEEL, S.WOOD)):
    xs = sorted(set(range(0, wx, spacing)) | {wx - 1})
    zs = sorted(set(range(0, wz, spacing)) | {wz - 1})
    rng = np.random.default_rng(seed)
    x, m, s, i = S.frame_structure(300, 300, wx, wz, storeys, 7, xs, zs, 0,
                                   lambda c: np.array(mats, np.uint8)[rng.integers(0, len(mats), len(c))])
    return S.Scene(x, m, s, i).contiguous()


@pytest.mark.parametrize("wx,wz,storeys", [(1, 1, 1), (2, 3, 1), (24, 24, 5), (24, 24, 6), (31, 29, 8), (40, 40, 9), (48, 47, 8),
                                           (60, 60, 5), (60, 60, 7), (55, 57, 12), (60, 60, 13)])
def test_cluster_solve_equals_grid_kernel(sf, wx, wz, storeys):
    sc = building(wx, wz, storeys, seed=wx + storeys)
    rng = np.random.default_rng(wx)
    a, b = (sf.World(sc, sor_cluster=c, detach_bodies=4, detach_bricks=16) for c in (1, 0))
    ext = rng.uniform(0, 200, sc.n_static).astype(np.float32)
    for sweeps, tol, cut in ((1, 0.0, 0), (2, 0.0, 200), (3, 0.0, 20), (64, 0.0, 4), (400, 1e-3, 0)):
        got = []
        for w in (a, b):
            w.set_phi(np.zeros(sc.n_static, np.float32))
            w.set_ext(ext)
            w.structure_solve(-1, 1.7, tol, sweeps)
            got.append((w.phi64(), *w.solve_detail()))
        for x, y in zip(*got):
            assert np.array_equal(x, y), (sweeps, tol)
        if cut:
            gone = rng.choice(sc.n_static, max(1, sc.n_static // cut), replace=False)
            gone = gone[sc.static_xyz[gone, 1] > 0]
            for w in (a, b):
                w.remove_bricks(gone)
    assert a.stats().cluster_solves == 5 and b.stats().cluster_solves == 0
    a.close()
    b.close()


def test_cluster_solve_with_bricks_no_solve_updates(sf):
    """Bricks of the materials a solve leaves out (6 and above) inside a structure: their links are read, they keep their
    potentials."""
    sc = building(30, 30, 9, seed=5)
    sc.static_mat[np.random.default_rng(2).choice(sc.n_static, sc.n_static // 30, replace=False)] = 6
    got = []
    for c in (1, 0):
        w = sf.World(sc, sor_cluster=c)
        w.structure_solve(-1, 1.7, 0.0, 150)
        got.append((w.phi64(), *w.solve_detail()))
        w.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y)
