"""The one-cluster-per-structure solve on solid and thick structures, whose layers are larger than a block's range of cells,
and on lattices with most cells of one parity, against the grid kernel bit for bit: they stay on the cluster path, and so
does a building solved beside them."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu


def solid(a, b, c, at=(100, 0, 100)):
    return np.stack(np.meshgrid(np.arange(a), np.arange(b), np.arange(c), indexing="ij"), -1).reshape(-1, 3) + np.array(at)


def trellis(a, b, c):
    """Every second line along each axis: three cells in four are of one parity."""
    p = solid(a, b, c, (0, 0, 0))
    return p[((p % 2) != 0).sum(1) <= 1] + np.array([100, 0, 100])


def plates():
    """Three thick plates at right angles: in any order of layers one of them has layers larger than a block's range."""
    return np.unique(np.concatenate([solid(92, 3, 92, (100, 40, 100)), solid(3, 90, 70, (140, 0, 100)), solid(70, 90, 3, (100, 0, 140))]), axis=0)


SHAPES = {
    "60x12x60": lambda: solid(60, 12, 60),
    "120x3x120": lambda: solid(120, 3, 120, (101, 0, 103)),
    "80x8x80": lambda: solid(80, 8, 80, (99, 0, 98)),
    "125x4x125": lambda: solid(125, 4, 125, (99, 3, 97)),
    "180x2x180": lambda: solid(180, 2, 180, (100, 0, 101)),
    "640x3x10": lambda: solid(640, 3, 10, (0, 0, 101)),
    "40x40x40": lambda: solid(40, 40, 40),
    "trellis": lambda: trellis(50, 50, 52),
    "plates": plates,
}


def scene(parts, seed=0):
    """Structure k is parts[k], of mixed materials."""
    rng = np.random.default_rng(seed)
    xyz = np.concatenate(parts).astype(np.int32)
    mat = np.array([S.CONC, S.MASON, S.STEEL, S.WOOD], np.uint8)[rng.integers(0, 4, len(xyz))]
    sid = np.concatenate([np.full(len(p), k, np.int32) for k, p in enumerate(parts)])
    return S.Scene(xyz, mat, sid, np.zeros(len(xyz), np.uint8)).contiguous()


def compare(sf, sc, runs, cut):
    rng = np.random.default_rng(1)
    a, b = (sf.World(sc, sor_cluster=c, detach_bodies=4, detach_bricks=16) for c in (1, 0))
    ext = rng.uniform(0, 200, sc.n_static).astype(np.float32)
    for sweeps, tol in runs:
        got = []
        for w in (a, b):
            w.set_phi(np.zeros(sc.n_static, np.float32))
            w.set_ext(ext)
            w.structure_solve(-1, 1.7, tol, sweeps)
            got.append((w.phi64(), *w.solve_detail()))
        for x, y in zip(*got):
            assert np.array_equal(x, y), (sweeps, tol)
        gone = rng.choice(sc.n_static, sc.n_static // cut, replace=False)
        for w in (a, b):
            w.remove_bricks(gone)
    assert a.stats().cluster_solves == len(runs) and b.stats().cluster_solves == 0
    a.close()
    b.close()


@pytest.mark.parametrize("name", list(SHAPES))
def test_solid_structures_equal_grid_kernel(sf, name):
    compare(sf, scene([SHAPES[name]()], len(name)), ((1, 0.0), (40, 0.0), (300, 1e-3)), 50)


def test_building_beside_a_solid_podium(sf):
    x, _, _, _ = S.frame_structure(300, 300, 31, 29, 8, 7, list(range(0, 31, 6)), list(range(0, 29, 7)), 0,
                                   lambda c: np.full(len(c), S.CONC, np.uint8))
    compare(sf, scene([SHAPES["60x12x60"](), x], 3), ((2, 0.0), (120, 0.0)), 200)


def test_more_bricks_than_a_cluster_takes(sf):
    """65,535 bricks take the grid kernel, and with them what is solved in the same call."""
    big = solid(255, 1, 257)
    assert len(big) == 65535
    sc = scene([big, solid(4, 4, 4, (400, 0, 400))])
    got = []
    for c in (1, 0):
        w = sf.World(sc, sor_cluster=c)
        w.structure_solve(-1, 1.7, 0.0, 20)
        got.append((w.phi64(), *w.solve_detail()))
        assert w.stats().cluster_solves == 0
        w.structure_solve(1, 1.7, 0.0, 20)
        assert w.stats().cluster_solves == c
        w.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y)
