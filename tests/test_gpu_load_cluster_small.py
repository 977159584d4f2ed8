"""Many small structures at once on the cluster path, several clusters an SM, against the grid kernel bit for bit: blocks of 32 and
of 96 cells of one parity, the most of the two smallest forms of the kernel, one more layer, both forms in one solve, and small
structures beside larger ones, which then all take larger forms."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu


def solid(a, b, c, at):
    return np.stack(np.meshgrid(np.arange(a), np.arange(b), np.arange(c), indexing="ij"), -1).reshape(-1, 3) + np.array(at)


def scene(sizes, n, gap=21):
    """n structures in rows of 30, of the sizes in turn, of mixed materials."""
    parts = [solid(*sizes[k % len(sizes)], (5 + gap * (k % 30), 0, 5 + gap * (k // 30))) for k in range(n)]
    xyz = np.concatenate(parts).astype(np.int32)
    mat = np.array([S.CONC, S.MASON, S.STEEL, S.WOOD], np.uint8)[np.random.default_rng(n).integers(0, 4, len(xyz))]
    sid = np.concatenate([np.full(len(p), k, np.int32) for k, p in enumerate(parts)])
    return S.Scene(xyz, mat, sid, np.zeros(len(xyz), np.uint8)).contiguous()


@pytest.mark.parametrize("sizes,n", [([(8, 8, 8)], 300), ([(8, 9, 8)], 300), ([(16, 12, 8)], 200), ([(16, 13, 8)], 200),
                                     ([(1, 1, 1), (4, 4, 4), (8, 8, 8), (8, 9, 8), (16, 12, 8), (2, 40, 3)], 600),
                                     ([(8, 8, 8), (3, 1, 2), (8, 9, 8)], 36), ([(8, 8, 8), (3, 1, 2), (8, 9, 8)], 38),
                                     ([(1, 1, 1), (4, 4, 4), (8, 9, 8), (16, 12, 8), (16, 13, 8), (20, 20, 20)], 400)],
                         ids=["32", "36", "96", "104", "small", "few", "more", "beside larger"])
def test_many_small_structures_equal_grid_kernel(sf, sizes, n):
    sc = scene(sizes, n)
    ext = np.random.default_rng(1).uniform(0, 200, sc.n_static).astype(np.float32)
    got = []
    for c in (1, 0):
        w = sf.World(sc, sor_cluster=c)
        w.set_ext(ext)
        for sweeps, tol in ((1, 0.0), (6, 0.0), (300, 1e-3)):
            w.structure_solve(-1, 1.7, tol, sweeps)
            got.append((w.phi64(), *w.solve_detail()))
        assert w.stats().cluster_solves == 3 * c
        w.close()
    for x, y in zip(got[:3], got[3:]):
        for u, v in zip(x, y):
            assert np.array_equal(u, v)


def test_few_sweeps_of_many_tiny_structures(sf):
    """Six sweeps of 900 structures of 64 bricks take no longer than 1.6 times those of 100 structures of 5,760."""
    ms = []
    for sc in (scene([(4, 4, 4)], 900), scene([(12, 40, 12)], 100)):
        w = sf.World(sc)
        ms.append(min(w.structure_solve(-1, 1.7, 0.0, 6).ms for _ in range(8)))
        w.close()
    assert ms[0] < 1.6 * ms[1], ms
