"""The cluster path's tables from bricks in any order: listed at random, a structure in two scenes, structures of one to three
bricks beside others, with gaps and with bricks that no solve updates; against the grid kernel bit for bit."""
import numpy as np
import pytest

from shatterforge_b200 import scenes as S

pytestmark = pytest.mark.gpu


def solid(a, b, c, at):
    return np.stack(np.meshgrid(np.arange(a), np.arange(b), np.arange(c), indexing="ij"), -1).reshape(-1, 3) + np.array(at)


def scene(parts, seed):
    """Structure k is parts[k] with one brick in ten left out where it has more than ten, its bricks listed at random."""
    rng = np.random.default_rng(seed)
    parts = [p[rng.random(len(p)) < 0.9] if len(p) > 10 else p for p in parts]
    xyz = np.concatenate(parts).astype(np.int32)
    sid = np.concatenate([np.full(len(p), k, np.int32) for k, p in enumerate(parts)])
    order = rng.permutation(len(xyz))
    mat = rng.integers(1, 9, len(xyz)).astype(np.uint8)
    return S.Scene(xyz[order], mat[order], sid[order], np.zeros(len(xyz), np.uint8))


@pytest.mark.parametrize("sizes", [[(1, 1, 1)], [(2, 1, 1), (1, 3, 1), (1, 1, 1)], [(9, 20, 7), (1, 2, 1), (30, 4, 30)],
                                   [(60, 8, 60), (5, 5, 5), (70, 2, 80)]], ids=str)
@pytest.mark.parametrize("n_scenes", [1, 2])
def test_bricks_in_any_order(sf, sizes, n_scenes):
    scenes = [scene([solid(a, b, c, (37 + 80 * k, 0, 41 + 3 * q)) for k, (a, b, c) in enumerate(sizes)], 10 * q + len(sizes))
              for q in range(n_scenes)]
    n = sum(s.n_static for s in scenes)
    ext = np.random.default_rng(n).uniform(0, 200, n).astype(np.float32)
    got = []
    for c in (1, 0):
        w = sf.World(scenes, sor_cluster=c)
        w.set_ext(ext)
        for sweeps in (1, 60):
            w.structure_solve(-1, 1.7, 0.0, sweeps)
            got.append((w.phi64(), *w.solve_detail()))
        assert w.stats().cluster_solves == 2 * c
        w.close()
    for x, y in zip(got[:2], got[2:]):
        for u, v in zip(x, y):
            assert np.array_equal(u, v)
