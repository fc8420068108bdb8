"""Voxel.build's bucket lists and ray crossings where the kernels change form, bit for bit:
buckets of more than 1024 triangles (the ordered walk), lists longer than the
block's room for them, more than 512 crossings of a ray, repeated and
degenerate triangles, triangles of many samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random(n, size, seed):
    r = np.random.default_rng(seed)
    c = r.uniform(-1, 1, (n, 1, 3))
    return (c + r.uniform(-size, size, (n, 3, 3))).astype(np.float32).ravel()


def _sheets(n):
    """n parallel squares across x: a ray along x crosses every one of them."""
    out = []
    for x in np.linspace(-1, 1, n):
        a, b, c, d = ([x, y, z] for y, z in ((-1, -1), (1, -1), (1, 1), (-1, 1)))
        out += [a, b, c, a, c, d]
    return np.array(out, np.float32).ravel()


MESHES = {
    "large": lambda: _random(1500, 2.0, 1),        # most triangles in most buckets
    "small": lambda: _random(4000, 0.05, 2),
    "few": lambda: _random(5, 1.0, 3),
    "sheets": lambda: _sheets(700),
    "twice": lambda: np.tile(_random(200, 0.3, 4), 3),
    "flat": lambda: np.concatenate([_random(50, 0.4, 5), np.zeros(9 * 7, np.float32),
                                    np.tile(np.float32([0.1, 0.2, 0.3]), 9)]),
}


@pytest.mark.parametrize("mesh", sorted(MESHES))
@pytest.mark.parametrize("res", [7, 40])
def test_voxel_build_is_the_oracle(wt_lib, oracle_lib, mesh, res):
    from oracle.oracle import voxel_build as oracle_build
    from windtunnel_b200.mesh import voxel_build
    p = MESHES[mesh]()
    v, (grid, info) = voxel_build(p, res), oracle_build(p, res)
    assert np.array_equal(v.grid, grid)
    assert v.solid == info["solid"] and v.openness == info["openness"]
