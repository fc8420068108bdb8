"""The step kernels' mappings and the pair kernel's odd-width and moving-wall forms.

A lane's cell is found by one division of its index in the plane, across row
ends; force segments, the road's block order and the outlet copy follow from
it. Each case runs AUTO against the direct kernel, whose threads are cells.
Tolerance: both collide in float32, so a population differs by the rounding of
some 20 operations of its size (0.1 at most, 2^-24 relative: 1.2e-7) a step,
added up like a random walk over 25 steps: 6e-7; 1e-6 is allowed, the bar of
the other kernel comparisons. Forces sum populations of both signs: 1e-5 of
the largest.
"""
import numpy as np
import pytest

from lbm_cases import apply_case, spinning_sphere_wallvel

pytestmark = pytest.mark.gpu

DIMS = [(3, 5, 5), (5, 6, 7), (17, 9, 9), (33, 9, 8), (63, 8, 9), (65, 9, 9), (129, 8, 7),
        (257, 7, 6), (4, 6, 6), (34, 9, 8), (66, 7, 9), (160, 9, 8), (256, 8, 7), (512, 6, 6)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("side_bc", ["eq", "freeslip"])
def test_auto_float32_agrees_with_direct(wt_lib, dims, moving, side_bc):
    from windtunnel_b200 import LBM
    nx, ny, nz = dims
    body = (nx - 4.5, ny / 2, nz / 2, 2.6) if nx > 8 else None   # touches the outlet column
    out = []
    for kernel in ("direct", "auto"):
        s = LBM(*dims, kernel=kernel, side_bc=side_bc)
        apply_case(s, sphere=body, side_bc=side_bc, ground=True, roadVel=0.03 if moving else 0.0,
                   wallVel=spinning_sphere_wallvel(*body[:3], 0.01) if moving and body else None)
        f1 = s.step_forces(7)
        u1 = s.fields()
        f2 = s.step_forces(18)
        p = s.populations("f", "raw").reshape(19, nz, ny, nx)
        assert np.array_equal(p[:, 1:-1, 1:-1, -1], p[:, 1:-1, 1:-1, -2])
        out.append((np.concatenate([f1, f2]), u1, s.fields(), s.populations("f"),
                    s.populations("g")))
    (fa, ua1, ua2, pa, ga), (fb, ub1, ub2, pb, gb) = out
    assert np.abs(fa - fb).max() <= 1e-5 * max(np.abs(fa).max(), 1e-30)
    for a, b in list(zip(ua1, ub1)) + list(zip(ua2, ub2)):
        assert np.abs(a - b).max() <= 1e-6
    assert np.abs(pa - pb).max() <= 1e-6
    assert np.abs(ga - gb).max() <= 1e-6


@pytest.mark.parametrize("dims", [(17, 9, 9), (33, 9, 8), (65, 9, 9), (257, 7, 6)])
@pytest.mark.parametrize("side_bc", ["eq", "freeslip"])
@pytest.mark.parametrize("les,trt", [(True, True), (True, False), (False, True)])
def test_odd_width_is_the_lean_kernel(wt_lib, dims, side_bc, les, trt):
    """The odd-width form performs the lean kernel's operations: the same bits."""
    _same_bits(dims, "lean", side_bc, les, trt, 0.0)


@pytest.mark.parametrize("dims", [(17, 9, 9), (34, 9, 8), (65, 9, 9), (160, 9, 8), (256, 8, 7)])
@pytest.mark.parametrize("side_bc", ["eq", "freeslip"])
@pytest.mark.parametrize("les,trt", [(True, True), (True, False), (False, True)])
def test_moving_walls_are_the_direct_kernel(wt_lib, dims, side_bc, les, trt):
    """The moving-wall form performs the direct kernel's operations: the same bits."""
    _same_bits(dims, "direct", side_bc, les, trt, 0.03)


def _same_bits(dims, kernel, side_bc, les, trt, road):
    from windtunnel_b200 import LBM
    nx, ny, nz = dims
    body = (nx - 4.5, ny / 2, nz / 2, 2.6)
    out = []
    for k in (kernel, "auto"):
        s = LBM(*dims, kernel=k, side_bc=side_bc)
        apply_case(s, sphere=body, side_bc=side_bc, ground=True, roadVel=road, les=les, trt=trt,
                   tau=0.53, wallVel=spinning_sphere_wallvel(*body[:3], 0.01) if road else None)
        f = s.step_forces(12)
        out.append([f, s.populations("f", "raw"), s.populations("g", "raw"), *s.fields()])
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-12 * np.abs(out[0][0]).max()
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dims", [(33, 9, 8), (34, 9, 8), (97, 12, 11), (160, 9, 8)])
@pytest.mark.parametrize("moving", [False, True])
def test_exact_form_is_the_oracle_across_row_ends(wt_lib, oracle_lib, dims, moving):
    """Widths whose warps cross row ends, odd and even, over a road: bit for bit."""
    from oracle.oracle import OracleLBM
    from windtunnel_b200 import LBM
    nx, ny, nz = dims
    body = (nx - 6.5, ny / 2, nz / 2, 2.9)
    sims = []
    for s in (LBM(*dims, math="exact"), OracleLBM(*dims)):
        apply_case(s, sphere=body, side_bc="eq", ground=True, roadVel=0.03 if moving else 0.0,
                   wallVel=spinning_sphere_wallvel(*body[:3], 0.01) if moving else None)
        sims.append((s.step_forces(21), s.populations("f", "raw")))
    (fg, pg), (fo, po) = sims
    assert np.array_equal(pg, po)
    assert np.abs(fg - fo).max() <= 1e-12 * np.abs(fo).max()
