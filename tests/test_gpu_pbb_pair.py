"""The float32 partial-bounce-back step on the pair kernel, against the oracle in float64.

Widths at the edges of warps and segments, odd and even, a box that touches the
outlet column, a body inside it, both side conditions. Tolerance: the float32
update rounds some 25 operations of populations of size 0.1 at most (2^-24
relative) a step, so 20 steps leave at most 20 * 25 * 0.1 * 6e-8 = 3e-6 if all
errors added up; 1e-6 is allowed. The force adds links of both signs:
1e-5 of its largest value.
"""
import numpy as np
import pytest

from lbm_cases import apply_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,box", [
    ((24, 12, 12), (6, 2, 2, 14, 10, 10)), ((25, 12, 11), (6, 2, 2, 14, 10, 9)),
    ((33, 9, 9), (25, 2, 2, 33, 7, 7)), ((34, 9, 9), (25, 2, 2, 34, 7, 7)),
    ((33, 9, 9), (32, 3, 3, 33, 5, 5)), ((65, 8, 9), (31, 1, 1, 34, 7, 8)),
    ((256, 7, 7), (63, 2, 2, 66, 5, 5)), ((100, 9, 8), (0, 0, 0, 100, 9, 8))])
@pytest.mark.parametrize("side_bc", ["eq", "freeslip"])
@pytest.mark.parametrize("body", [False, True])
def test_pbb_float32_close_to_float64_oracle(wt_lib, oracle_lib, dims, box, side_bc, body):
    from oracle.oracle import OracleLBM
    from windtunnel_b200 import LBM
    nx, ny, nz = dims
    x0, y0, z0, x1, y1, z1 = box
    s = np.random.default_rng(3).uniform(0, 1, (z1 - z0, y1 - y0, x1 - x0))
    s[s < 0.2] = 0.0
    sphere = (x0 + 1.5, ny / 2, nz / 2, 1.6) if body and x0 > 4 else None
    out = []
    for sim in (LBM(*dims, side_bc=side_bc), OracleLBM(*dims, "f64", side_bc=side_bc)):
        apply_case(sim, u0=0.05, tau=0.53, side_bc=side_bc, sphere=sphere)
        sim.set_solid_fraction(box, s)
        f = sim.step_forces(20)
        out.append((f, sim.fields(), sim.populations("f", "f64")))
    (fa, ua, pa), (fb, ub, pb) = out
    assert np.abs(fa - fb).max() <= 1e-5 * np.abs(fb).max()
    for a, b in zip(ua, ub):
        assert np.abs(a - b).max() <= 1e-6
    assert np.abs(pa - pb).max() <= 1e-6


@pytest.mark.parametrize("storage,nx", [("f32", 34), ("f32", 33), ("f32", 256), ("f16dev", 34),
                                        ("f16dev", 130)])
@pytest.mark.parametrize("side_bc", ["eq", "freeslip"])
@pytest.mark.parametrize("les,trt", [(True, True), (True, False), (False, True)])
def test_pbb_is_the_one_cell_kernel(wt_lib, storage, nx, side_bc, les, trt):
    """The pair form performs the one-cell kernel's operations: the same bits. The
    moving-walls switch selects the one-cell kernel; with walls at rest its
    correction is zero."""
    from windtunnel_b200 import LBM
    out = []
    for moving in (True, False):
        s = LBM(nx, 10, 9, storage=storage, side_bc=side_bc)
        apply_case(s, u0=0.05, tau=0.53, side_bc=side_bc, sphere=(9.0, 5.0, 4.0, 2.2), les=les,
                   trt=trt)
        s.set_solid_fraction((12, 2, 2, 25, 8, 7),
                             np.random.default_rng(2).uniform(0, 1, (5, 6, 13)).round(1))
        s.movingWalls = moving
        f = s.step_forces(15)
        out.append([f, s.populations("f", "raw"), *s.fields()])
    # the blend's force adds its directions in float32 in another order
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-5 * np.abs(out[0][0]).max()
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)


def test_pbb_adjoint_is_independent_of_the_checkpoints(wt_lib):
    """Forward sweep and recomputation run the same kernel: equal gradients."""
    from windtunnel_b200 import LBM
    for nx in (40, 41):
        got = []
        for c in (3, 7, 20):
            sim = LBM(nx, 12, 11, side_bc="freeslip")
            apply_case(sim, u0=0.05, tau=0.53, side_bc="freeslip")
            s = np.random.default_rng(1).uniform(0, 1, (6, 6, 8))
            sim.set_solid_fraction((10, 3, 2, 18, 9, 8), s)
            J, g, _ = sim.adjoint(20, 7, 0, c)
            got.append((J, g))
        assert all(J == got[0][0] and np.array_equal(g, got[0][1]) for J, g in got[1:])
