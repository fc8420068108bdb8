"""Device snapshots: a restored lattice is the lattice that was, bit for bit."""
import numpy as np
import pytest

from lbm_cases import apply_case, spinning_sphere_wallvel

pytestmark = pytest.mark.gpu


def _lattice(storage="f32", nx=40, moving=False, **kw):
    from windtunnel_b200 import LBM
    s = LBM(nx, 12, 11, storage=storage)
    wall = spinning_sphere_wallvel(20.0, 6.0, 5.0, 0.01) if moving else None
    apply_case(s, sphere=(20.0, 6.0, 5.0, 3.0), ground=True, roadVel=0.02 if moving else 0.0,
               wallVel=wall, **kw)
    return s


def _all(s):
    return [s.populations("f", "raw"), s.populations("g", "raw"), s.solid, s.near,
            *s.fields(), s.force, np.array([s.steps, s.parity, s.movingWalls])]


@pytest.mark.parametrize("storage,nx,moving", [("f32", 40, False), ("f32", 41, True),
                                               ("f16dev", 40, True), ("f64", 41, False)])
@pytest.mark.parametrize("revoxelize", [False, True])
def test_restore_is_the_state(wt_lib, storage, nx, moving, revoxelize):
    s = _lattice(storage, nx, moving)
    s.step_forces(5)
    want = _all(s)
    snap = s.snapshot()
    follow = s.step_forces(7)
    end = _all(s)
    if revoxelize:   # another body: flags, masks and slots have to come back too
        apply_case(s, sphere=(15.0, 5.0, 6.0, 2.2), ground=False, amp=0)
        s.step_forces(2)
    s.restore(snap)
    for a, b in zip(_all(s), want):
        assert np.array_equal(a, b)
    assert np.array_equal(s.step_forces(7), follow)
    for a, b in zip(_all(s), end):
        assert np.array_equal(a, b)
    snap.close(keep=True)
    again = s.snapshot()   # from the kept block
    s.step_forces(3)
    s.restore(again)
    for a, b in zip(_all(s), end):
        assert np.array_equal(a, b)


def test_restore_into_a_like_lattice(wt_lib):
    from windtunnel_b200 import LBM, WTError
    a, b = _lattice(seed=5), LBM(40, 12, 11)
    a.step_forces(4)
    snap = a.snapshot()
    b.restore(snap)
    assert np.array_equal(a.step_forces(6), b.step_forces(6))
    assert np.array_equal(a.populations("f", "raw"), b.populations("f", "raw"))
    for other in (LBM(41, 12, 11), LBM(40, 12, 11, storage="f64")):
        with pytest.raises(WTError):
            other.restore(snap)


def test_drag_gradient_twice_and_after_other_steps(wt_lib):
    """autograd keeps its own start state: the lattice may move on in between,
    and ends where it was."""
    import torch
    from windtunnel_b200.autograd import drag
    out = []
    for disturb in (False, True):
        sim = _lattice("f32", 40)
        s = torch.full((4, 4, 4), 0.4, dtype=torch.float64, requires_grad=True)
        J = drag(s, sim, (26, 4, 4, 30, 8, 8), 12, 4, keep=disturb)
        if disturb:
            sim.step_forces(3)
        before = _all(sim)
        J.backward(retain_graph=True)
        J.backward()
        for a, b in zip(_all(sim), before):
            assert np.array_equal(a, b)
        out.append((float(J.detach()), s.grad.clone()))
    assert out[0][0] == out[1][0] and torch.equal(out[0][1], out[1][1])
