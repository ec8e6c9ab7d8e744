"""Calls of ilbm_ib_update_forcing at the edges of what it takes, for bodies
whose chain is one launch and for those that take a launch per stage (FP64:
the exported force bit for bit, explicit coupling summing in a fixed order)."""
import ctypes as C

import numpy as np
import pytest

from ilbmrex_b200 import capi, cases

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.level import LevelSolver  # noqa: E402


def stepped(n, cy=35.6, coupling=0, steps=3):
    case, ib, init = cases.cylinder(nx=96, ny=72, D=30, center=(40.3, cy), U=0.05, Re=40, n_marker=n,
                                    coupling=coupling)
    s = LevelSolver(case, "f64", ib=ib)
    s.set_macro(*init())
    s.step(steps)
    s.ctx.sync()
    return s


def update(s, box):
    torch.cuda.synchronize()
    capi.check(s.L.ilbm_ib_update_forcing(s.ib, C.byref(box), 1, C.byref(s.params), s.case.dt, s.time), "update_forcing")
    s.ctx.sync()


@pytest.mark.parametrize("n", [60, 512, 513])
def test_force_in_place(n):
    """One array for F^{n-1} (read) and F^n (written)."""
    s = stepped(n)
    apart = torch.zeros_like(s.force_prev)
    update(s, s._box(s.f, None, force=apart, force_prev=s.force_prev))
    one = s.force_prev.clone()
    update(s, s._box(s.f, None, force=one, force_prev=one))
    assert float(apart.abs().max()) > 0.0
    np.testing.assert_array_equal(one.cpu().numpy(), apart.cpu().numpy())
    s.close()


@pytest.mark.parametrize("n", [40, 513])
def test_caller_filled_band_over_a_periodic_face(n):
    """Caller-filled macro fields: the band's ghosts beyond a periodic face are
    their images whatever the caller's ghost cells hold there."""
    s = stepped(n, cy=6.2)
    m = torch.zeros_like(s.macro)
    s._valid(m, s.gm).copy_(torch.as_tensor(s.get_macro()).to(m.device))
    p = s.params
    s.params = type(p).from_buffer_copy(p)
    s.params.ghost_mode = capi.GHOST_CALLER
    out = []
    for fill in (False, True):
        if fill:  # the two ghost rows on each y face
            m[..., 0:2, :] = m[..., -4:-2, :]
            m[..., -2:, :] = m[..., 2:4, :]
        f = torch.zeros_like(s.force_prev)
        update(s, s._box(s.f, None, macro_in=m, force=f))
        out.append(f.cpu().numpy())
    s.params = p
    f = torch.zeros_like(s.force_prev)
    update(s, s._box(s.f, None, force=f, force_prev=s.force_prev))  # self-filled, from the populations
    assert np.abs(out[1]).max() > 0.0
    np.testing.assert_array_equal(out[0], out[1])
    np.testing.assert_array_equal(f.cpu().numpy(), out[1])
    s.close()


@pytest.mark.parametrize("center", [(15.2, 2.4, 13.7), (15.2, 14.9, 26.1), (15.2, 1.2, 0.8)])
def test_sphere_over_a_periodic_face(center):
    """The 3D chain's band beyond periodic faces, an edge of two among them:
    explicit coupling against the oracle."""
    from oracle.checker import CpuLevel
    case, ib, init = cases.sphere(36, 30, 28, D=8.0, center=center, U=0.04, Re=30.0, coupling=0)
    cpu = CpuLevel(case, "oracle")
    cpu.set_macro(*init())
    cpu.init_equilibrium()
    cpu.ib_create(ib)
    cpu.step(4)
    s = LevelSolver(case, "f64", ib=ib)
    s.set_macro(*init())
    s.step(4)
    f, g = s.get_f(), cpu.get_f()
    assert np.sqrt(np.sum((f - g) ** 2) / np.sum(g ** 2)) <= 1e-12
    s.close()


@pytest.mark.parametrize("n,refused", [(240, False), (400, True), (440, True), (600, True)])
def test_markers_too_dense_are_refused(n, refused):
    """A rebuilt 2D operator holds 96 neighbours per row on average; on 31 cells of
    circumference 240 markers have about 70, 400 about 120.  Alone and in a batch,
    whichever solve takes them."""
    from ilbmrex_b200.batch import Batch
    from ilbmrex_b200.lattice import D2Q9
    case, ib, init = cases.cylinder(nx=64, ny=48, D=10, center=(24.3, 23.6), U=0.05, Re=40, n_marker=n)
    ib.ivc_rebuild_matrix = 1
    B = Batch(D2Q9, "f32")
    s, joined = B.solver(case, ib, init), False
    try:
        s.step(1)
        for _ in range(2):
            if refused:
                with pytest.raises(capi.IlbmError, match="capacity"):
                    s.step(1, record_force=True)
            else:
                s.step(1, record_force=True)
        joined = B.add(s, max_steps=8) > 0
        B.step(2)
        if refused:
            with pytest.raises(capi.IlbmError, match="capacity"):
                B.progress()
        else:
            B.progress()
    finally:
        if not joined:
            s.close()
        B.close()
