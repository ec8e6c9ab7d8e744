"""The grid-wide IVC solve (more than 1024 markers): the Chebyshev iteration where
the operator's largest row sum is at most twice its regularisation, CG above.
Both against the stored inverse (FP64: relative L2 <= 1e-12 in populations, 1e-11
in the force), and both report what they cannot solve: a flow that is no longer
finite, an operator that exceeded its capacity, on every step."""
import numpy as np
import pytest

from ilbmrex_b200 import capi, cases

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.level import LevelSolver  # noqa: E402


def rel_l2(a, b):
    return float(np.sqrt(np.sum((a - b) ** 2) / max(np.sum(b ** 2), 1e-300)))


def body(reg, n=1100, D=330.0):
    case, ib, init = cases.cylinder(nx=380, ny=376, D=D, center=(190.3, 187.6), U=0.05, Re=200, n_marker=n)
    ib.ivc_diag_reg = reg
    return case, ib, init


def solver(reg, kind, storage="f64", **kw):
    case, ib, init = body(reg, **kw)
    s = LevelSolver(case, storage, ib=ib)
    s.set_ivc_solver(kind)
    s.set_macro(*init())
    return s


def row_sum_ratio(reg, n=1100, D=330.0):
    """Largest row sum of the operator over its regularisation (4-point kernel)."""
    th = 2.0 * np.pi * np.arange(n) / n
    dv = np.pi * D / n

    def weights(p):
        c = np.floor(p)[:, None] + np.arange(-2, 3)
        r = np.abs(c + 0.5 - p[:, None])
        inner = 0.125 * (3 - 2 * r + np.sqrt(np.maximum(1 + 4 * r - 4 * r * r, 0)))
        outer = 0.125 * (5 - 2 * r - np.sqrt(np.maximum(-7 + 12 * r - 4 * r * r, 0)))
        w = np.where(r < 1, inner, np.where(r < 2, outer, 0.0))
        full = np.zeros((n, 400))
        np.add.at(full, (np.arange(n)[:, None], c.astype(int)), w)
        return full

    wx, wy = weights(190.3 + D / 2 * np.cos(th)), weights(187.6 + D / 2 * np.sin(th))
    return float((dv * (wx @ wx.T) * (wy @ wy.T)).sum(1).max() + reg) / reg


@pytest.mark.parametrize("reg,chebyshev", [(1.3, True), (0.5, True), (0.25, False), (0.05, False)])
def test_grid_solve_equals_stored_inverse(reg, chebyshev):
    assert (row_sum_ratio(reg) <= 2.0) == chebyshev
    a, b = solver(reg, capi.IVC_CG), solver(reg, capi.IVC_DENSE)
    a.step(4, record_force=True)
    b.step(4, record_force=True)
    assert rel_l2(a.get_f(), b.get_f()) <= 1e-12
    assert rel_l2(a.get_force(), b.get_force()) <= 1e-11
    assert 0 < a.cg_iterations() < 500 and b.cg_iterations() == 0
    a.close()
    b.close()


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("reg", [1.3, 0.05])
def test_flow_that_is_not_finite_is_reported(reg, storage):
    s = solver(reg, capi.IVC_CG, storage)
    s.step(2, record_force=True)
    s.f[0, 0, 180:200, 20:40] = float("nan")  # (the body's left edge is at x = 25)
    torch.cuda.synchronize()
    for _ in range(2):
        with pytest.raises(capi.IlbmError, match="did not converge"):
            s.step(1, record_force=True)
    s.close()


def test_operator_beyond_its_capacity_is_reported_every_step():
    """1,500 markers on 63 cells of circumference: about 200 neighbours per row
    where the operator holds 96."""
    s = solver(1.3, capi.IVC_CG, n=1500, D=20.0)
    with pytest.raises(capi.IlbmError, match="capacity"):
        s.step(1, record_force=True)
    for _ in range(2):
        with pytest.raises(capi.IlbmError, match="did not converge"):
            s.step(1, record_force=True)
    s.close()
