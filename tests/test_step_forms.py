"""The two forms of the level step agree bit for bit: rows that start on
V-cell boundaries (the library's own layout) take the vector form, AMReX's
plane layout takes the cell form.  The same case is stepped in both layouts,
at row lengths around the vector width and the 30-lane window of a warp, with
every face type, a uniform force, and a body (force arrays, skipped band,
stored macro fields on the first step)."""
import numpy as np
import pytest

from ilbmrex_b200 import cases
from ilbmrex_b200.lattice import D2Q9, D3Q19, D3Q27

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.level import LevelSolver  # noqa: E402

BC = {"periodic": (0, 0), "walls": (cases.USER_1, cases.USER_1), "mirror": (cases.USER_2, cases.USER_2),
      "flow": (cases.EXT_DIR, cases.FOEXTRAP)}


def level(lat, n, faces, force=None):
    per = tuple(f == "periodic" for f in faces)
    val = ((1.0, 0.02, 0.01, 0.0),) * 3
    return cases.LevelCase(lat, n, periodic=per, bc_lo=tuple(BC[f][0] for f in faces),
                           bc_hi=tuple(BC[f][1] for f in faces), bc_lo_val=val, bc_hi_val=val, nu=0.07,
                           prescribed_force=force)


def run(case, ib, storage, plane, steps=3):
    s = LevelSolver(case, storage, ib=ib)
    if plane:  # contiguous planes: odd strides, rows on no boundary
        s.f, s.f_next = (torch.zeros(s.fshape, dtype=s.f.dtype, device=s.dev) for _ in range(2))
    rng = np.random.default_rng(5)
    sh = case.shape
    u = [0.02 * rng.standard_normal(sh) for _ in range(3)]
    s.set_macro(1.0 + 0.01 * rng.standard_normal(sh), u[0], u[1], u[2] if case.dim == 3 else None)
    s.step(steps)
    f = s.get_f()
    s.close()
    return f


P, W, M, F = "periodic", "walls", "mirror", "flow"


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("n,faces,force", [
    ((1, 7, 1), (P, P, P), None), ((3, 5, 1), (W, W, P), None), ((4, 4, 1), (P, W, P), (1e-4, 0.0, 0.0)),
    ((119, 9, 1), (F, P, P), None), ((120, 6, 1), (P, M, P), None), ((121, 6, 1), (W, F, P), None),
    ((130, 11, 1), (F, W, P), (0.0, 1e-4, 0.0)), ((257, 5, 1), (M, P, P), None), ((500, 3, 1), (P, F, P), None)])
def test_forms_agree_2d(storage, n, faces, force):
    case = level(D2Q9, n, faces, force)
    np.testing.assert_array_equal(run(case, None, storage, False), run(case, None, storage, True))


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("lat", [D3Q19, D3Q27], ids=["q19", "q27"])
@pytest.mark.parametrize("n,faces,force", [
    ((2, 3, 4), (P, P, P), None), ((33, 5, 3), (P, M, W), (1e-4, 0.0, 0.0)), ((61, 4, 5), (F, P, P), None),
    ((60, 3, 3), (W, W, W), None), ((125, 4, 3), (P, P, M), None), ((130, 3, 4), (M, F, P), None)])
def test_forms_agree_3d(storage, lat, n, faces, force):
    case = level(lat, n, faces, force)
    np.testing.assert_array_equal(run(case, None, storage, False), run(case, None, storage, True))


@pytest.mark.parametrize("nx", [61, 96, 131])
def test_forms_agree_with_a_body(nx):
    """The band is stepped apart from the rest (a skipped box inside the rows).
    Spreading sums with FP64 atomics, whose order may move a force by one
    float: relative L2 <= 1e-6 instead of equality."""
    case, ib, _ = cases.cylinder(nx=nx, ny=48, D=10, center=(22.3, 23.7), U=0.05, Re=40)
    a, b = run(case, ib, "f32", False), run(case, ib, "f32", True)
    assert np.sqrt(np.sum((a - b) ** 2) / np.sum(b ** 2)) <= 1e-6
