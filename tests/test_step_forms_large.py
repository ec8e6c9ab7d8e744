"""The two forms of the level step agree bit for bit on levels with enough cells
for the vector form: more than 2^17 with reflecting faces, 2^15 without (below,
every level takes the cell form), at row lengths around the vector width and the
30-lane window of a warp, and on both sides of those limits."""
import numpy as np
import pytest

from ilbmrex_b200 import cases
from ilbmrex_b200.lattice import D2Q9, D3Q19, D3Q27

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from tests.test_step_forms import F, M, P, W, level, run  # noqa: E402


def rows(faces, cells):
    return -(-((1 << 17 if W in faces else 1 << 15) + 1) // cells)


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("nx,faces,force", [
    (1, (P, P, P), None), (3, (W, W, P), None), (4, (P, W, P), (1e-4, 0.0, 0.0)), (119, (F, P, P), None),
    (120, (P, M, P), None), (121, (W, F, P), None), (130, (F, W, P), (0.0, 1e-4, 0.0)), (257, (M, P, P), None),
    (500, (P, F, P), None), (32769, (W, P, P), None)])
def test_forms_agree_2d(storage, nx, faces, force):
    case = level(D2Q9, (nx, rows(faces, nx), 1), faces, force)
    np.testing.assert_array_equal(run(case, None, storage, False, 2), run(case, None, storage, True, 2))


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("lat", [D3Q19, D3Q27], ids=["q19", "q27"])
@pytest.mark.parametrize("nx,ny,faces,force", [
    (2, 30, (P, P, P), None), (33, 25, (P, M, W), (1e-4, 0.0, 0.0)), (61, 14, (F, P, P), None),
    (60, 43, (W, W, W), None), (125, 14, (P, P, M), None), (130, 13, (M, F, P), None)])
def test_forms_agree_3d(storage, lat, nx, ny, faces, force):
    case = level(lat, (nx, ny, rows(faces, nx * ny)), faces, force)
    np.testing.assert_array_equal(run(case, None, storage, False, 2), run(case, None, storage, True, 2))


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("n,faces", [((128, 1024, 1), (P, W, P)), ((128, 1025, 1), (P, W, P)),
                                     ((128, 256, 1), (P, M, P)), ((128, 257, 1), (P, M, P))])
def test_forms_agree_around_the_limits(storage, n, faces):
    case = level(D2Q9, n, faces)
    np.testing.assert_array_equal(run(case, None, storage, False), run(case, None, storage, True))


@pytest.mark.parametrize("nx", [261, 296, 331])
def test_forms_agree_with_a_body(nx):
    """A skipped box inside the rows; FP64 atomics in the spreading may move a
    force by one float: relative L2 <= 1e-6 instead of equality."""
    case, ib, _ = cases.cylinder(nx=nx, ny=160, D=10, center=(62.3, 83.7), U=0.05, Re=40)
    a, b = run(case, ib, "f32", False), run(case, ib, "f32", True)
    assert np.sqrt(np.sum((a - b) ** 2) / np.sum(b ** 2)) <= 1e-6
