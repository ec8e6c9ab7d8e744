"""Calls of the level step at the edges of what it takes."""
import ctypes as C

import numpy as np
import pytest

from ilbmrex_b200 import capi, cases
from ilbmrex_b200.lattice import D2Q9

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.level import Context, LevelSolver, level_params  # noqa: E402


@pytest.mark.parametrize("count,table", [(65, True), (2, False)])
def test_self_filled_level_ignores_the_level_boxes(count, table):
    """Self-filled ghosts: level_boxes is a caller-mode field, whatever it holds."""
    case, init = cases.taylor_green(24, U0=0.02, tau=0.7)
    out = []
    for listed in (False, True):
        s = LevelSolver(case, "f64")
        s.set_macro(*init())
        if listed:
            lb = (C.c_int * (6 * count))()
            s.params.nlevel_boxes = count
            if table:
                s.params.level_boxes = C.cast(lb, C.POINTER(C.c_int))
        s.step(3)
        out.append(s.get_f())
        s.close()
    np.testing.assert_array_equal(out[0], out[1])
