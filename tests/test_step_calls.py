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


@pytest.mark.parametrize("nx,ny", [((1 << 26) - 4, 1), ((1 << 26) + 5, 1), (32771, 32800)])
def test_box_of_very_many_cells(nx, ny):
    """One box of a level of two, its rows longer or its cells more (2^30 and
    some) than one several-box launch takes: the same bits as the box taken as
    its level's only one (no ghost cell is covered by the other box)."""
    from ilbmrex_b200.level import alloc_populations
    ctx = Context(D2Q9, "f16")
    dev = torch.device("cuda")
    fi = alloc_populations(9, 1, ny + 2, nx + 2, torch.float16, dev)
    outs = [alloc_populations(9, 1, ny + 2, nx + 2, torch.float16, dev) for _ in range(2)]
    torch.manual_seed(1)
    for q in range(9):
        fi[q].normal_(0.0, 20.0)
    case = cases.LevelCase(D2Q9, (nx + 300, ny + 40, 1), nu=0.06)
    for fo, boxes in zip(outs, (1, 2)):
        b = capi.Box_t()
        for d, (lo, hi) in enumerate(((100, 100 + nx - 1), (20, 20 + ny - 1), (0, 0))):
            b.lo[d], b.hi[d] = lo, hi
        b.ngrow_f, b.ngrow_m = 1, 2
        fs = fi.stride()
        b.fstride[:] = [fs[2], fs[1], fs[0]]
        b.f_in, b.f_out = fi.data_ptr(), fo.data_ptr()
        lb = (C.c_int * 12)(100, 20, 0, 100 + nx - 1, 20 + ny - 1, 0, 0, 0, 0, 9, 4, 0)
        p = level_params(case, uniform_force=False)
        p.ghost_mode, p.nlevel_boxes = capi.GHOST_CALLER, boxes
        p.level_boxes = C.cast(lb, C.POINTER(C.c_int))
        torch.cuda.synchronize()
        capi.check(ctx.L.ilbm_level_step(ctx.h, C.byref(b), 1, C.byref(p)), "level_step")
        ctx.sync()
    for q in range(9):
        assert torch.equal(outs[0][q, 0, 1:-1, 1:-1], outs[1][q, 0, 1:-1, 1:-1])
    assert float(outs[0][1, 0, -2, 1:-1].abs().max()) > 0.0
    ctx.close()
    del fi, fo, outs
    torch.cuda.empty_cache()


@pytest.mark.parametrize("nx,ny", [(1024, 96), (32771, 32800)])
def test_batched_case_of_very_many_cells(nx, ny):
    """One step of a batched periodic case, of more than 2^30 cells too, is the
    level step's, bit for bit."""
    from ilbmrex_b200.level import alloc_populations
    ctx = Context(D2Q9, "f16")
    dev = torch.device("cuda")
    fi, one, two = (alloc_populations(9, 1, ny + 2, nx + 2, torch.float16, dev) for _ in range(3))
    torch.manual_seed(2)
    for q in range(9):
        fi[q].normal_(0.0, 20.0)
    case = cases.LevelCase(D2Q9, (nx, ny, 1), nu=0.06)
    p = level_params(case, uniform_force=False)
    b = capi.Box_t()
    for d, n in enumerate((nx, ny, 1)):
        b.lo[d], b.hi[d] = 0, n - 1
    b.ngrow_f, b.ngrow_m = 1, 2
    fs = fi.stride()
    b.fstride[:] = [fs[2], fs[1], fs[0]]
    b.f_in, b.f_out = fi.data_ptr(), one.data_ptr()
    torch.cuda.synchronize()
    capi.check(ctx.L.ilbm_level_step(ctx.h, C.byref(b), 1, C.byref(p)), "level_step")
    h, cid = C.c_void_p(), C.c_int()
    capi.check(ctx.L.ilbm_batch_create(ctx.h, 8, C.byref(h)), "batch_create")
    b.f_out = two.data_ptr()
    capi.check(ctx.L.ilbm_batch_add(h, C.byref(b), C.byref(p), None, 1.0, 0.0, 4, C.byref(cid)), "batch_add")
    capi.check(ctx.L.ilbm_batch_step(h, 1), "batch_step")
    ctx.sync()
    for q in range(9):
        assert torch.equal(one[q, 0, 1:-1, 1:-1], two[q, 0, 1:-1, 1:-1])
    ctx.L.ilbm_batch_destroy(h)
    ctx.close()
    del fi, one, two
    torch.cuda.empty_cache()


def test_average_down_of_an_empty_box():
    """A fine box of no cells on a level in between: nothing to average, and the
    next call on the context works."""
    ctx = Context(D2Q9, "f64")
    dev = torch.device("cuda")
    f, m = torch.zeros((9, 1, 34, 34), device=dev, dtype=torch.float64), torch.zeros((4, 1, 36, 36), device=dev, dtype=torch.float64)
    case = cases.LevelCase(D2Q9, (64, 64, 1), nu=0.06)

    def box(lo, hi):
        b = capi.Box_t()
        for d in range(2):
            b.lo[d], b.hi[d] = lo, hi
        b.ngrow_f, b.ngrow_m = 1, 2
        b.fstride[:] = [34, 34 * 34, 34 * 34]
        b.mstride[:] = [36, 36 * 36, 36 * 36]
        b.f_in, b.macro_in = f.data_ptr(), m.data_ptr()
        return b

    pc, pf = level_params(case, uniform_force=False), level_params(case, uniform_force=False)
    pc.ghost_mode = pf.ghost_mode = capi.GHOST_CALLER
    for d in range(2):
        pf.domain_hi[d] = 2 * pc.domain_hi[d] + 1
    coarse, fine = box(0, 31), box(16, 15)
    torch.cuda.synchronize()
    capi.check(ctx.L.ilbm_average_down(ctx.h, C.byref(coarse), C.byref(pc), C.byref(fine), C.byref(pf)), "average_down")
    out = torch.zeros_like(f)
    b = box(0, 31)
    b.f_out, b.macro_in = out.data_ptr(), None
    p = level_params(cases.LevelCase(D2Q9, (32, 32, 1), nu=0.06), uniform_force=False)
    capi.check(ctx.L.ilbm_level_step(ctx.h, C.byref(b), 1, C.byref(p)), "level_step")
    ctx.sync()
    ctx.close()
