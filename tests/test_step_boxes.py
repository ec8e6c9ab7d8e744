"""A periodic level cut into boxes (caller-filled ghosts, all of them covered by
other boxes): ilbm_level_step on all boxes equals the one-box step bit for bit,
populations and macro fields, with fewer and more boxes than one launch takes,
with and without stored macro fields, in rows that do and do not start on
vector boundaries."""
import ctypes as C

import numpy as np
import pytest

from ilbmrex_b200 import capi, cases
from ilbmrex_b200.lattice import D2Q9, D3Q19

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.level import Context, LevelSolver, alloc_populations, level_params  # noqa: E402


def cuts(n, k):
    e = [round(n * i / k) for i in range(k + 1)]
    return [(e[i], e[i + 1] - 1) for i in range(k)]


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("aligned", [False, True])
@pytest.mark.parametrize("lat,n,k", [(D2Q9, (37, 41, 1), (1, 2, 1)), (D2Q9, (60, 50, 1), (4, 4, 1)),
                                     (D2Q9, (85, 61, 1), (5, 5, 1)), (D3Q19, (24, 21, 19), (3, 2, 3))])
def test_boxes_equal_one_box(lat, n, k, storage, aligned):
    case = cases.LevelCase(lat, n, nu=0.06)
    d3 = case.dim == 3
    rng = np.random.default_rng(3)
    u = [0.02 * rng.standard_normal(case.shape) for _ in range(3)]
    one = LevelSolver(case, storage)
    one.set_macro(1.0 + 0.01 * rng.standard_normal(case.shape), u[0], u[1], u[2] if d3 else None)
    one.step(2)
    f0 = one._valid(one.f, one.gf).clone()
    m0 = torch.as_tensor(one.get_macro()).to(one.macro.dtype).to(one.dev)
    one.step(1)
    f1, m1 = one.get_f(), one.get_macro()

    ctx = Context(lat, storage)
    boxes = [((x[0], y[0], z[0]), (x[1], y[1], z[1])) for z in cuts(n[2], k[2]) for y in cuts(n[1], k[1])
             for x in cuts(n[0], k[0])]
    arr, keep, lb = (capi.Box_t * len(boxes))(), [], []

    def grown(t, lo, hi, w):
        ix = [torch.arange(lo[d] - w, hi[d] + 1 + w, device=t.device) % n[d] if d < case.dim else
              torch.zeros(1, dtype=torch.long, device=t.device) for d in range(3)]
        return t[:, ix[2]][:, :, ix[1]][:, :, :, ix[0]]

    for b, (lo, hi) in zip(arr, boxes):
        src = grown(f0, lo, hi, 1)
        if aligned:
            fi, fo = (alloc_populations(*src.shape, src.dtype, src.device) for _ in range(2))
            fi.copy_(src)
        else:
            fi, fo = src.contiguous(), torch.zeros_like(src).contiguous()
        mi = grown(m0, lo, hi, 2).contiguous()
        mo = torch.zeros_like(mi)
        keep.append((fi, fo, mi, mo))
        for d in range(3):
            b.lo[d], b.hi[d] = lo[d], hi[d]
        b.ngrow_f, b.ngrow_m = 1, 2
        fs, ms = fi.stride(), mi.stride()
        b.fstride[:] = [fs[2], fs[1], fs[0]]
        b.mstride[:] = [ms[2], ms[1], ms[0]]
        b.f_in, b.f_out, b.macro_out = fi.data_ptr(), fo.data_ptr(), mo.data_ptr()
        # stored macro fields where they are exactly the populations' (FP32 ones carry 1 + drho rounded)
        b.macro_in = mi.data_ptr() if aligned and storage == "f64" else None
        lb += [*lo, *hi]
    p = level_params(case, uniform_force=False)
    lbc = (C.c_int * len(lb))(*lb)
    p.ghost_mode, p.nlevel_boxes = capi.GHOST_CALLER, len(boxes)
    p.level_boxes = C.cast(lbc, C.POINTER(C.c_int))
    torch.cuda.synchronize()
    capi.check(ctx.L.ilbm_level_step(ctx.h, arr, len(boxes), C.byref(p)), "level_step")
    ctx.sync()
    w = torch.tensor(lat.w, dtype=torch.float64, device=one.dev).view(-1, 1, 1, 1)
    for (lo, hi), (_, fo, _, mo) in zip(boxes, keep):
        s = (slice(None), slice(lo[2], hi[2] + 1), slice(lo[1], hi[1] + 1), slice(lo[0], hi[0] + 1))
        cut = lambda t, g: t[:, g:-g, g:-g, g:-g] if d3 else t[:, :, g:-g, g:-g]
        got = cut(fo, 1).double()
        got = got + w if storage != "f64" else got
        np.testing.assert_array_equal(got.cpu().numpy(), f1[s])
        nm = 4 if d3 else 3
        np.testing.assert_array_equal(cut(mo, 2)[:nm].double().cpu().numpy(), m1[s][:nm])
    one.close()
    ctx.close()
