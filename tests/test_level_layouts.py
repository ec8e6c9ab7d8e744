"""The same levels in other layouts and forms: several boxes in one launch for
every lattice and storage form (raw populations, bit for bit the one-box
step), hierarchies whose fine rows start on no pair of cells, and force sums on
both sides of the one-block limit (12,288 cells)."""
import ctypes as C

import numpy as np
import pytest

from ilbmrex_b200 import capi, cases
from ilbmrex_b200.lattice import D2Q9, D3Q19, D3Q27

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.hierarchy import HierarchySolver  # noqa: E402
from ilbmrex_b200.level import Context, LevelSolver, alloc_populations, level_params  # noqa: E402


def cuts(n, k):
    e = [round(n * i / k) for i in range(k + 1)]
    return [(e[i], e[i + 1] - 1) for i in range(k)]


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("aligned", [False, True])
@pytest.mark.parametrize("lat,n,k", [(D2Q9, (70, 34, 1), (3, 2, 1)), (D3Q19, (19, 14, 13), (2, 2, 2)),
                                     (D3Q27, (34, 11, 9), (3, 3, 2))], ids=["q9", "q19", "q27"])
def test_boxes_in_one_launch(lat, n, k, storage, aligned):
    case = cases.LevelCase(lat, n, nu=0.06)
    d3 = case.dim == 3
    rng = np.random.default_rng(4)
    u = [0.02 * rng.standard_normal(case.shape) for _ in range(3)]
    one = LevelSolver(case, storage)
    one.set_macro(1.0 + 0.01 * rng.standard_normal(case.shape), u[0], u[1], u[2] if d3 else None)
    one.step(2)
    one.ctx.sync()
    f0 = one._valid(one.f, one.gf).clone()
    one.step(1)
    one.ctx.sync()
    f1 = one._valid(one.f, one.gf).clone()
    ctx = Context(lat, storage)
    boxes = [((x[0], y[0], z[0]), (x[1], y[1], z[1])) for z in cuts(n[2], k[2]) for y in cuts(n[1], k[1])
             for x in cuts(n[0], k[0])]
    arr, keep, lb = (capi.Box_t * len(boxes))(), [], []
    for b, (lo, hi) in zip(arr, boxes):
        ix = [torch.arange(lo[d] - 1, hi[d] + 2, device=f0.device) % n[d] if d < case.dim else
              torch.zeros(1, dtype=torch.long, device=f0.device) for d in range(3)]
        src = f0[:, ix[2]][:, :, ix[1]][:, :, :, ix[0]]
        make = (lambda: alloc_populations(*src.shape, src.dtype, src.device)) if aligned else \
            (lambda: torch.zeros(src.shape, dtype=src.dtype, device=src.device))
        fi, fo = make(), make()
        fi.copy_(src)
        keep.append((fi, fo))
        for d in range(3):
            b.lo[d], b.hi[d] = lo[d], hi[d]
        b.ngrow_f, b.ngrow_m = 1, 2
        fs = fi.stride()
        b.fstride[:] = [fs[2], fs[1], fs[0]]
        b.f_in, b.f_out = fi.data_ptr(), fo.data_ptr()
        lb += [*lo, *hi]
    p = level_params(case, uniform_force=False)
    lbc = (C.c_int * len(lb))(*lb)
    p.ghost_mode, p.nlevel_boxes = capi.GHOST_CALLER, len(boxes)
    p.level_boxes = C.cast(lbc, C.POINTER(C.c_int))
    torch.cuda.synchronize()
    capi.check(ctx.L.ilbm_level_step(ctx.h, arr, len(boxes), C.byref(p)), "level_step")
    ctx.sync()
    for (lo, hi), (_, fo) in zip(boxes, keep):
        got = fo[:, 1:-1, 1:-1, 1:-1] if d3 else fo[:, :, 1:-1, 1:-1]
        want = f1[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1]
        assert torch.equal(got, want)
    one.close()
    ctx.close()


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("lat,nlev", [(D2Q9, 3), (D3Q19, 2), (D3Q27, 2)], ids=["q9", "q19", "q27"])
def test_hierarchy_rows_on_no_pair(lat, nlev, storage):
    """Average-down loads two fine cells at once where every fine row starts on
    a pair, else one by one."""
    hc, inits = cases.shear_layer_hierarchy(n=32, nlev=nlev, lattice=lat)
    got = []
    for plane in (False, True):
        s = HierarchySolver(hc, storage)
        if plane:
            for lvl in s.levels:
                lvl.f, lvl.f_next = (torch.zeros(lvl.f.shape, dtype=lvl.f.dtype, device=s.dev) for _ in range(2))
        s.set_macro(*(i() for i in inits))
        s.step(3)
        s.ctx.sync()
        got.append([lvl.valid(lvl.f, lvl.gf).clone() for lvl in s.levels])
        s.close()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("lat,ext", [(D2Q9, (1, 1, 1)), (D2Q9, (1117, 11, 1)), (D2Q9, (128, 96, 1)),
                                     (D2Q9, (1, 12289, 1)), (D2Q9, (145, 113, 1)), (D3Q19, (32, 32, 12)),
                                     (D3Q19, (29, 113, 5))], ids=str)
def test_force_sum_around_the_limit(lat, ext, storage):
    n = tuple(e + 4 if d < lat.dim else 1 for d, e in enumerate(ext))
    case = cases.LevelCase(lat, n, nu=0.06)
    s = LevelSolver(case, storage)
    torch.manual_seed(3)
    s.force_cur.normal_()
    torch.cuda.synchronize()
    lo = [2 if d < lat.dim else 0 for d in range(3)]
    hi = [lo[d] + ext[d] - 1 for d in range(3)]
    out = (C.c_double * 3)()
    box = s._box(s.f, None, force=s.force_cur)
    capi.check(s.L.ilbm_force_integrals(s.ctx.h, C.byref(box), 1, capi.ivec3(lo), capi.ivec3(hi), out), "force")
    F = s._valid(s.force_cur, s.gm).double().cpu().numpy()
    F = F[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1]
    for c in range(lat.dim):
        assert abs(out[c] - F[c].sum()) <= 1e-13 * np.abs(F[c]).sum()
    s.close()
