"""Values at the edges of the number formats.

FP64: a cell whose numbers leave the range of the exact constant division is
redone with plain divisions; populations and stored macro fields that are
subnormal, huge, infinite or not a number against the CPU oracle, bit for bit
(NaN equal to NaN).

2-byte storage: the vector form stores v / s by a multiplication and one
correction, the cell form (rows on no vector boundary) divides; both store the
same bits for every kind of half, at scales inside and outside the vector form's
range."""
import numpy as np
import pytest

from ilbmrex_b200 import cases
from ilbmrex_b200.lattice import D2Q9, D3Q19, D3Q27
from oracle.checker import CpuLevel

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.level import LevelSolver  # noqa: E402

LAT = {"q9": D2Q9, "q19": D3Q19, "q27": D3Q27}


def level(lat, n, force=None, tau=None):
    nu = 0.07 if tau is None else (tau - 0.5) / 3.0
    return cases.LevelCase(lat, n if lat.dim == 3 else (n[0], n[1], 1), nu=nu, prescribed_force=force)


@pytest.mark.parametrize("lat", list(LAT))
@pytest.mark.parametrize("force", [None, (1e-4, -2e-5, 3e-5)], ids=["plain", "forced"])
@pytest.mark.parametrize("special", [(1e-310, -4e-320, 5e-324, 2.2e-308), (1e200, -1e300, 1e-200, 1e153),
                                     (float("inf"), float("nan"), -float("inf"), 0.0)],
                         ids=["subnormal", "huge", "nonfinite"])
def test_fp64_cells_outside_the_exact_division(lat, force, special):
    case = level(LAT[lat], (24, 18, 12), force)
    rng = np.random.default_rng(11)
    f = np.asarray(case.lattice.w).reshape(-1, 1, 1, 1) * (1.0 + 0.05 * rng.standard_normal((case.lattice.q,) + case.shape))
    m = [1.0 + 0.01 * rng.standard_normal(case.shape)] + [0.03 * rng.standard_normal(case.shape) for _ in range(3)]
    for a in [f] + m:  # one cell in thirty, each value alone and beside others
        hit = rng.random(a.shape) < 1.0 / 30
        a[hit] = rng.choice(np.array(special), size=int(hit.sum()))
    cpu, gpu = CpuLevel(case, "oracle"), LevelSolver(case, "f64")
    for s in (cpu, gpu):
        s.set_macro(m[0], m[1], m[2], m[3] if case.dim == 3 else None)
    cpu.set_f(f)
    gpu.set_f(f)
    gpu.first_step_macro = True  # the first step reads the stored fields, as the oracle's
    for _ in range(2):
        cpu.step(1)
        gpu.step(1)
        np.testing.assert_array_equal(gpu.get_f(), cpu.get_f())
    gpu.close()


@pytest.mark.parametrize("tau", [0.5000001, 2.0 ** 49, 2.0 ** 51])
def test_fp64_relaxation_times(tau):
    """Up to 2^50 the divisor's reciprocal is used, above it plain divisions."""
    case, init = cases.taylor_green(32, U0=0.02, tau=0.7)
    case.nu = (tau - 0.5) / 3.0
    cpu, gpu = CpuLevel(case, "oracle"), LevelSolver(case, "f64")
    cpu.set_macro(*init())
    cpu.init_equilibrium()
    gpu.set_macro(*init())
    cpu.step(3)
    gpu.step(3)
    np.testing.assert_array_equal(gpu.get_f(), cpu.get_f())
    gpu.close()


@pytest.mark.parametrize("lat", list(LAT))
@pytest.mark.parametrize("scale", [1024.0, 1.0, 3.7, 2.0 ** -30, 2.0 ** 37, 2.0 ** -39, 2.0 ** 39, 2.0 ** 45],
                         ids=lambda s: f"{s:.3g}")
def test_f16_stores_agree(lat, scale):
    case = level(LAT[lat], (67, 9, 5))
    special = torch.tensor([0x7c00, -0x400, 0x7e01, 0x0001, -0x7fff, 0x03ff, 0x7bff, -0x8000, 0x0400],
                           dtype=torch.int16).view(torch.float16)  # inf, -inf, NaN, subnormals, largest, -0
    got = []
    for plane in (False, True):
        s = LevelSolver(case, "f16", f16_scale=scale)
        if plane:
            s.f, s.f_next = (torch.zeros(s.fshape, dtype=s.f.dtype, device=s.dev) for _ in range(2))
        g = torch.Generator().manual_seed(7)
        f = 30.0 * torch.randn((case.lattice.q,) + case.shape, generator=g)
        f = (f * torch.exp2(torch.randint(-20, 11, f.shape, generator=g).float())).half()
        hit = torch.rand(f.shape, generator=g) < 0.002
        f[hit] = special[torch.randint(0, len(special), (int(hit.sum()),), generator=g)]
        s._valid(s.f, s.gf).copy_(f)
        torch.cuda.synchronize()
        s.step(1)
        s.ctx.sync()
        got.append(s._valid(s.f, s.gf).clone().contiguous().cpu())
        s.close()
    a, b = got
    same = (a.view(torch.int16) == b.view(torch.int16)) | (a.isnan() & b.isnan())
    assert bool(same.all())
    assert int(a.isfinite().sum()) > 0
