"""The batch's solve of bodies whose operator is rebuilt every step: a cluster of
eight blocks per body where the rows of all of them fit the blocks' shared
memory and all clusters run in two waves, the sparse operators and one block's CG
each otherwise.  Each body in the batch equals the same body advanced alone
(relative L2 <= 1e-12 in populations, records to 1e-9: both solve to 1e-14), at
marker counts with blocks that own no rows, around the blocks' and warps'
shares, on both sides of the shared-memory limit (400 markers in 2D), with bodies
of both sides, and with more bodies than one and two waves hold."""
import numpy as np
import pytest

from ilbmrex_b200 import capi, cases
from ilbmrex_b200.lattice import D2Q9

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from ilbmrex_b200.batch import Batch  # noqa: E402
from ilbmrex_b200.level import LevelSolver  # noqa: E402


def rel_l2(a, b):
    return float(np.sqrt(np.sum((a - b) ** 2) / max(np.sum(b ** 2), 1e-300)))


def body(n):
    case, ib, init = cases.cylinder(nx=96, ny=72, D=30, center=(40.3, 35.6), U=0.05, Re=40, n_marker=n)
    ib.ivc_rebuild_matrix = 1
    return case, ib, init


@pytest.mark.parametrize("counts", [(1, 2, 7, 8, 9), (15, 16, 17, 63, 65), (127, 128, 129, 241),
                                    (399, 400), (401, 449), (33, 400, 401), (1, 9, 17, 33) * 6, (1, 9, 17, 33) * 10],
                         ids=lambda c: "-".join(map(str, c[:4])) + f"x{len(c)}")
def test_rebuilt_bodies_match_alone(counts):
    steps = 5
    B = Batch(D2Q9, "f64")
    ids = [B.add(B.solver(*body(n)), max_steps=16) for n in counts]
    B.step(steps)
    for n, cid in zip(counts, ids):
        s = B.sync(cid)
        case, ib, init = body(n)
        ref = LevelSolver(case, "f64", ib=ib)
        ref.set_macro(*init())
        ref.step(1 + steps, record_force=True)
        assert rel_l2(s.get_f(), ref.get_f()) <= 1e-12, n
        np.testing.assert_allclose(s.rec[3:5], ref.rec[3:5], rtol=1e-9, atol=1e-12, err_msg=str(n))
        ref.close()
    B.close()


def test_status_is_the_last_steps(tmp_path):
    """A stencil that left its band on an earlier step (the body took another
    one's checkpoint, and its own again) is no error of the batch's later steps;
    one that leaves in the batch's last step is."""
    def make(x, make_solver):
        case, ib, init = cases.cylinder(nx=128, ny=64, D=16, center=(x, 31.7), U=0.05, Re=40, n_marker=48)
        return make_solver(case, ib, init)

    B = Batch(D2Q9, "f32")
    s, other = make(32.3, B.solver), make(90.3, B.solver)
    for t, name in ((s, "own"), (other, "other")):
        t.step(2, record_force=True)
        t.save_checkpoint(tmp_path / name)
    s.load_checkpoint(tmp_path / "other")
    with pytest.raises(capi.IlbmError, match="band"):
        s.step(1, record_force=True)
    s.load_checkpoint(tmp_path / "own")
    s.ib_ready = True  # (its operator is built)
    cid = B.add(s, max_steps=16)
    B.step(3)
    assert B.sync(cid).istep == 5
    B.remove(cid)
    s.load_checkpoint(tmp_path / "other")
    s.ib_ready = True
    B.add(s, max_steps=16)
    with pytest.raises(capi.IlbmError, match="band"):
        B.step(2)
        B.progress()
    other.close()
    B.close()


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("wall,ncase", [(False, 1), (False, 16), (False, 17), (True, 4), (True, 5)])
def test_small_batches_keep_the_single_levels_bits(storage, wall, ncase):
    """Batches on both sides of the cell form's limits (2^16 cells, 2^17 with
    reflecting walls): bit for bit the levels alone."""
    def make():
        return cases.channel_bounce_back(nx=256, ny=128) if wall else cases.taylor_green(64, U0=0.02, tau=0.7)

    B = Batch(D2Q9, storage)
    ids = []
    for _ in range(ncase):
        case, init = make()
        ids.append(B.add(B.solver(case, None, init), max_steps=8))
    B.step(4)
    case, init = make()
    ref = LevelSolver(case, storage)
    ref.set_macro(*init())
    ref.step(5)
    want = ref.get_f()
    for cid in ids:
        np.testing.assert_array_equal(B.sync(cid).get_f(), want)
    ref.close()
    B.close()


def small_sphere(center=(15.2, 14.9, 13.7), rebuild=0, coupling=1):
    case, ib, init = cases.sphere(36, 30, 28, D=8.0, center=center, U=0.04, Re=30.0, coupling=coupling)
    ib.ivc_rebuild_matrix = rebuild
    return case, ib, init


def near_face(coupling):
    return cases.cylinder(nx=80, ny=64, D=12, center=(30.3, 2.4), U=0.05, Re=40, coupling=coupling)


@pytest.mark.parametrize("storage,tol", [("f64", 1e-12), ("f32", 1e-5), ("f16", 1e-4)])
@pytest.mark.parametrize("name,make", [
    ("spheres", lambda: [small_sphere(), small_sphere(rebuild=1), small_sphere(coupling=0)]),
    ("sphere over a periodic face", lambda: [small_sphere(center=(15.2, 2.4, 13.7), coupling=0)]),
    ("cylinders over a periodic face", lambda: [near_face(0), near_face(2)])], ids=lambda x: x if isinstance(x, str) else "")
def test_bodies_match_alone(name, make, storage, tol):
    """3D bodies with each solve, and bands that reach over a periodic face.  The
    2-byte form: a force that differs by one float may flip the rounding of a
    half, 2^-11 of a shifted population, about 3e-5 of the population."""
    members = make()
    B = Batch(members[0][0].lattice, storage)
    ids = [B.add(B.solver(*m), max_steps=16) for m in members]
    B.step(5)
    for cid, (case, ib, init) in zip(ids, make()):
        s = B.sync(cid)
        ref = LevelSolver(case, storage, ib=ib)
        ref.set_macro(*init())
        ref.step(6)
        assert rel_l2(s.get_f(), ref.get_f()) <= tol
        ref.close()
    B.close()
