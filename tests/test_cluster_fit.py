"""Bodies whose forcing takes a cluster launch keep working where the device
refuses the cluster's attributes or cannot hold one: the decision (host code)
against a fake runtime, and the launches a small body takes on this device."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include "cluster_fit.h"
#include <cstdio>
int main() {
  struct { int prepare, query, resident; } fake[] = {{0, 0, 3}, {0, 0, 1}, {0, 0, 0}, {1, 0, 3}, {0, 912, 3}};
  for (auto &f : fake) {
    int cleared = 0, asked = 0;
    int n = ilbm::clusters_resident([&] { return f.prepare; },
                                    [&](int *r) { ++asked; *r = f.resident; return f.query; }, [&] { ++cleared; });
    std::printf("%d%d%d ", n, asked, cleared);
  }
}
"""


def test_refusals_are_no_error(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'ilbmrex_b200' / 'csrc'}", str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    # (clusters, query asked, error cleared)
    assert out == ["310", "110", "010", "001", "011"]


@pytest.mark.gpu
@pytest.mark.parametrize("n,chain", [(64, True), (512, True), (513, False)])
def test_small_bodies_take_the_cluster(n, chain):
    """Explicit coupling: the chain, the cells outside the band and the band are
    three launches; a launch per stage makes it six or more."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ilbmrex_b200 import cases
    from ilbmrex_b200.level import LevelSolver
    case, ib, init = cases.cylinder(nx=96, ny=72, D=30, center=(40.3, 35.6), U=0.05, Re=40, n_marker=n, coupling=0)
    s = LevelSolver(case, "f32", ib=ib)
    s.set_macro(*init())
    s.step(2)
    before = s.ctx.launches()
    s.step(1)
    took = s.ctx.launches() - before
    assert (took == 3) if chain else (took >= 6)
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("q,storage,coupling,D,chain", [
    (19, "f64", 0, 9.0, True), (19, "f64", 1, 10.0, False), (19, "f32", 1, 9.0, True), (19, "f32", 0, 9.0, False),
    (19, "f32", 1, 10.0, False), (27, "f32", 1, 9.0, False), (19, "f16", 1, 9.0, False)])
def test_spheres_that_take_the_cluster(q, storage, coupling, D, chain):
    """3D: up to 256 markers (diameter 9: 254) in FP64, and in D3Q19 FP32 with the
    stored inverse."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ilbmrex_b200 import cases
    from ilbmrex_b200.lattice import D3Q19, D3Q27
    from ilbmrex_b200.level import LevelSolver
    case, ib, init = cases.sphere(36, 30, 28, D=D, center=(15.2, 14.9, 13.7), U=0.04, Re=30.0, coupling=coupling,
                                  lattice=D3Q19 if q == 19 else D3Q27)
    s = LevelSolver(case, storage, ib=ib)
    s.set_macro(*init())
    s.step(2)
    before = s.ctx.launches()
    s.step(1)
    took = s.ctx.launches() - before
    assert (took == 3) if chain else (took >= 6)
    s.close()
