"""The plans of the Poisson kernels on a chip of 148 SMs, 227 KB of shared memory per CTA and
126 MiB of L2.  Which grids beyond the chip take the one-sweep streaming CG
(csrc/afl_sweep_plan.h): those on which it measured faster than two passes, and none of those
on which mostly empty tiles or idle CTAs made it slower.  Which bricks a grid on the chip gets
(csrc/afl_brick.cuh): those that the GPU tests name for it."""
import subprocess

import pytest

from test_gpu_brick_plans import BRICKS, COLUMNS, SWEEPS

CODE = r"""
#include "afl_brick.cuh"
#include "afl_sweep_plan.h"
#include <cstdio>
#include <cstdlib>
using namespace afl;
int main(int argc, char **v) {
  for (int q = 1; q + 3 < argc; q += 4) {
    Dims g{};
    g.nx = atoi(v[q]), g.ny = atoi(v[q + 1]), g.nz = atoi(v[q + 2]);
    g.nxy = g.nx * g.ny, g.n = g.nxy * g.nz;
    if (atoi(v[q + 3]) == 2) {
      BrickPlan p{};
      if (plan_brick_on(g, 148, 227 << 10, &p)) printf("%d,%d,%d\n", p.bx, p.cz, p.ctas());
      else puts("none");
      continue;
    }
    const bool f64 = atoi(v[q + 3]) == 0;
    const int nc = sweep_wide(g) || !f64 ? 4 : 1, ctas = f64 && nc == 4 ? 148 : 296;
    const SweepPlan pl = sweep_plan(g, nc, ctas);
    long long planes = 0;  // the chunks cover the grid, each with at least one plane
    for (int c = 0; c < pl.chunks; ++c) {
      const int left = g.nz - c * pl.depth;
      if (left < 1) return 1;
      planes += left < pl.depth ? left : pl.depth;
    }
    if (planes != g.nz || pl.tiles_x * 32 * nc < g.nx || pl.tiles_y * kSweepRows < g.ny) return 1;
    printf("%d\n", sweep_fits(g, f64, size_t(126) << 20) && sweep_pays(g, pl, nc, ctas, f64));
  }
}
"""

FASTER = {  # precision: shapes on which the sweep measured faster
    0: [(256, 256, 256), (220, 220, 220), (160, 160, 161), (250, 300, 60), (512, 34, 400),
        (1000, 1000, 8), (1024, 1024, 12), (320, 16, 1200), (96, 250, 300), (64, 300, 400),
        (158, 43, 784), (290, 63, 333), (384, 384, 48), (4096, 2048, 6), (150, 300, 300)],
    1: [(256, 256, 256), (220, 220, 220), (252, 203, 180), (1024, 16, 700), (124, 400, 300),
        (384, 384, 80), (108, 69, 1876), (4096, 2048, 6), (256, 200, 256)],
}
SLOWER = {
    0: [(6, 1200, 1200), (20, 600, 600), (34, 500, 500), (256, 17, 1600), (512, 18, 600),
        (2048, 20, 160), (7100, 6, 531), (324, 566, 41), (420, 368, 25), (128, 7, 6836),
        (136, 136, 400), (144, 323, 78), (44, 156, 701), (6, 399179, 9), (530, 38, 730)],
    1: [(256, 17, 3000), (512, 18, 1200), (512, 34, 800), (2048, 20, 320), (932, 17, 784),
        (480, 3618, 6), (5588, 113, 16), (168308, 6, 25), (1052, 97, 87), (55568, 68, 6)],
}


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    from aether_fluid import build
    d = tmp_path_factory.mktemp("sweep")
    src, exe = d / "t.cu", d / "t"
    src.write_text(CODE)
    subprocess.check_call([build.nvcc(), *build.ARCH, "-std=c++17", "-O1",
                           "--expt-relaxed-constexpr", "-extended-lambda", "-I", build.CSRC,
                           str(src), "-o", str(exe)])

    def run(shapes, precision):
        args = [str(x) for s in shapes for x in (*s, precision)]
        out = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=60)
        assert out.returncode == 0, out.stdout
        words = out.stdout.split()
        return dict(zip(shapes, words if precision == 2 else (w == "1" for w in words)))
    return run


@pytest.mark.parametrize("precision", [0, 1])
def test_sweep_where_it_is_faster(plans, precision):
    got = plans(FASTER[precision], precision)
    assert all(got.values()), got


@pytest.mark.parametrize("precision", [0, 1])
def test_two_passes_where_the_sweep_is_slower(plans, precision):
    got = plans(SLOWER[precision], precision)
    assert not any(got.values()), got


def test_brick_plans_of_the_gpu_tests(plans):
    assert plans(list(BRICKS), 2) == {s: "%d,%d,%d" % p for s, p in BRICKS.items()}
    assert set(plans(list(COLUMNS), 2).values()) == {"none"}
    reached = {(bx, next(c for c in (4, 8, 16, 32) if cz <= c)) for bx, cz, _ in BRICKS.values()}
    assert reached >= {(bx, c) for bx in (16, 64) for c in (4, 8, 16, 32) if (bx, c) != (64, 32)}
    assert any(ctas == 148 for _, _, ctas in BRICKS.values())


@pytest.mark.parametrize("precision", [0, 1])
def test_sweeps_of_the_gpu_tests(plans, precision):
    got = plans([s for s, p in SWEEPS if p == precision], precision)
    assert got and all(got.values()), got
