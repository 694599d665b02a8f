"""The resident Poisson kernels by plan: every brick width and plane class of the brick kernels,
launches of all 148 SMs among them, and the column tiles on grids that only they fit, each
against the streaming kernels on the same system; the one-sweep CG with ragged tiles against
numpy.  Which plan a shape gets is checked on the CPU (test_plans_cpu.py).  Bounds as in
test_gpu_brick.py: 30 CG iterations to 1e-10 of the pressure's norm, mixed to 1e-4, FP64 RB-SOR
the same bits, mixed to 1e-5."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import rel_l2
from test_gpu_brick import numpy_cg, solve, system

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# shape: brick width, planes per brick, CTAs
BRICKS = {
    (13, 119, 73): (16, 2, 148), (53, 25, 147): (32, 4, 148), (128, 16, 256): (32, 7, 148),
    (11, 122, 177): (16, 5, 144), (43, 130, 93): (16, 11, 135), (33, 97, 194): (16, 17, 144),
    (62, 94, 209): (32, 18, 144), (47, 191, 250): (16, 32, 144),
    (62, 55, 82): (64, 4, 147), (33, 33, 123): (64, 5, 125), (34, 33, 240): (64, 9, 135),
    (191, 55, 110): (64, 16, 147),
}
# shape: rows of a column tile
COLUMNS = {(205, 168, 37): 16, (232, 71, 112): 8, (123, 68, 236): 4}
# (shape, precision) of the one-sweep CG: tiles of 128 and of 32, ragged in x, y and z chunks
SWEEPS = [((250, 300, 60), 0), ((472, 122, 120), 0), ((158, 43, 784), 0), ((290, 63, 333), 0),
          ((220, 220, 220), 1), ((252, 203, 180), 1)]

name = "x".join
ids = [name(map(str, s)) for s in BRICKS] + [name(map(str, s)) + "-columns" for s in COLUMNS]


def check_plan(af, shape):
    s = af.FluidSolver3D(*shape)
    plan = s.poisson_plan()
    s.close()
    assert plan["resident"]
    if shape in COLUMNS:
        assert plan["tile"][1] == COLUMNS[shape]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [*BRICKS, *COLUMNS], ids=ids)
def test_resident_cg_matches_streaming(af, shape, precision):
    check_plan(af, shape)
    b, p0 = system(shape, 15, False)
    knobs = dict(precision=1, mixed_inner_iters=15, mixed_max_refinements=2) if precision else {}
    ref, ri = solve(af, shape, 1, b, p0, 30, **knobs)
    got, gi = solve(af, shape, 0, b, p0, 30, **knobs)
    assert (gi.iterations, gi.refinements) == (ri.iterations, ri.refinements)
    assert rel_l2(got, ref) <= (1e-4 if precision else 1e-10)
    if precision:
        assert abs(gi.final_residual - ri.final_residual) <= 1e-2 * ri.final_residual
    else:
        assert abs(gi.final_residual - ri.final_residual) <= 1e-9 * ri.rhs_norm


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [*BRICKS, *COLUMNS], ids=ids)
def test_resident_sor_matches_streaming(af, shape, precision):
    b, p0 = system(shape, 19, True)
    out = []
    for kernel in (1, 2):  # AUTO streams FP64 RB-SOR on grids that fit no bricks
        s = af.FluidSolver3D(*shape, precision=precision, poisson_kernel=kernel)
        s.set_params(solver_kind=1, sor_omega=1.7)
        s.set_field("divergence", b)
        s.set_field("pressure", p0)
        assert s.solve_poisson_gauss_seidel(9).iterations == 9
        out.append(s.get_field("pressure"))
        s.close()
    if precision == 0:
        assert np.array_equal(out[0], out[1])
    else:
        assert rel_l2(out[1], out[0]) <= 1e-5


@pytest.mark.parametrize("iters", [4, 5])
@pytest.mark.parametrize("shape,precision", SWEEPS,
                         ids=[name(map(str, s)) + ("-mixed" if p else "") for s, p in SWEEPS])
def test_ragged_sweep_matches_numpy(af, shape, precision, iters):
    b, p0 = system(shape, 21, False)
    got, info = solve(af, shape, 1, b, p0, iters, precision=precision, mixed_max_refinements=1)
    want, res = numpy_cg(shape, b, p0, iters)
    assert info.iterations == iters
    inner = got.reshape(shape[::-1])[1:-1, 1:-1, 1:-1]
    assert rel_l2(inner.ravel(), want.ravel()) <= (1e-4 if precision else 1e-10)
    assert abs(info.final_residual - res) <= (1e-3 if precision else 1e-9) * res


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [(64, 64, 75), *COLUMNS, (160, 160, 161)],
                         ids=["bricks", "columns16", "columns8", "columns4", "sweep"])
def test_right_hand_side_on_the_walls_matches_oracle(af, oracle, shape, precision):
    """Three iterations on a right-hand side of the caller's own that is not 0 on two walls,
    which the operator neither reads nor changes."""
    nx, ny, nz = shape
    b, p0 = system(shape, 25, False)
    b = b.reshape(nz, ny, nx)
    b[0], b[:, :, -1] = 0.01, -0.02
    o = oracle.OracleSolver(*shape)
    o.field("divergence")[:] = b.ravel()
    o.field("pressure")[:] = p0
    assert o.solve_poisson_conjugate_gradient(3) == 3
    got, info = solve(af, shape, 0, b.ravel(), p0, 3, precision=precision,
                      mixed_max_refinements=1)
    assert info.iterations == 3
    assert rel_l2(got, np.array(o.field("pressure"))) <= (1e-4 if precision else 1e-10)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [(40, 20, 18), (205, 168, 37), (160, 160, 161)],
                         ids=["bricks", "columns", "sweep"])
def test_pressure_untouched_by_a_nan_on_a_wall(af, shape, precision):
    """A right-hand side that is NaN, or infinite with no iterations to do, on a wall cell
    stops the solve before its first step: the pressure stays as it was, the NaN is reported."""
    b, p0 = system(shape, 23, False)
    for bad, iters in ((np.nan, 5), (np.inf, 0)):
        if precision and iters == 0:
            continue  # the mixed form does one iteration at least
        s = af.FluidSolver3D(*shape, precision=precision, mixed_max_refinements=1)
        s.set_field("divergence", np.concatenate(([bad], b[1:])))
        s.set_field("pressure", p0)
        with pytest.raises(af.AetherFluidError):
            s.solve_poisson_conjugate_gradient(iters)
        assert np.array_equal(s.get_field("pressure"), p0)
        s.close()


# every kernel with waits of its own: its shape, precision and solver
WAITS = {"mixed bricks": ((64, 64, 64), 1, "conjugate_gradient"),
         "sor bricks": ((64, 64, 64), 0, "gauss_seidel"),
         "mixed sor bricks": ((64, 64, 64), 1, "gauss_seidel"),
         "columns": ((123, 68, 236), 0, "conjugate_gradient"),
         "sweep": ((250, 300, 60), 0, "conjugate_gradient"),
         "mixed sweep": ((252, 203, 180), 1, "conjugate_gradient")}


@pytest.mark.parametrize("kernel", list(WAITS))
def test_wait_limit_is_reported_not_hung(af, kernel):
    """A wait limit of 0 ns, set by the host: the first wait that is not already over gives up,
    the solve returns AFL_ERR_TIMEOUT, and the context stays usable."""
    shape, precision, solver = WAITS[kernel]
    code = f"""
import os, sys
sys.path.insert(0, os.path.join(sys.argv[1], "aether-core-engine_b200"))
os.environ["AFL_BARRIER_TIMEOUT_NS"] = "0"
import aether_fluid as af, numpy as np
s = af.FluidSolver3D(*{shape}, precision={precision})
s.set_field("divergence", np.random.default_rng(0).standard_normal(s.n))
try:
    s.solve_poisson_{solver}(50)
    print("NO-ERROR")
except af.AetherFluidError as e:
    print("STATUS", e.status)
os.environ.pop("AFL_BARRIER_TIMEOUT_NS")
t = af.FluidSolver3D(16, 20, 16)
print("STEP-OK", t.step(0.08, 0.2).kinetic_energy > 0)
"""
    out = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True,
                         timeout=120)
    assert "STATUS 5" in out.stdout, out.stdout + out.stderr
    assert "STEP-OK True" in out.stdout, out.stdout + out.stderr
