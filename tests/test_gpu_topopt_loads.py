"""The banded displacement solve with loads anywhere in the band order: the forward
substitution comes out of the elimination, so no refinement and no PCG is needed, and
nothing depends on what the device's memory held before."""
import numpy as np
import pytest

import tpt_fem as F
from tpt_fem import topopt as T

pytestmark = pytest.mark.gpu

# A Cholesky solve's residual is bw eps |K| |u| / |f| at most: 1e-10 for these grids.  An
# elimination whose right-hand side is wrong in a percent of an entry leaves 1e-2.
TOL = 1e-8
GRIDS = [(1, 5), (9, 31), (33, 12), (60, 20), (31, 31), (100, 40), (20, 64), (90, 91)]


def _problem(nelx, nely, where, iters=2, density=False):
    g = T.Grid(nelx + 1, nely + 1, 1.0)
    kw = dict(emin=1e-9, density_filter=True) if density else {}
    P = T.TopOptParams(grid=g, vol_frac=0.4, max_iter=iters, **kw)
    f, bcs = T.cantilever_load(g)
    f[:] = 0.0
    if where == "middle":
        f[2 * (g.nx * (g.ny // 2) + g.nx // 2) + 1] = -1.0
    elif where == "top":
        f[2 * (g.nx * (g.ny - 1) + np.arange(g.nx)) + 1] = -1.0 / g.nx
    else:
        f[:] = np.random.default_rng(nelx).uniform(-1.0, 1.0, len(f)) / len(f)
    return P, f, bcs


@pytest.mark.parametrize("where", ["middle", "top", "all"])
@pytest.mark.parametrize("nelx,nely", GRIDS)
def test_no_refinement_wherever_the_load_is(ctx, nelx, nely, where):
    prob = _problem(nelx, nely, where)
    (d,), st = T.topopt_batch(ctx, [prob], rel_tol=TOL)
    assert st["direct_instances"] == 1 and st["not_converged"] == 0
    assert st["refinement_steps"] == 0 and st["pcg_iterations"] == 0
    (p,), _ = T.topopt_batch(ctx, [prob], rel_tol=1e-11, pcg_only=True)
    # |f.(u - v)| <= |f| |K^-1| (|r_u| + |r_v|): TOL times |f|^2 |K^-1| / f.u, which is 2e4 at most for
    # these loads on the uniform start, and five times that for the design after one step
    assert np.allclose(d.compliance, p.compliance, rtol=1e-3, atol=0)


@pytest.mark.parametrize("nelx,nely,density", [(33, 12, True), (60, 20, True), (9, 31, False), (100, 40, False)])
def test_what_ran_before_has_no_effect(ctx, nelx, nely, density):
    prob = _problem(nelx, nely, "all", iters=4, density=density)
    runs = []
    m = F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, [60] * 3, ctx=ctx)
    for fill in (0.0, np.nan, 1e300):
        # device memory full of it, freed to the pool, and other kernels' shared memory
        F.apply_traction(m, 3, 0, 1.0, [0.0, 0.0, 0.0], np.full(3 * m.n_nodes, fill))
        T.topopt_batch(ctx, [_problem(112, 112, "all", iters=1)], rel_tol=1e-3)
        F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, [20] * 3, ctx=ctx)
        (r,), st = T.topopt_batch(ctx, [prob], rel_tol=TOL)
        assert st["pcg_iterations"] == 0 and st["refinement_steps"] == 0
        runs.append(r)
    # and beside a grid whose panels leave room for two chunk buffers only
    res, st = T.topopt_batch(ctx, [_problem(90, 91, "middle", iters=1), prob], rel_tol=TOL)
    assert st["pcg_iterations"] == 0 and st["refinement_steps"] == 0
    runs.append(res[1])
    for r in runs[1:]:
        assert np.array_equal(r.densities, runs[0].densities)
        assert np.array_equal(r.compliance, runs[0].compliance)
