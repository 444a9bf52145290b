"""Right-hand sides that are not finite, or whose squares are not: the same error whether the
solve is one launch or the engine's kernels."""
import numpy as np
import pytest

import tpt_fem as F

pytestmark = pytest.mark.gpu


# Poisson cubes: one block, a grid of blocks, the engine (past the row limits)
@pytest.mark.parametrize("n", [6, 20, 75])
@pytest.mark.parametrize("value,error", [(np.inf, "BREAKDOWN"), (-np.inf, "BREAKDOWN"), (np.nan, "BREAKDOWN"),
                                         (1e200, "NOT_CONVERGED")])
@pytest.mark.parametrize("kw", [dict(solver=F.SOLVER_JACOBI_PCG), dict(solver=F.SOLVER_FSAI_MP_PCG),
                                dict(solver=F.SOLVER_FSAI_MP_PCG, coarse=True)])
def test_right_hand_side_out_of_range(ctx, n, value, error, kw):
    mesh = F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, [n] * 3, ctx=ctx)
    K = F.assemble_poisson(mesh, 1.0, 2)
    left = np.nonzero(mesh.coords_array[:, 0] < 1e-9)[0]
    rhs = np.ones(K.nrows)
    rhs[-1] = value
    S = F.reduce_system(K, rhs, [(int(i), 0.0) for i in left])
    with pytest.raises(F.TptFemError) as e:
        S.solve(tol=1e-10, max_iter=50, **kw)
    assert e.value.name == error
