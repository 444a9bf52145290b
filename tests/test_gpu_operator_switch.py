"""Jacobi-PCG with new values under another operator than the last solve's: each operator's
preconditioner is the new matrix's, as for a system reduced from it."""
import numpy as np
import pytest

import tpt_fem as F

pytestmark = pytest.mark.gpu


def _system(K, mesh):
    left = np.nonzero(mesh.coords_array[:, 0] < 1e-9)[0]
    rhs = F.load_body(mesh, [0.0, 0.0, -1e-2], 2)
    return rhs, F.reduce_system(K, rhs, [(3 * int(i) + c, 0.0) for i in left for c in range(3)])


@pytest.mark.parametrize("first,between", [(dict(full_operator=True), {}), ({}, dict(full_operator=True)),
                                           (dict(full_operator=True), dict(csr_only=True)),
                                           (dict(csr_only=True), {})])
def test_new_values_reach_every_operator(ctx, first, between):
    mesh = F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, [12] * 3, ctx=ctx)
    E = np.exp(2.0 * np.random.default_rng(3).standard_normal(mesh.n_elems))
    K = F.assemble_elasticity(mesh, "3d", 1.0, 0.3, 2)
    rhs, S = _system(K, mesh)
    S.solve(tol=1e-8, **first)
    K.reassemble(E)
    S.refresh(K, rhs)
    S.solve(tol=1e-8, **between)
    got = S.solve(tol=1e-8, **first)
    _, new = _system(K, mesh)
    ref = new.solve(tol=1e-8, **first)
    assert got["iterations"] == ref["iterations"]
    assert np.array_equal(S.solution(), new.solution())


def test_non_positive_diagonal_is_found_under_every_operator(ctx):
    mesh = F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, [12] * 3, ctx=ctx)
    K = F.assemble_elasticity(mesh, "3d", 1.0, 0.3, 2)
    rhs, S = _system(K, mesh)
    S.solve(tol=1e-8, full_operator=True)
    K.reassemble(-1.0)
    S.refresh(K, rhs)
    for kw in ({}, dict(full_operator=True), dict(csr_only=True)):
        with pytest.raises(F.TptFemError) as e:
            S.solve(tol=1e-8, **kw)
        assert "diagonal" in str(e.value)
