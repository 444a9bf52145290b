"""The banded elimination's pivot reciprocal (csrc/pivot_rcp.cuh) over its whole range, and
what becomes of pivots outside of it."""
import os

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

KERNEL = """
extern "C" __global__ void rcp(const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = tptfem::td_rcp(x[i]);
}
"""


def test_pivot_reciprocal():
    import torch
    with open(os.path.join(ROOT, "tpt-fem_b200", "csrc", "pivot_rcp.cuh")) as f:
        source = f.read().replace("#pragma once", "")
    kernel = torch.cuda._compile_kernel(source + KERNEL, "rcp")
    rng = np.random.default_rng(1)
    x = np.ldexp(rng.uniform(1.0, 2.0, 400000), rng.integers(-1021, 1021, 400000))
    powers = 2.0 ** np.arange(-1020.0, 1021.0)
    x = np.concatenate([x, powers, np.nextafter(powers, 0.0), np.nextafter(powers, np.inf), [2.0 ** -1021, 2.0 ** 1021]])
    d, y = torch.from_numpy(x).cuda(), torch.empty(len(x), dtype=torch.float64, device="cuda")
    kernel(((len(x) + 255) // 256, 1, 1), (256, 1, 1), (d, y, len(x)))
    # 2 - x r and the last product are rounded once each, to half a unit of 2^-52; the
    # approximation's 2^-20 is squared twice
    err = np.abs(y.cpu().numpy().astype(np.longdouble) * x - 1)
    assert np.max(err) <= 2.0 ** -52 * (1 + 2.0 ** -10)


def test_pivots_out_of_range_leave_the_solve_to_pcg(ctx):
    from tpt_fem import topopt as T
    g = T.Grid(21, 9, 1.0)
    runs = []
    for k in (0, 1022):  # moduli 2^k and loads 2^(k / 2): the same optimisation, compliances too
        P = T.TopOptParams(grid=g, e0=2.0 ** k, vol_frac=1.0, max_iter=4)
        f, bcs = T.cantilever_load(g, 2.0 ** (k // 2))
        (r,), st = T.topopt_batch(ctx, [(P, f, bcs)], rel_tol=1e-10)
        assert st["direct_instances"] == 1 and st["not_converged"] == 0 and st["refinement_steps"] == 0
        assert (st["pcg_iterations"] > 0) == (k > 0)
        runs.append(r)
    # compliances of two solutions to 1e-10, conditioned by at most 1e4
    assert np.allclose(runs[0].compliance, runs[1].compliance, rtol=1e-6, atol=0)
    assert np.max(np.abs(runs[0].densities - runs[1].densities)) <= 1e-6
