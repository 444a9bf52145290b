"""Contexts in threads of their own: solves and topology batches of different sizes at the same
time give what they give alone (shared-memory limits of kernels are the process's, not a launch's)."""
import threading

import numpy as np
import pytest

import tpt_fem as F
from tpt_fem import topopt as T

pytestmark = pytest.mark.gpu


def _in_threads(jobs, rounds):
    """Every job (context -> result) alone, then all at once in threads, `rounds` times each."""
    errors, alone = [], [job(F.Context(0)) for job in jobs]
    gate = threading.Barrier(len(jobs))

    def work(k):
        try:
            ctx = F.Context(0)
            gate.wait()
            for _ in range(rounds):
                got = jobs[k](ctx)
                if not all(np.array_equal(a, b) for a, b in zip(got, alone[k])):
                    raise AssertionError("job %d differs" % k)
        except Exception as e:  # noqa: BLE001 -- reported by the test
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]


def _solves(n, count):
    def job(ctx):
        mesh = F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, [n] * 3, ctx=ctx)
        K = F.assemble_poisson(mesh, 1.0, 2)
        c = mesh.coords_array
        on = np.nonzero(np.any((c < 1e-9) | (c > 1 - 1e-9), axis=1))[0]
        S = F.reduce_system(K, F.load_poisson_source(mesh, 1.0, 2), [(int(i), 0.0) for i in on])
        for _ in range(count):
            S.solve(tol=1e-2)
        return (S.solution(),)
    return job


@pytest.mark.parametrize("sizes", [(4, 6, 8, 10), (14, 40, 56, 64)])  # one block; a grid of blocks
def test_solves_in_threads(ctx, sizes):
    _in_threads([_solves(n, 60) for n in sizes], 4)


def test_topology_in_threads(ctx):
    def batch(nelx, nely):
        def job(c):
            P = T.TopOptParams(grid=T.Grid(nelx + 1, nely + 1, 1.0), vol_frac=0.4, max_iter=2)
            f, bcs = T.cantilever_load(P.grid)
            (r,), _ = T.topopt_batch(c, [(P, f, bcs)])
            return r.densities, r.compliance
        return job
    _in_threads([batch(6, 2), batch(60, 20), batch(40, 36)], 25)


def _fan(n):  # one node with n + 1 neighbours
    a = np.arange(n) * 2 * np.pi / n
    coords = np.vstack([[0.0, 0.0], np.stack([np.cos(a), np.sin(a)], axis=1)])
    conn = np.stack([np.zeros(n, int), 1 + np.arange(n), 1 + (np.arange(n) + 1) % n], axis=1)

    def job(ctx):
        for _ in range(20):
            out = F.assemble_elasticity(F.Mesh.from_arrays(F.CELL_TRI3, coords, conn, ctx=ctx), "plane-stress", 1.0,
                                        0.3, 2).to_csr()
        return out
    return job


def _field(m):
    rng = np.random.default_rng(m)
    p, w, phi = rng.uniform(size=(50, 3)), rng.standard_normal((3, m)), rng.uniform(size=m)

    def job(ctx):
        for _ in range(40):
            out = F.grf_eval(p, w, phi, 1.0, ctx=ctx)
        return (out,)
    return job


def test_assembly_and_fields_in_threads(ctx):
    _in_threads([_fan(6), _fan(40), _fan(200), _field(8), _field(700), _field(2048)], 8)
