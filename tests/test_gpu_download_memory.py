"""Downloads of any size go through a few pinned chunks: the process does not grow with them."""
import numpy as np
import pytest

import tpt_fem as F

pytestmark = pytest.mark.gpu


def _mapped_bytes():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[0]) * 4096


def test_download_memory_does_not_grow_with_the_matrix(ctx):
    def matrix(n):
        m = F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, [n] * 3, ctx=ctx)
        return F.assemble_elasticity(m, "3d", 1.0, 0.3, 2)

    big, small = matrix(72), matrix(16)
    small.to_csr()  # threads and the ring exist from here on
    before = _mapped_bytes()
    rp, ci, va = big.to_csr()
    staged = 12 * big.nnz  # int32 columns and values as they cross
    arrays = rp.nbytes + ci.nbytes + va.nbytes
    assert staged > 400 << 20
    assert _mapped_bytes() - before - arrays < 100 << 20
    assert rp[-1] == big.nnz


@pytest.mark.parametrize("n", [[9, 9, 8], [31, 17, 5], [40, 40, 33]])
def test_chunked_download_is_the_matrix(ctx, n):
    # arrays of less than a chunk, of one and a piece, and of more than the ring's
    m = F.Mesh.box_mesh([0.0] * 3, [1.0] * 3, n, ctx=ctx)
    K = F.assemble_elasticity(m, "3d", np.random.default_rng(1).uniform(0.5, 1.0, m.n_elems), 0.3, 2)
    rp, ci, va = K.to_csr()
    x = np.random.default_rng(2).standard_normal(K.nrows)
    y = np.add.reduceat(va * x[ci], rp[:-1])  # every entry counts
    ref = K.matvec(x)
    assert rp[0] == 0 and rp[-1] == K.nnz == len(ci)
    assert np.max(np.abs(y - ref)) <= 1e-13 * np.max(np.abs(ref)) * 60
