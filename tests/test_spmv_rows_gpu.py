"""SpMV rows and descriptors at their edges: row counts around a block and
above one grid of threads, the three outputs with descriptors that differ in
index width and length, and the largest operands.  Bit-exact against the
oracle's restatement of batch_sparse_matrix_vector_multiplication
(include/operator/poly.cuh:5-30)."""
import numpy as np
import pytest

from helpers import R_MINUS_1_CANON
from oracle import FR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 255, 256, 257, 148 * 8 * 256 + 3])
def test_spmv_row_counts_and_extremes(cuda, orc, rng_state, rows):
    from liblightzk_b200 import device, ntt
    rng = np.random.default_rng(rows)
    cols = 50
    top = np.array([R_MINUS_1_CANON], np.uint64)
    one = orc.to_mont(FR, np.array([[1, 0, 0, 0]], np.uint64))[0]
    z = orc.rand_field(FR, cols, rng_state)
    z[::5], z[1] = top[0], 0
    descs, outs, expect, keep = [], [], [], []
    for k, index in enumerate((np.uint32, np.uint64, np.uint32)):
        n = max(1, rows - 7 * k)
        per = rng.integers(0, 4, n)
        ptr, nnz = np.concatenate([[0], np.cumsum(per)[:-1]]), int(per.sum())
        col = rng.integers(0, cols, nnz)
        val = orc.rand_field(FR, max(nnz, 1), rng_state)[:nnz]
        val[::4], val[1::4], val[2::16] = one, top[0], 0
        t = [device.to_device(x) for x in (val, col.astype(index), ptr.astype(index), np.full((n, 4), 7, np.uint64))]
        keep.append(t)
        descs.append(ntt.csr(t[0], t[1], t[2], n, cols, nnz))
        outs.append(t[3])
        expect.append(orc.spmv(val, col.astype(np.uint64), ptr.astype(np.uint64), z))
    ntt.spmv3(*descs, device.to_device(z), *outs)
    for o, e in zip(outs, expect):
        assert (device.to_host(o) == e).all()
