"""SpMV rows longer than a thread takes at once (csrc/spmv.cu): lengths around
the line, few and many in a block, more than a block keeps for its end, and
the time of one beside the same entries in short rows.  Bit-exact against the
oracle."""
import numpy as np
import pytest

from oracle import FR

pytestmark = pytest.mark.gpu


def _lengths(kind, rng):
    if kind == "edges":
        return np.array([0, 63, 64, 65, 66, 95, 96, 97, 1, 0, 127, 128, 129, 1000, 0, 2, 64, 65])
    if kind == "last":                       # the last row runs to nnz
        return np.array([1] * 300 + [700])
    if kind == "one":
        return np.array([5000])
    if kind == "few":                        # the warps of a block share them
        per = rng.integers(0, 3, 600)
        per[[0, 31, 32, 255, 256, 599]] = [65, 300, 70, 2000, 90, 100]
        return per
    if kind == "all":                        # every thread keeps its own
        return rng.integers(65, 90, 700)
    per = rng.integers(0, 2, 148 * 8 * 256 + 700)     # two rows a thread of the first blocks
    per[:300] = rng.integers(60, 75, 300)
    per[-300:] = rng.integers(60, 75, 300)
    return per


@pytest.mark.parametrize("kind", ["edges", "last", "one", "few", "all", "two a thread"])
@pytest.mark.parametrize("index", [np.uint32, np.uint64])
def test_long_rows(cuda, orc, rng_state, kind, index):
    from liblightzk_b200 import device, ntt
    rng = np.random.default_rng(7)
    per = _lengths(kind, rng)
    rows, cols, nnz = len(per), 50, int(per.sum())
    ptr = np.concatenate([[0], np.cumsum(per)[:-1]])
    col, val = rng.integers(0, cols, nnz), orc.rand_field(FR, nnz, rng_state)
    val[::3] = orc.to_mont(FR, np.array([[1, 0, 0, 0]], np.uint64))[0]
    z = orc.rand_field(FR, cols, rng_state)
    t = [device.to_device(x) for x in (val, col.astype(index), ptr.astype(index), np.full((rows, 4), 7, np.uint64))]
    m = ntt.csr(t[0], t[1], t[2], rows, cols, nnz)
    other = device.to_device(np.full((rows, 4), 7, np.uint64))
    ntt.spmv3(m, None, m, device.to_device(z), t[3], None, other)
    want = orc.spmv(val, col.astype(np.uint64), ptr.astype(np.uint64), z)
    assert (device.to_host(t[3]) == want).all() and (device.to_host(other) == want).all()


def test_long_row_time(cuda):
    import torch
    from liblightzk_b200 import device, ntt, synth
    nnz = 8192
    val, z = synth.random_fr(nnz, 1, 1), synth.random_fr(1000, 1, 2)
    col = device.to_device(np.random.default_rng(1).integers(0, 1000, nnz).astype(np.uint32))

    def us(rows, calls=20):
        ptr = device.to_device((np.arange(rows) * (nnz // rows)).astype(np.uint32))
        out = device.empty((rows, 4))
        m = ntt.csr(val, col, ptr, rows, 1000, nnz)
        ntt.spmv3(m, None, None, z, out, None, None)
        torch.cuda.synchronize()
        g, best = torch.cuda.CUDAGraph(), float("inf")
        with torch.cuda.graph(g):
            for _ in range(calls):
                ntt.spmv3(m, None, None, z, out, None, None)
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best * 1000 / calls

    # 8192 / 32 steps of a warp against 64 of a thread
    assert us(1) < 16 * us(128)
