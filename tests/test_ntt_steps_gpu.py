"""The radix-4 passes (csrc/ntt.cu) where their steps change: one- and
two-element transforms, one block (natural order written by the pass itself),
odd and even stage counts in first and later passes, element-wise and tiled bit
reversal, several vectors at a stride that leaves gaps."""
import pytest

from oracle import FR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [0, 1, 2, 3, 4, 8, 9, 10, 11, 13, 17])
@pytest.mark.parametrize("block", [256, 1024, 4096])
def test_directions(cuda, orc, rng_state, k, block):
    from liblightzk_b200 import autotune, device, ntt
    n, stride, count = 1 << k, (1 << k) + 3, 3
    a = orc.rand_field(FR, count * stride, rng_state)
    a[:: 5] = 0
    try:
        autotune.set_value("ntt", 0, k, block)
        for d in range(4):
            x = device.to_device(a.copy())
            ntt.ntt_batch(x, k, count, stride, d)
            got = device.to_host(x)
            for i in range(count):
                at = slice(i * stride, i * stride + n)
                assert (got[at] == orc.ntt(a[at], k, d)).all(), (d, i)
                assert (got[i * stride + n:(i + 1) * stride] == a[i * stride + n:(i + 1) * stride]).all()
    finally:
        autotune.set_value("ntt", 0, k, 0)
