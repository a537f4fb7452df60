"""The divstep inverse (csrc/inverse.cuh) against Python's modular inverse:
element limbs x stand for x / R, so the inverse's limbs are R^2 / x mod p.
Powers of two and their negatives make the longest runs of even and of odd
steps; batches that are no multiple of a warp mix them with random values."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = {0: 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001,
     1: 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47}


@pytest.mark.parametrize("field", [0, 1], ids=["fr", "fq"])
@pytest.mark.parametrize("extra", [0, 1, 1000])
def test_inverse_values(cuda, field, extra):
    from liblightzk_b200 import device
    from liblightzk_b200.field import INV, field_op
    p, rng = P[field], random.Random(field + 2 * extra)
    xs = [0, 1, 2, 3, p - 1, p - 2, (p - 1) // 2, (p + 1) // 2]
    xs += [1 << i for i in range(254)] + [p - (1 << i) for i in range(253)]
    xs = [x for x in xs if x < p] + [rng.randrange(p) for _ in range(extra)]
    a = np.array([[x >> (64 * j) & (1 << 64) - 1 for j in range(4)] for x in xs], np.uint64)
    got = device.to_host(field_op(field, INV, device.to_device(a)))
    r2 = pow(2, 512, p)
    want = [pow(x, -1, p) * r2 % p if x else 0 for x in xs]
    assert [sum(int(l) << (64 * j) for j, l in enumerate(row)) for row in got] == want
