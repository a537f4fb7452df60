"""Persistent plans over tables with enough points (2^15) take widths and a
chunk of their own (csrc/batch.cu, persistent_window): the sums of MSMs on both
sides of each line, and just below and at the plan size where the rule begins."""
import pytest

from helpers import bases, same_point, scalars

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("sizes", [[1024, 1025, 2048, 2049, 8192, 8193, 1, 300], [16384, 16383], [16384, 16384]])
def test_sums(cuda, orc, rng_state, group, sizes):
    from liblightzk_b200 import batch, device
    total = sum(sizes)
    s, b = scalars(orc, total, rng_state), bases(orc, group, min(total, 4096), rng_state)
    b = b[[i % len(b) for i in range(total)]]
    ds, db = device.to_device(s), device.to_device(b)
    msms, at = [], 0
    for n in sizes:
        msms.append((ds[at:at + n], db[at:at + n], device.empty((3, 4) if group == 1 else (3, 2, 4))))
        at += n
    plan = batch.BatchPlan(group, msms=msms, fixed_bases=True, persistent=True)
    plan.run()
    at = 0
    for n, (_, _, out) in zip(sizes, msms):
        assert same_point(orc, group, device.to_host(out), orc.msm(group, s[at:at + n], b[at:at + n])), n
        at += n
    plan.close()
