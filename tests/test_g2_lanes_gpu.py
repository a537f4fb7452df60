"""G2 points over two lanes (Fq2P, csrc/curve.cuh): accumulation, fix-up and
bucket reduction at the shapes where the lane layout changes: sets smaller than
a warp's 16 points, runs of every length, buckets with many partial sums."""
import pytest

from helpers import bases, same_point, scalars

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [2, 3, 4, 5, 6, 7, 9, 11])
@pytest.mark.parametrize("run", [1, 4, 16])
def test_widths_and_runs(cuda, orc, rng_state, c, run):
    from liblightzk_b200 import autotune, device, msm
    n = 150
    s, b = scalars(orc, n, rng_state), bases(orc, 2, n, rng_state)
    b[3:6], b[9] = b[2], 0
    s[20:60] = s[20]          # one bucket a window with many partials
    want = orc.msm(2, s, b)
    old = [autotune.get_value(k, 2, 8) for k in ("run", "chunk")]
    try:
        autotune.set_value("run", 2, 8, run)
        autotune.set_value("chunk", 2, 8, 8)
        got = msm.msm(2, device.to_device(s), device.to_device(b), window_bits=c)
    finally:
        for k, v in zip(("run", "chunk"), old):
            autotune.set_value(k, 2, 8, v)
    assert same_point(orc, 2, device.to_host(got), want)


def test_many_partials(cuda, orc, rng_state):
    from liblightzk_b200 import device, msm
    n = 3000
    s, b = scalars(orc, n, rng_state), bases(orc, 2, n, rng_state)
    s[:] = s[7]
    got = msm.msm(2, device.to_device(s), device.to_device(b), window_bits=13)
    assert same_point(orc, 2, device.to_host(got), orc.msm(2, s, b))


def test_batch_g2(cuda, orc, rng_state):
    from liblightzk_b200 import batch, device
    jobs = []
    for n, c in ((70, 4), (1, 5), (260, 6), (130, 10)):
        jobs.append((scalars(orc, n, rng_state), bases(orc, 2, n, rng_state), device.empty((3, 2, 4)), c))
    plan = batch.BatchPlan(2, msms=[(device.to_device(s), device.to_device(b), o, c) for s, b, o, c in jobs])
    plan.run()
    for s, b, o, _ in jobs:
        assert same_point(orc, 2, device.to_host(o), orc.msm(2, s, b))
    plan.close()
