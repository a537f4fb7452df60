"""Transforms of 2^2 to 2^8 elements in one block (csrc/ntt.cu, k_ntt_short):
with the reference's tables and factor, through a batch plan's pointers, and
that they are not slower than their stages account for."""
import pytest

from oracle import FR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", range(1, 10))
def test_reference_table(cuda, orc, rng_state, k):
    from liblightzk_b200 import device, ntt
    n = 1 << k
    tab, a = orc.ntt_setup(n), orc.rand_field(FR, n, rng_state)
    dt, x = device.to_device(tab), device.to_device(a)
    ntt.number_theory_transformation(n, k, x, dt[n:2 * n], dt[2 * n:2 * n + 1])
    assert (device.to_host(x) == orc.ntt_ref(a, tab[n:2 * n], tab[2 * n])).all()


@pytest.mark.parametrize("d", range(4))
def test_batch_plan(cuda, orc, rng_state, d):
    from liblightzk_b200 import batch, device
    vecs = [(k, orc.rand_field(FR, 1 << k, rng_state)) for k in (2, 5, 6, 7, 7, 7, 8, 8, 9)]
    ntts = [(device.to_device(a), k, d) for k, a in vecs]
    plan = batch.BatchPlan(1, ntts=ntts)
    plan.run()
    for (k, a), (x, _, _) in zip(vecs, ntts):
        assert (device.to_host(x) == orc.ntt(a, k, d)).all(), k
    plan.close()


def _graph_us(k, d, calls=64):
    """device time of a transform in a captured chain of them"""
    import torch
    from liblightzk_b200 import ntt, synth
    x = synth.random_fr(1 << k, 5, 5)
    ntt.ntt(x, k, d)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _ in range(calls):
            ntt.ntt(x, k, d)
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        g.replay()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best * 1000 / calls


@pytest.mark.parametrize("d", [0, 1, 2, 3])
def test_short_against_longer(cuda, d):
    # the passes, which 2^9 takes, have about 0.75 of its time at 2^6
    assert _graph_us(6, d) < 0.6 * _graph_us(9, d)
