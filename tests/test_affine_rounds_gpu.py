"""The batched affine rounds of the MSM (csrc/affine.cuh) against the oracle:
narrow windows make full buckets out of few points, so every number of rounds
is reached at sizes the oracle does quickly.  The bases repeat (pairs of equal
points), come with their negatives (pairs that cancel) and hold points at
infinity; sizes are no multiples of the rounds' pairs or threads."""
import numpy as np
import pytest

from helpers import bases, same_point, scalars
from oracle import FR

pytestmark = pytest.mark.gpu

Q = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47


def _neg_y(pts):
    out = pts.copy()
    for y in out[:, 1].reshape(-1, 4):
        v = sum(int(l) << (64 * i) for i, l in enumerate(y))
        y[:] = [((Q - v) % Q) >> (64 * i) & (1 << 64) - 1 for i in range(4)]
    return out


def _special_bases(orc, g, n, state, distinct=7):
    pool = bases(orc, g, distinct, state)
    pool = np.concatenate([pool, _neg_y(pool), np.zeros_like(pool[:1])])
    pick = np.random.default_rng(5).integers(0, pool.shape[0], n)
    b = pool[pick]
    b[n // 2:] = bases(orc, g, n - n // 2, state)
    return b


# rounds = entries per bucket: n ceil(255 / c) entries over ceil(255 / c) 2^(c-1)
# buckets for plain bases, 2^(c-1) for a table
@pytest.mark.parametrize("g,n,c", [(1, 701, 2), (1, 1033, 3), (1, 2049, 6), (1, 6001, 9), (2, 701, 2), (2, 1031, 4)])
def test_plain(cuda, orc, rng_state, g, n, c):
    import torch
    from liblightzk_b200 import device, msm
    s, b = scalars(orc, n, rng_state), _special_bases(orc, g, n, rng_state)
    ds, db = device.to_device(s), device.to_device(b)
    want = orc.msm(g, s, b)
    assert same_point(orc, g, device.to_host(msm.msm(g, ds, db, window_bits=c)), want)
    # one byte short of the rounds' scratch: the same sum without them
    ws = torch.empty(msm.workspace_bytes(g, n, c) - 1, dtype=torch.uint8, device="cuda")
    assert same_point(orc, g, device.to_host(msm.msm(g, ds, db, window_bits=c, workspace=ws)), want)


@pytest.mark.parametrize("g,n,c", [(1, 2500, 9), (1, 4097, 7), (2, 2500, 8)])
@pytest.mark.parametrize("kind", ["uniform", "equal", "bits"])
def test_table(cuda, orc, rng_state, g, n, c, kind):
    from liblightzk_b200 import device, msm
    s, b = scalars(orc, n, rng_state), _special_bases(orc, g, n, rng_state)
    if kind == "equal":
        s[:] = s[0]
    elif kind == "bits":
        s[: 2 * n // 3] = orc.to_mont(FR, np.array([[i % 2, 0, 0, 0] for i in range(2 * n // 3)], np.uint64))
    w = msm.windows_for(c)
    table = msm.precompute(g, device.to_device(b), c)
    got = msm.msm_precomputed(g, device.to_device(s), table, c, w, n)
    assert same_point(orc, g, device.to_host(got), orc.msm(g, s, b))


@pytest.mark.parametrize("fixed", [False, True])
def test_batch(cuda, orc, rng_state, fixed):
    import torch
    from liblightzk_b200 import batch, device
    jobs = []
    for n, c in ((900, 3), (1500, 5), (1, 4), (2200, 8)):
        s, b = scalars(orc, n, rng_state), _special_bases(orc, 1, n, rng_state)
        jobs.append((s, b, device.empty((3, 4)), c))
    plan = batch.BatchPlan(1, msms=[(device.to_device(s), device.to_device(b), o, c) for s, b, o, c in jobs],
                           fixed_bases=fixed)
    st = torch.cuda.Stream()
    for _ in range(2):
        plan.run(use_graph=True, stream=st)
    st.synchronize()
    for s, b, o, _ in jobs:
        assert same_point(orc, 1, device.to_host(o), orc.msm(1, s, b))
    plan.close()


def test_server_without_room_for_the_rounds(cuda, orc, rng_state):
    """budgets that a context (or a prover) with the rounds' scratch exceeds
    are still served, without the rounds"""
    from liblightzk_b200 import device, groth16, serve, synth
    circ = synth.Circuit(12, seed=3, n_public=1, n_free=16, block=256)
    prover = groth16.Prover(circ, synth.ProvingKey(circ, seed=4), window_bits=8)
    z = circ.witness(5)
    r, s = orc.rand_field(FR, 2, rng_state)
    want = device.to_host(groth16.to_wire(prover.prove(z, r, s)))
    zh, rb = device.to_host(z), prover.device_bytes()
    sizes = []
    for budget in (64 << 30, None, rb - 1):
        if budget is None:
            budget = rb + sizes[0] - 1
        srv = serve.Server(budget, max_inflight=1)
        cid = srv.add(prover)
        got = srv.wait(srv.submit(cid, zh, r, s))
        sizes.append(srv.stats()["device_bytes"] - prover.device_bytes())
        assert srv.stats()["device_bytes"] <= budget
        srv.close()
        assert (device.to_host(groth16.to_wire(device.to_device(got))) == want).all()
    assert sizes[1] < sizes[0] and prover.device_bytes() < rb
    assert (device.to_host(groth16.to_wire(prover.prove(z, r, s))) == want).all()
