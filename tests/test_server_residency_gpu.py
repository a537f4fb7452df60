"""Contexts of the proof server under a tight budget: the larger contexts (with
the affine rounds' scratch) cost no circuit its context and no proof its place
in flight that smaller ones would have had."""
import numpy as np
import pytest

from oracle import FR, Oracle

pytestmark = pytest.mark.gpu


class _Sized:
    """a prover, a witness, its proof's wire form, and the bytes of its contexts"""

    def __init__(self, orc, seed, log_m=12):
        from liblightzk_b200 import device, groth16, serve, synth
        self.circ = synth.Circuit(log_m, seed=seed, n_public=1, n_free=16, block=256)
        self.prover = groth16.Prover(self.circ, synth.ProvingKey(self.circ, seed=seed + 1), window_bits=8)
        z = self.circ.witness(seed + 2)
        self.rs = orc.rand_field(FR, 2, np.array([seed], np.uint64))
        self.want = device.to_host(groth16.to_wire(self.prover.prove(z, *self.rs)))
        self.z, self.bytes = device.to_host(z), self.prover.device_bytes()
        self.full = self._context(serve, 64 << 30)
        self.lean = self._context(serve, self.bytes + self.full - 1)
        assert self.lean < self.full

    def _context(self, serve, budget):
        srv = serve.Server(budget, max_inflight=1)
        self.served(srv, srv.add(self.prover))
        size = srv.stats()["device_bytes"] - self.bytes
        srv.close()
        return size

    def submit(self, srv, cid):
        return srv.submit(cid, self.z, *self.rs)

    def check(self, proof):
        from liblightzk_b200 import device, groth16
        assert (device.to_host(groth16.to_wire(device.to_device(proof))) == self.want).all()

    def served(self, srv, cid):
        self.check(srv.wait(self.submit(srv, cid)))


@pytest.fixture(scope="module")
def pair(cuda):
    orc = Oracle()
    return _Sized(orc, 21), _Sized(orc, 31)


def _no_more_memory(on):
    from liblightzk_b200 import _capi
    _capi.lib().lzk_debug_fail_allocations(0 if on else -1)


def _resident(a, b, room, inflight=1):
    """alternating requests of two circuits, the first ones making contexts;
    after that no allocation may be needed"""
    from liblightzk_b200 import serve
    srv = serve.Server(a.bytes + b.bytes + room, max_inflight=inflight)
    ids = [(x, srv.add(x.prover)) for x in (a, b)]
    for x, cid in ids * 2:
        x.served(srv, cid)
    _no_more_memory(True)
    try:
        for x, cid in ids * 3:
            x.served(srv, cid)
    finally:
        _no_more_memory(False)
    size = srv.stats()["device_bytes"] - a.bytes - b.bytes
    assert size <= room
    srv.close()
    return size


def test_two_lean_contexts_stay(pair):
    a, b = pair
    assert _resident(a, b, a.lean + b.lean) == a.lean + b.lean


def test_full_context_beside_a_lean_one(pair):
    a, b = pair
    assert _resident(a, b, a.full + b.lean) == a.full + b.lean


def test_both_full(pair):
    a, b = pair
    assert _resident(a, b, a.full + b.full) == a.full + b.full


def test_as_many_in_flight_as_lean_contexts(pair):
    from liblightzk_b200 import serve
    a, _ = pair
    k = int(a.full // a.lean) + 1         # the full one and k - 1 lean ones do not fit
    room = k * a.lean
    srv = serve.Server(a.bytes + room, max_inflight=k)
    cid = srv.add(a.prover)
    a.served(srv, cid)                    # one request alone, then bursts
    for _ in range(8):
        [a.check(srv.wait(rid)) for rid in [a.submit(srv, cid) for _ in range(6 * k)]]
        if srv.stats()["device_bytes"] - a.bytes == room:
            break
    else:
        pytest.fail("never %d contexts" % k)
    srv.close()


def test_full_contexts_go_first(pair):
    """a circuit added later takes the room of a full context; after that all
    three stay"""
    from liblightzk_b200 import serve
    a, b = pair
    c = _Sized(Oracle(), 41)
    room = max(a.lean + b.lean + c.lean, a.full + b.lean)
    assert room < a.full + b.lean + c.lean
    srv = serve.Server(a.bytes + b.bytes + c.bytes + room, max_inflight=1)
    ids = [(x, srv.add(x.prover)) for x in (a, b)]
    for x, cid in ids:
        x.served(srv, cid)
    assert srv.stats()["device_bytes"] - a.bytes - b.bytes >= a.full + b.lean
    ids.append((c, srv.add(c.prover)))
    for x, cid in ids * 2:
        x.served(srv, cid)
    _no_more_memory(True)
    try:
        for x, cid in ids * 2:
            x.served(srv, cid)
    finally:
        _no_more_memory(False)
    srv.close()

