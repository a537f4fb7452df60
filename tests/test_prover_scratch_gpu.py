"""A server that makes a prover's own scratch lean to fit its budget: with
little device memory free, with none to be had for a while, and beside threads
that read the prover's size and prove with it."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from oracle import FR, Oracle

pytestmark = pytest.mark.gpu

MARGIN = 48 << 20
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _prover(log_m, window):
    from liblightzk_b200 import groth16, synth
    circ = synth.Circuit(log_m, seed=3, n_public=1, n_free=16, block=256)
    return circ, groth16.Prover(circ, synth.ProvingKey(circ, seed=4), window_bits=window)


def _wire(prover, z, r, s):
    from liblightzk_b200 import device, groth16
    return device.to_host(groth16.to_wire(prover.prove(z, r, s)))


def _lean_bytes(log_m, window):
    from liblightzk_b200 import serve
    _, p = _prover(log_m, window)
    rb = p.device_bytes()
    srv = serve.Server(rb - 1, max_inflight=1)
    srv.add(p)
    lean = p.device_bytes()
    srv.close()
    p.close()
    assert lean < rb
    return lean


def test_shrinks_on_a_full_device(cuda, orc, rng_state):
    import torch
    from liblightzk_b200 import serve
    lean = _lean_bytes(18, 13)
    circ, prover = _prover(18, 13)
    z, (r, s) = circ.witness(5), orc.rand_field(FR, 2, rng_state)
    want = _wire(prover, z, r, s)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog, chunk = [], 1 << 34
    try:
        while chunk >= (4 << 20):
            if torch.cuda.mem_get_info()[0] <= MARGIN + chunk:
                chunk //= 2
                continue
            hog.append(torch.empty(chunk, dtype=torch.uint8, device="cuda"))
        srv = serve.Server(prover.device_bytes() - 1, max_inflight=1)
        srv.add(prover)
        assert prover.device_bytes() == lean
    finally:
        del hog
        torch.cuda.empty_cache()
    assert (_wire(prover, z, r, s) == want).all()
    srv.close()


def test_short_prover_made_on_a_full_device(cuda):
    """too few entries for rounds, but a workspace more that lets B1 run beside
    A: without room for it the prover is made lean.  In a process of its own, where
    no pool holds memory that an allocation could take back."""
    code = f"import sys; sys.path[:0] = {[ROOT, os.path.join(ROOT, 'tests')]!r}; import test_prover_scratch_gpu as t; t.short_prover()"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]


def short_prover():
    import torch
    from liblightzk_b200 import groth16, synth
    orc, rng_state = Oracle(), np.array([0x5EED], np.uint64)
    lean = _lean_bytes(13, 22)
    circ, prover = _prover(13, 22)
    full = prover.device_bytes()
    assert full - lean > 128 << 20
    z, (r, s) = circ.witness(5), orc.rand_field(FR, 2, rng_state)
    want = _wire(prover, z, r, s)
    pk = synth.ProvingKey(circ, seed=4)
    prover.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog, chunk = [], 1 << 34
    try:
        while chunk >= (4 << 20):
            if torch.cuda.mem_get_info()[0] <= (full + lean) // 2 + chunk:
                chunk //= 2
                continue
            hog.append(torch.empty(chunk, dtype=torch.uint8, device="cuda"))
        prover = groth16.Prover(circ, pk, window_bits=22)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert prover.device_bytes() == lean
    assert (_wire(prover, z, r, s) == want).all()


def test_no_memory_for_the_lean_scratch(cuda, orc, rng_state):
    from liblightzk_b200 import LzkError, _capi, serve
    lean = _lean_bytes(12, 8)
    circ, prover = _prover(12, 8)
    z, (r, s) = circ.witness(5), orc.rand_field(FR, 2, rng_state)
    want = _wire(prover, z, r, s)
    srv = serve.Server(prover.device_bytes() - 1, max_inflight=1)
    L = _capi.lib()
    L.lzk_debug_fail_allocations(0)
    try:
        with pytest.raises(LzkError) as e:
            srv.add(prover)
        assert e.value.status == -2
        with pytest.raises(LzkError) as e:
            prover.prove(z, r, s)
        assert e.value.status == -2
    finally:
        L.lzk_debug_fail_allocations(-1)
    assert (_wire(prover, z, r, s) == want).all()
    assert prover.device_bytes() == lean
    srv.add(prover)
    srv.close()


def test_size_read_and_proofs_made_meanwhile(cuda, orc, rng_state):
    import torch
    from liblightzk_b200 import _capi, serve
    L = _capi.lib()
    circ, first = _prover(12, 8)
    z, (r, s) = circ.witness(5), orc.rand_field(FR, 2, rng_state)
    want = _wire(first, z, r, s)
    first.close()
    for _ in range(8):
        _, prover = _prover(12, 8)
        full, seen, stop, proofs = prover.device_bytes(), set(), threading.Event(), []

        def read():
            while not stop.is_set():
                seen.add(L.lzk_prover_device_bytes(prover.handle))

        def prove():
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                while not stop.is_set():
                    proofs.append(_wire(prover, z, r, s))

        threads = [threading.Thread(target=f) for f in (read, read, prove)]
        [t.start() for t in threads]
        servers = [serve.Server(full - 1, max_inflight=1) for _ in range(2)]
        try:
            [srv.add(prover) for srv in servers]
        finally:
            stop.set()
            [t.join() for t in threads]
        assert seen <= {full, prover.device_bytes()} and prover.device_bytes() < full
        assert all((p == want).all() for p in proofs)
        [srv.close() for srv in servers]
        prover.close()
