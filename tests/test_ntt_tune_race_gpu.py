"""A transform beside another thread that sets its tuning entry: every call
uses one block size throughout, so passes and bit reversal agree."""
import threading

import pytest

from oracle import FR

pytestmark = pytest.mark.gpu

NTT_BLOCK = 3


@pytest.mark.parametrize("k", [9, 10, 12])
def test_block_set_while_transforms_run(cuda, orc, rng_state, k):
    import torch
    from liblightzk_b200 import _capi, device, ntt
    L = _capi.lib()
    a = orc.rand_field(FR, 1 << k, rng_state)
    want = device.to_device(orc.ntt(a, k, ntt.FORWARD))
    ntt.prepare(k)
    calls = 3000
    x = device.to_device(a).repeat(calls, 1, 1)
    stop = threading.Event()

    def flip():
        while not stop.is_set():
            for block in (256, 4096):      # several passes, or one that writes natural order
                L.lzk_tune_set(NTT_BLOCK, 0, k, block)

    t = threading.Thread(target=flip)
    t.start()
    try:
        for i in range(calls):
            ntt.ntt(x[i], k, ntt.FORWARD)
    finally:
        stop.set()
        t.join()
        L.lzk_tune_set(NTT_BLOCK, 0, k, 0)
    torch.cuda.synchronize()
    wrong = (x != want).flatten(1).any(1).sum().item()
    assert wrong == 0, f"{wrong} of {calls} transforms"
