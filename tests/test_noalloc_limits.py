"""lzk_msm_g1_noalloc at the edge of its scratch: a short accumulation chunk in
the tuning table, whose partial sums take more of the array, refuses no size
that fits with a longer one."""
import pytest
import torch

EINVAL, CHUNK = -1, 1
SIZES = [13116, 15000, 16384]      # class 2^14, two-bit windows


@pytest.fixture(params=[0, 8, 16, 32])
def chunk(request):
    from liblightzk_b200 import _capi
    L = _capi.lib()
    assert L.lzk_tune_set(CHUNK, 1, 14, request.param) == 0
    yield request.param
    L.lzk_tune_set(CHUNK, 1, 14, 0)


@pytest.mark.parametrize("n", SIZES)
def test_accepted_with_any_chunk(chunk, n):
    if torch.cuda.is_available():
        pytest.skip("the arguments point nowhere: only where no device can read them")
    from liblightzk_b200 import _capi
    assert _capi.lib().lzk_msm_g1_noalloc(256, 256, n, 256, 2, None) != EINVAL


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_sum_with_any_chunk(cuda, orc, rng_state, chunk, n):
    from helpers import bases, same_point, scalars
    from liblightzk_b200 import _capi, device
    s, b = scalars(orc, n, rng_state), bases(orc, 1, n, rng_state)
    ds, db, out = device.to_device(s), device.to_device(b), device.empty((3, 4))
    _capi.call("lzk_msm_g1_noalloc", ds.data_ptr(), db.data_ptr(), n, out.data_ptr(), 2, None)
    assert same_point(orc, 1, device.to_host(out), orc.msm(1, s, b))
