"""Sorted entries are numbered with 32 bits: an MSM whose two halves a scalar
(csrc/glv.cuh) would make too many takes the plain digits, one that is too
large in either form is refused, and a batch plan falls back the same way.

The sizes are at the limits, so the tests on the CPU stop at the first device
allocation (any status but LZK_EINVAL means the size was accepted); the GPU
test is one MSM just above 2^28 points."""
import ctypes

import numpy as np
import pytest
import torch

EINVAL = -1
WINDOW, TABLE_WINDOW = 0, 4
MAX_ENTRIES = (1 << 32) - 1


def _lib():
    from liblightzk_b200 import _capi
    return _capi.lib()


def _no_gpu():
    if torch.cuda.is_available():
        pytest.skip("the arguments point nowhere: only where no device can read them")


def _msm_status(group, n, c):
    from liblightzk_b200 import _capi
    cfg = _capi.MsmCfg()
    cfg.window_bits = c
    f = _lib().lzk_msm_g1 if group == 1 else _lib().lzk_msm_g2
    return f(256, 256, n, 256, ctypes.byref(cfg), None)


def _plain(n, c):
    return n * -(-255 // c)


def _halves(n, c):
    return n * 2 * -(-127 // c)


@pytest.mark.parametrize("c", [13, 16, 17, 22, 24])
@pytest.mark.parametrize("edge", [0, 1])
def test_msm_accepted_up_to_the_limit(c, edge):
    _no_gpu()
    from liblightzk_b200 import msm
    per = min(_plain(1, c), _halves(1, c))
    n = MAX_ENTRIES // per + edge
    assert (_msm_status(1, n, c) == EINVAL) == (edge == 1)
    assert (msm.workspace_bytes(1, n, c) == 0) == (edge == 1)
    n = MAX_ENTRIES // _plain(1, c) + edge
    assert (_msm_status(2, n, c) == EINVAL) == (edge == 1)


def test_halved_scalars_only_where_their_entries_fit():
    # at 17 bits the halves make 16 entries a scalar, the plain digits 15
    from liblightzk_b200 import msm
    n = MAX_ENTRIES // 16
    assert _halves(n + 1, 17) > MAX_ENTRIES >= _plain(n + 1, 17)
    # the doubled bases, 128 bytes a point, are in the scratch of the first only
    assert msm.workspace_bytes(1, n, 17) - msm.workspace_bytes(1, n + 1, 17) > 64 * n


@pytest.mark.parametrize("n", [(1 << 28) + 1, 300_000_000, 357_000_000])
def test_tuned_width_that_does_not_fit_is_passed_over(n):
    from liblightzk_b200 import msm
    L = _lib()
    saved = L.lzk_tune_get(WINDOW, 1, 29)
    assert L.lzk_tune_set(WINDOW, 1, 29, 16) == 0
    try:
        c = msm.autotune_window(1, n)
        assert min(_plain(n, c), _halves(n, c)) <= MAX_ENTRIES
        assert msm.workspace_bytes(1, n) > 0
    finally:
        L.lzk_tune_set(WINDOW, 1, 29, saved)


def _plan_status(sizes, flags=0, window=0):
    from liblightzk_b200 import _capi
    md = (_capi.MsmDesc * len(sizes))()
    for m, n in zip(md, sizes):
        m.scalars = m.bases = m.out = 256
        m.n, m.window_bits = n, window
    h = ctypes.c_void_p()
    return _lib().lzk_batch_plan_create_ex(1, md, len(sizes), None, 0, flags, ctypes.byref(h))


def test_plan_without_the_endomorphism():
    _no_gpu()
    n = MAX_ENTRIES // 16 + 1
    assert _plan_status([n // 2, n - n // 2], window=17) != EINVAL
    assert _plan_status([MAX_ENTRIES // 15 + 1], window=17) == EINVAL


def test_fixed_plan_with_the_widths_of_its_msms():
    # by total work these would take narrow windows, whose tables hold more
    # points than can be numbered
    _no_gpu()
    L = _lib()
    assert L.lzk_tune_set(TABLE_WINDOW, 1, 10, 16) == 0
    try:
        assert _plan_status([1000] * 130000, flags=1) != EINVAL
    finally:
        L.lzk_tune_set(TABLE_WINDOW, 1, 10, 0)


def test_persistent_plan_of_too_many_widths_stays_unsupported():
    _no_gpu()
    from liblightzk_b200 import _capi
    md = (_capi.MsmDesc * 21)()
    for i, m in enumerate(md):
        m.scalars = m.bases = m.out = 256
        m.n, m.window_bits = 10, 2 + i
    h = ctypes.c_void_p()
    assert _lib().lzk_batch_plan_create_ex(1, md, 21, None, 0, 2, ctypes.byref(h)) == -5


@pytest.mark.gpu
def test_plain_g1_msm_above_2e28_points(cuda, orc, rng_state):
    """Tiles of 2^14 points and scalars: the sum is the tile's times the number
    of tiles, plus the rest of one."""
    from helpers import bases, same_point, scalars
    from oracle import FR
    from liblightzk_b200 import autotune, device, msm
    tile, reps, rest = 1 << 14, (1 << 14) + 3, 777
    n = tile * reps + rest
    s, b = scalars(orc, tile, rng_state), bases(orc, 1, tile, rng_state)
    L = _lib()
    saved = L.lzk_tune_get(WINDOW, 1, 29)
    assert L.lzk_tune_set(WINDOW, 1, 29, 16) == 0      # 16 entries a scalar would not fit
    try:
        ds, db = device.to_device(s).repeat(reps + 1, 1), device.to_device(b).repeat(reps + 1, 1, 1)
        got = device.to_host(msm.msm(1, ds[:n], db[:n]))
    finally:
        L.lzk_tune_set(WINDOW, 1, 29, saved)
        del ds, db
        torch.cuda.empty_cache()
    parts = np.stack([orc.msm(1, s, b), orc.msm(1, s[:rest], b[:rest])])
    k = orc.to_mont(FR, np.array([[reps, 0, 0, 0], [1, 0, 0, 0]], np.uint64))
    assert same_point(orc, 1, got, orc.msm(1, k, orc.jac_to_aff(1, parts)))
