"""G2 MSMs without the affine rounds: over two lanes a point below 4096 chunks,
with whole points from there on, for both base layouts and a plan."""
import ctypes

import pytest

from helpers import bases, same_point, scalars

pytestmark = pytest.mark.gpu


def _reference_records(b):
    """affine (n, x/y, c0/c1, 4) to the reference's lane records with Z = 1"""
    import torch
    r = torch.zeros((b.shape[0], 2, 3, 4), dtype=torch.int64, device=b.device)
    r[:, 0, :2], r[:, 1, :2] = b[:, :, 0], b[:, :, 1]
    r[:, 0, 2, 0] = (b != 0).flatten(1).any(1)
    return r


@pytest.mark.parametrize("n", [300, 885, 886, 2500])      # 37 windows of 7 bits, 8 entries a chunk
@pytest.mark.parametrize("layout", ["affine", "reference", "table"])
def test_sum(cuda, orc, rng_state, n, layout):
    import torch
    from liblightzk_b200 import _capi, device, msm
    s, b = scalars(orc, n, rng_state), bases(orc, 2, n, rng_state)
    b[::50] = 0
    b[1::50] = b[2]
    ds, db, out = device.to_device(s), device.to_device(b), device.empty((3, 2, 4))
    cfg = _capi.MsmCfg()
    cfg.window_bits, cfg.acc_chunk = 7, 8
    if layout == "affine":
        # the scratch of a list too short for the rounds, which fits them nowhere
        ws = torch.empty(_capi.lib().lzk_msm_workspace_bytes(2, n, ctypes.byref(cfg)) - 1, dtype=torch.uint8, device="cuda")
        if n * 37 >= 1 << 16:
            cfg.workspace, cfg.workspace_bytes = ws.data_ptr(), ws.numel()
    else:
        cfg.base_layout = _capi.BASES_REF_G2_LANES
        if layout == "table":
            cfg.flags, cfg.precomp_windows, cfg.level_stride = _capi.LZK_MSM_PRECOMPUTED, 37, n
            db = msm.precompute(2, db, 7)
        db = _reference_records(db)
    _capi.call("lzk_msm_g2", ds.data_ptr(), db.data_ptr(), n, out.data_ptr(), ctypes.byref(cfg), None)
    assert same_point(orc, 2, device.to_host(out), orc.msm(2, s, b))


@pytest.mark.parametrize("n", [100, 1500])
def test_plan_too_short_for_rounds(cuda, orc, rng_state, n):
    from liblightzk_b200 import batch, device
    s, b = scalars(orc, n, rng_state), bases(orc, 2, n, rng_state)
    out = device.empty((3, 2, 4))
    plan = batch.BatchPlan(2, msms=[(device.to_device(s), device.to_device(b), out, 13)], fixed_bases=True)
    plan.run()
    assert same_point(orc, 2, device.to_host(out), orc.msm(2, s, b))
    plan.close()
