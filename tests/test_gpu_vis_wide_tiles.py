"""The 16 x 16-tap kernel with four warps (tile sides whose eight subgrids do not
fit shared memory) and the group kernels beyond (tiles of 64, where four do
not fit either), every pass against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import synth
from conftest import rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,supports,f64", [(40, [8] * 6, False), (48, [8] * 6, False), (48, [3, 4, 5, 6, 7, 8], True),
                                               (56, [5] * 6, False), (64, [8] * 6, False)])
def test_passes_vs_oracle(sdp, device, oracle32, oracle64, tile, supports, f64):
    import torch
    w = synth.make_workload("tiles", 48, 800.0, "disc", 20, 256, 5, 0.05, 1.0, 1e-3, 6, supports, oversampling=16, seed=11)
    G, us, ws = 256, w.cfg.uv_scale, w.cfg.w_scale
    o = oracle64 if f64 else oracle32
    uvw, gk, dk, sup = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w.uvw, w.gkernels, w.dkernels, w.supports))
    rng = np.random.default_rng(5)
    model = (rng.standard_normal((G * G, 2)) * 1e-2).astype(np.float32)
    model_d, meas = torch.from_numpy(model).cuda(), torch.from_numpy(w.vis).cuda()
    plan = device.plan(G, 16, us, ws, uvw, sdp.Device.wkernels(gk, sup, w.supports), sdp.Device.wkernels(dk, sup, w.supports),
                       mode=sdp.SDP_GRID_STD | (sdp.SDP_PLAN_COORD_F64 if f64 else 0), keep=(uvw, gk, dk, sup),
                       options=sdp.PlanOptions(tile, 512, 0, 0))
    plan.set_measured(meas)
    res, grid = (torch.empty((G * G, 2), device="cuda") for _ in range(2))
    pred, pred2 = torch.empty_like(meas), torch.empty_like(meas)
    plan.cycle(model_d, res, sdp.SDP_DEGRID_CONV, predicted=pred)
    plan.degrid(model_d, pred2, sdp.SDP_DEGRID_CONV)
    plan.grid(meas, grid)
    torch.cuda.synchronize()
    plan.check_flags()
    plan.close()
    p_ref = o.std_degridding(G, 16, w.dkernels, w.supports, model, w.uvw, us, ws, nearest=False)
    r_ref = o.std_gridding(G, 16, w.gkernels, w.supports, w.uvw, o.subtract_vis(w.vis, p_ref), us, ws)
    g_ref = o.std_gridding(G, 16, w.gkernels, w.supports, w.uvw, w.vis, us, ws)
    for name, got, ref in (("predicted", pred, p_ref), ("degrid", pred2, p_ref), ("residual", res, r_ref), ("grid", grid, g_ref)):
        assert rel_rms(got.cpu().numpy(), ref) <= 2e-6, name


def test_snapped_vs_oracle(sdp, device, oracle32):
    import torch
    w = synth.make_workload("tiles", 48, 800.0, "disc", 20, 256, 5, 0.05, 1.0, 1e-3, 6, [8] * 6, oversampling=16, seed=11)
    uvw, gk, sup, vis = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w.uvw, w.gkernels, w.supports, w.vis))
    wk = sdp.Device.wkernels(gk, sup, w.supports)
    plan = device.plan(256, 16, w.cfg.uv_scale, w.cfg.w_scale, uvw, wk, wk, mode=sdp.SDP_GRID_SNAPPED, keep=(uvw, gk, sup),
                       options=sdp.PlanOptions(48, 512, 0, 0))
    out = torch.empty((256 * 256, 2), device="cuda")
    plan.grid(vis, out)
    torch.cuda.synchronize()
    plan.check_flags()
    plan.close()
    ref = oracle32.gridding_cpu(256, 16, w.gkernels, w.supports, w.uvw, w.vis, w.cfg.uv_scale, w.cfg.w_scale)
    assert rel_rms(out.cpu().numpy(), ref) <= 2e-6
