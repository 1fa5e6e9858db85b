"""Warps per work item of the warp-per-visibility kernel: 16 or 8 in place of 4
where there are few work items, fewer where that many private subgrids do not
fit shared memory.

* values of every pass against the oracle for 4, 8 and 16 warps (by the number
  of items), tile sides that leave room for 16, 8 or 4 subgrids, and half
  supports with and without the compile-time form;
* the accuracy of a small set is that of items of 512 visibilities: error
  against a reference summed in doubles from 64 parts of the visibilities,
  within 1.35 of the same items with eight warps (two runs of one plan differ
  by 10 %; items of 64 to 224 visibilities had 1.8 times the error);
* the options that a plan reports build the same plan again;
* the autotuner's choice is no slower than the default plan."""
from __future__ import annotations

import numpy as np
import pytest

import synth
from conftest import rel_rms

pytestmark = pytest.mark.gpu


def _workload(n_ant, n_time, G, hs, seed=11, layout="disc", radius=800.0):
    return synth.make_workload("warps", n_ant, radius, layout, n_time, G, 5, 0.05, 1.0, 1e-3, 6, [hs] * 6, oversampling=16,
                               seed=seed)


def _tables(sdp, w):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w.uvw, w.gkernels, w.dkernels, w.supports)]
    return t, sdp.Device.wkernels(t[1], t[3], w.supports), sdp.Device.wkernels(t[2], t[3], w.supports)


def _plan(sdp, device, w, tables, options=None):
    t, wg, wd = tables
    return device.plan(w.cfg.grid_size, 16, w.cfg.uv_scale, w.cfg.w_scale, t[0], wg, wd, keep=t, options=options)


@pytest.mark.parametrize("n_time,hs,tile,chunk,f64", [
    (20, 3, 16, 512, False), (20, 4, 16, 512, False),  # 44 full items: 16 warps
    (20, 4, 16, 64, False), (20, 2, 16, 64, True),     # 352: 8 warps
    (48, 4, 16, 64, False), (48, 3, 16, 64, False),    # 846: 4 warps
    (20, 3, 16, 512, True),                            # 16 warps, FP64 coordinates
    (20, 4, 32, 512, False), (20, 4, 48, 512, True)])  # 16 subgrids do not fit; nor do 8
def test_values(sdp, device, oracle32, oracle64, n_time, hs, tile, chunk, f64):
    import torch
    w = _workload(48, n_time, 256, hs)
    G, us, ws = 256, w.cfg.uv_scale, w.cfg.w_scale
    o = oracle64 if f64 else oracle32
    rng = np.random.default_rng(5)
    model = (rng.standard_normal((G * G, 2)) * 1e-2).astype(np.float32)
    model_d, meas = torch.from_numpy(model).cuda(), torch.from_numpy(w.vis).cuda()
    t, wg, wd = _tables(sdp, w)
    plan = device.plan(G, 16, us, ws, t[0], wg, wd, keep=t, options=sdp.PlanOptions(tile, chunk, 0, 4),
                       mode=sdp.SDP_GRID_STD | (sdp.SDP_PLAN_COORD_F64 if f64 else 0))
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


def test_small_sets_keep_their_accuracy(sdp, device):
    import torch
    w = _workload(64, 30, 512, 4, 2, "log_spiral", 5000.0)
    tables, vis = _tables(sdp, w), torch.from_numpy(w.vis).cuda()
    ref, part = torch.zeros((512 * 512, 2), dtype=torch.float64, device="cuda"), torch.empty((512 * 512, 2), device="cuda")
    for k in range(64):
        t = [tables[0][0][k::64].contiguous(), *tables[0][1:]]
        plan = _plan(sdp, device, w, (t, *tables[1:]))
        plan.grid(vis[k::64].contiguous(), part)
        ref += part.double()
        torch.cuda.synchronize()
        plan.close()
    err = []
    for options in (None, sdp.PlanOptions(16, 512, 0, 8)):
        plan = _plan(sdp, device, w, tables, options)
        e = []
        for _ in range(16):
            plan.grid(vis, part)
            e.append(float((part.double() - ref).norm() / ref.norm()))
        plan.close()
        err.append(np.mean(e))
    assert err[0] <= 1.35 * err[1], err


def test_options_build_the_same_plan(sdp, device):
    w = _workload(48, 20, 256, 3)
    tables = _tables(sdp, w)
    plan = _plan(sdp, device, w, tables)
    again = _plan(sdp, device, w, tables, plan.options())
    a, b = plan.options(), again.options()
    assert (a.tile, a.chunk, a.lanes, a.warps) == (b.tile, b.chunk, b.lanes, b.warps)
    assert plan.num_work_items() == again.num_work_items()
    plan.close()
    again.close()


@pytest.mark.parametrize("n_ant,n_time,G", [(48, 20, 256), (64, 60, 512)])
def test_autotune_no_slower_than_the_default(sdp, device, n_ant, n_time, G):
    import torch
    w = _workload(n_ant, n_time, G, 3)
    tables, meas = _tables(sdp, w), torch.from_numpy(w.vis).cuda()
    model, res = torch.randn((G * G, 2), device="cuda"), torch.empty((G * G, 2), device="cuda")
    best, ms, _ = device.autotune(G, 16, w.cfg.uv_scale, w.cfg.w_scale, tables[0][0], tables[1], tables[2], meas, model, res)
    times = {}
    plans = {"default": _plan(sdp, device, w, tables), "best": _plan(sdp, device, w, tables, best)}
    for _ in range(5):
        for name, plan in plans.items():
            plan.set_measured(meas)
            plan.cycle(model, res, sdp.SDP_DEGRID_CONV)
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            for _ in range(50):
                plan.cycle(model, res, sdp.SDP_DEGRID_CONV)
            t1.record()
            torch.cuda.synchronize()
            times[name] = min(times.get(name, float("inf")), t0.elapsed_time(t1))
    for plan in plans.values():
        plan.close()
    assert times["best"] <= 1.15 * times["default"], times
