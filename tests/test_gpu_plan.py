"""Path counts at the edges of the launch plan: the line between the
warp-per-path and the thread-per-path kernels (two fills of the device), single
warps per SM, partly filled last batches, one path more than whole waves, and
several scenarios in short units. FP32 results against the FP64 kernel on the
same normals within the FP32 rule (1e-4 per Greek, Greeks below 1% of their
group's largest against that 1%); the forward/backward pair's value equals the
fused call's, whichever kernels the size selects."""
import numpy as np
import pytest

from conftest import cfgs, pkg

pytestmark = pytest.mark.gpu

FILL = 2 * 152 * 6 * 4       # the line at 80/40 and 160/120 on 152 SMs


def _scaled(g, r, nn):
    e = 0.0
    for sl in (slice(0, 1), slice(1, 1 + nn), slice(1 + nn, 1 + 2 * nn)):
        floor = 1e-2 * np.abs(r[sl]).max() if r[sl].size > 1 else 0.0
        e = max(e, float((np.abs(g[sl] - r[sl]) / np.maximum(np.abs(r[sl]), max(floor, 1e-300))).max()))
    return e


def _run(cfg, paths, seed, pair=False, philox=False):
    import torch
    P = pkg()
    dz = torch.empty(paths * cfg.nmat, dtype=torch.float32, device="cuda")
    P.normals_f32_device(seed, paths, cfg.nmat, dz.data_ptr())
    dz64 = dz.double()
    with P.Engine(cfg) as e:
        o = torch.zeros(3, e.nscen, e.nout, dtype=torch.float64, device="cuda")
        val = torch.zeros(e.nscen, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        e.greeks_f32_device(dz.data_ptr(), paths, o[0].data_ptr())
        e.greeks_f64_device(dz64.data_ptr(), paths, o[1].data_ptr())
        if philox:
            e.greeks_philox_device(seed, paths, o[2].data_ptr())
        if pair:
            t = e.tape(paths)
            grad = torch.zeros(e.nscen, 2 * e.nn, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            e.forward_f32_device(dz.data_ptr(), paths, t, val.data_ptr())
            e.backward_f32_device(dz.data_ptr(), t, [1.0] * e.nscen, grad.data_ptr())
            e.synchronize()
            t.close()
        e.synchronize()
    a, r, ph = o.cpu().numpy()
    for s in range(a.shape[0]):
        assert _scaled(a[s], r[s], cfg.nn) <= 1e-4
    if philox:
        np.testing.assert_allclose(ph, a, rtol=1e-11, atol=1e-11 * np.abs(a).max())
    if pair:
        np.testing.assert_allclose(val.cpu().numpy(), a[:, 0], rtol=1e-12)
        np.testing.assert_allclose(grad.cpu().numpy(), a[:, 1:], rtol=2e-6, atol=1e-6 * np.abs(a[:, 1:]).max())


@pytest.mark.parametrize("paths", [1, 31, FILL, FILL + 1, 152 * 32 * 2 + 1, 152 * 128 + 1, 152 * 256 + 33, 152 * 384, 152 * 384 + 1,
                                   131072, 152 * 384 * 2 + 95])
def test_80x40_counts(paths):
    _run(cfgs().workload(4, paths), paths, 70 + paths % 7, pair=True, philox=True)


@pytest.mark.parametrize("paths", [3, FILL, FILL + 1, 152 * 256 + 1])
def test_160x120_counts(paths):
    _run(cfgs().workload(3, paths), paths, 80 + paths % 7, pair=True)


@pytest.mark.parametrize("curves,paths", [(3, FILL // 3), (3, FILL // 3 + 1), (7, 4099), (200, 385)])
def test_scenarios(curves, paths):
    cfg = cfgs().workload(5, paths)
    cfg.L0 = np.ascontiguousarray(cfg.L0[:curves])
    _run(cfg, paths, 90 + curves)
