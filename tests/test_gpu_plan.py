"""Shapes and path counts at the edges of the launch plan: the line between the
warp-per-path and the thread-per-path kernels (in fills of the device), single
warps per SM, partly filled last batches, one path more than whole waves, and
several scenarios in short units. FP32 results against the FP64 kernel on the
same normals within the FP32 rule (1e-4 per Greek, Greeks below 1% of their
group's largest against that 1%); the forward/backward pair's value equals the
fused call's, whichever kernels the size selects."""
import numpy as np
import pytest

from conftest import cfgs, pkg

pytestmark = pytest.mark.gpu

FILL = 2 * 152 * 6 * 4       # two fills on 152 SMs, the line at 160/120; one and a half at 80/40


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


@pytest.mark.parametrize("paths", [FILL * 3 // 4, FILL * 3 // 4 + 1, 152 * 512, 152 * 512 + 1, 152 * 512 + 152 * 416 + 5])
def test_80x40_counts_of_blocks_of_512(paths):
    _run(cfgs().workload(4, paths), paths, 71 + paths % 5, pair=True, philox=True)


@pytest.mark.parametrize("paths", [3, FILL, FILL + 1, 152 * 256 + 1])
def test_160x120_counts(paths):
    _run(cfgs().workload(3, paths), paths, 80 + paths % 7, pair=True)


@pytest.mark.parametrize("curves,paths", [(3, FILL // 3), (3, FILL // 3 + 1), (7, 4099), (200, 385)])
def test_scenarios(curves, paths):
    cfg = cfgs().workload(5, paths)
    cfg.L0 = np.ascontiguousarray(cfg.L0[:curves])
    _run(cfg, paths, 90 + curves)


def _shape(nn, nmat, paths, seed, nopt=7, vol=(0.1, 0.2)):
    rng = np.random.default_rng(seed)
    return cfgs().LmmConfig("shape", nn, nmat, 0.25, rng.uniform(0.02, 0.07, nn), rng.uniform(*vol, nn),
                            rng.integers(1, nn - nmat + 1, nopt).astype(np.int32), rng.uniform(0.03, 0.06, nopt), paths)


# rate counts at the edges of the blocks of 20 and passes of 40, step counts with every remainder by 4, block sizes
# of 512, 384, 256 and 128 threads
SHAPES = [(2, 1), (3, 2), (19, 7), (20, 10), (21, 6), (33, 7), (40, 39), (41, 20), (61, 33), (79, 40), (96, 60), (100, 99),
          (121, 62), (160, 80), (181, 45), (200, 100), (256, 40), (256, 131)]


@pytest.mark.parametrize("nn,nmat", SHAPES, ids=lambda v: str(v))
def test_shapes_beyond_the_line(nn, nmat):
    """More paths than the warp-per-path kernels take, with a ragged end; the
    vols keep the Euler paths of the long shapes tame."""
    paths = 2 * 152 * 16 * 4 + 257
    cfg = _shape(nn, nmat, paths, nn * 1000 + nmat, vol=(0.05, 0.12) if nmat > 90 else (0.1, 0.2))
    _run(cfg, paths, nn + nmat, pair=True, philox=True)


@pytest.mark.parametrize("ck", [0, 4, 6, 8, 12, 60])
def test_checkpoint_intervals_beyond_the_line(ck):
    """Intervals that are a multiple of 4 and one that is not (warp per path)."""
    cfg = _shape(96, 60, 15007, 5)
    cfg.ckpt_every = ck
    _run(cfg, 15007, 6, pair=True)


def test_scenarios_of_a_shape_beyond_the_line():
    cfg = _shape(50, 22, 4001, 7)
    rng = np.random.default_rng(1)
    cfg.L0 = rng.uniform(0.02, 0.07, (5, 50))
    _run(cfg, 4001, 8, pair=True)


@pytest.mark.parametrize("wl,curves,paths", [(4, 1, 1), (4, 1, 3001), (4, 1, 20_001), (3, 1, 500), (3, 1, 9_001), (5, 3, 777)])
def test_normals_may_change_between_forward_and_backward(wl, curves, paths):
    """The 80/40 and 160/120 tapes hold what the backward needs, whichever
    kernels the size selects."""
    import torch
    P = pkg()
    cfg = cfgs().workload(wl, paths)
    if curves > 1:
        cfg.L0 = np.ascontiguousarray(cfg.L0[:curves])
    z = torch.randn(paths * cfg.nmat, device="cuda")
    grads = []
    for spoil in (False, True):
        with P.Engine(cfg) as e:
            t = e.tape(paths)
            zz, v = z.clone(), torch.zeros(e.nscen, dtype=torch.float64, device="cuda")
            g = torch.zeros(e.nscen, 2 * e.nn, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            e.forward_f32_device(zz.data_ptr(), paths, t, v.data_ptr())
            e.synchronize()
            if spoil:
                zz.fill_(3.0)
                torch.cuda.synchronize()
            e.backward_f32_device(zz.data_ptr(), t, [1.0] * e.nscen, g.data_ptr())
            e.synchronize()
            t.close()
            grads.append(g.cpu())
    assert torch.equal(*grads)


@pytest.mark.parametrize("wl,paths", [(3, 2000), (3, 9001), (4, 3000), (4, 20_001)])
@pytest.mark.parametrize("shock", [30.0, 100.0, -100.0])
def test_rates_beyond_fp32(wl, paths, shock):
    """One path whose rates outgrow FP32: its discount factor is 0, and the call
    prices the others, whichever kernel the size selects."""
    cfg = cfgs().workload(wl, paths)
    z = np.random.default_rng(3).standard_normal(paths * cfg.nmat).astype(np.float32)
    z[cfg.nmat * 7 + 3] = shock
    ref = np.delete(z.reshape(paths, cfg.nmat), 7, 0).ravel()
    with pkg().Engine(cfg) as e:
        out, _ = e.greeks_f32(z, paths)
        base, _ = e.greeks_f32(ref, paths - 1)
    assert np.isfinite(out).all()
    # one path more or less moves the mean by at most its share of the largest values
    np.testing.assert_allclose(out.reshape(-1)[0], base.reshape(-1)[0], rtol=10.0 / paths)
