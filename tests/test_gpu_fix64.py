"""The FP64 kernels' fixed-point steps and the plain FP64 code beside them:
shapes at the edges (one step, an odd number of steps, one moving rate), path
counts at the edges of warps and blocks, and models or normals outside the
fixed-point range, alone and mixed with ordinary paths in one warp. Same
tolerances as the other FP64 parity tests: 1e-12 per output, with 1e-12 of
the largest where a horizon's rounding is larger than an output."""
import numpy as np
import pytest

from conftest import cfgs, pkg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _cfg(nn, nmat, paths, L0=(0.02, 0.07), lam=(0.1, 0.2), delta=0.25, seed=3):
    rng = np.random.default_rng(seed)
    nopt = 5
    return cfgs().LmmConfig("f", nn, nmat, delta, rng.uniform(*L0, nn), rng.uniform(*lam, nn),
                            rng.integers(1, nn - nmat + 1, nopt).astype(np.int32), rng.uniform(0.03, 0.06, nopt), paths)


def _check(cfg, z):
    with pkg().Engine(cfg) as e:
        g, _ = e.greeks_f64(z)
    m, _ = O.greeks(cfg, z)
    np.testing.assert_allclose(g[0], m, rtol=1e-11, atol=1e-12 * np.abs(m).max())
    return g[0]


@pytest.mark.parametrize("nn,nmat,paths", [(2, 1, 33), (3, 2, 32), (3, 1, 31), (8, 7, 257), (33, 7, 100), (41, 21, 4865),
                                           (80, 40, 1), (256, 129, 65)])
def test_edges(nn, nmat, paths):
    cfg = _cfg(nn, nmat, paths)
    _check(cfg, O.normals_f64(nn * 100 + nmat, paths, nmat))


@pytest.mark.parametrize("kw", [dict(lam=(0.6, 0.9)), dict(lam=(0.0, 0.0)), dict(L0=(1e-19, 1e-16)), dict(L0=(900.0, 1200.0)),
                                dict(delta=1.0, lam=(0.3, 0.4)), dict(delta=0.01), dict(L0=(0.5, 3.0), lam=(0.05, 0.1))])
def test_models_outside_the_range(kw):
    cfg = _cfg(20, 9, 130, **kw)
    _check(cfg, O.normals_f64(5, cfg.paths, cfg.nmat))


def test_paths_outside_the_range_beside_others():
    cfg = _cfg(24, 11, 96)
    z = O.normals_f64(6, cfg.paths, cfg.nmat).reshape(cfg.paths, cfg.nmat)
    z[3, 0], z[40, 5], z[95, 10], z[64, 4] = 15.5, -16.0, 40.0, -15.49
    z = z.reshape(-1)
    alone = _check(cfg, z)
    with pkg().Engine(cfg) as e:
        bad = z.copy()
        bad[7] = np.nan
        with pytest.raises(pkg().LmmError) as ei:
            e.greeks_f64(bad)
        assert ei.value.code == -4
        again, _ = e.greeks_f64(z)
    assert np.array_equal(again[0], alone)


def test_rates_at_powers_of_two():
    """delta L0 = 2^-6 puts zero low words through every integer sum of the first
    steps. The oracle's and the kernel's sums over 4,096 paths each round to a
    few units in 2^53."""
    cfg = _cfg(24, 11, 4096, L0=(0.0625, 0.0625))
    z = O.normals_f64(8, cfg.paths, cfg.nmat)
    with pkg().Engine(cfg) as e:
        g, _ = e.greeks_f64(z)
    m, _ = O.greeks(cfg, z)
    np.testing.assert_allclose(g[0], m, rtol=2e-14, atol=2e-14 * np.abs(m).max())


@pytest.mark.parametrize("nn,nmat,central", [(12, 5, False), (9, 4, True)])
def test_bump_values_match_oracle(nn, nmat, central):
    """Each difference against the oracle's values at the bumped inputs: V is
    good to 1e-13 of itself on either side, so a difference to 2e-13 V / h."""
    cfg, h = _cfg(nn, nmat, 200), 1e-4
    z = O.normals_f64(9, cfg.paths, nmat)
    z[17] = 20.0                                   # one path outside the fixed-point range
    with pkg().Engine(cfg) as e:
        g, _ = e.bump_greeks_f64(z, h, central=central)
    base = O.greeks(cfg, z)[0][0]
    assert g[0, 0] == pytest.approx(base, rel=1e-12)

    def value(j, x):
        c = cfg.with_paths(cfg.paths)
        a = np.zeros(nn)
        a[j % nn] = x
        c.L0, c.lam = (cfg.L0 + a, cfg.lam) if j < nn else (cfg.L0, cfg.lam + a)
        return O.greeks(c, z)[0][0]

    for j in (0, nmat, nn - 1, nn, nn + 1, 2 * nn - 1):
        want = (value(j, h) - value(j, -h)) / (2 * h) if central else (value(j, h) - base) / h
        assert abs(g[0, 1 + j] - want) <= 2e-13 * abs(base) / h
