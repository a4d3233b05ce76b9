"""The re-pick in pairs of FP32 numbers against the same plan's FP64 re-pick (GPU): picks,
semblances and stacks, bit for bit (plans that keep the extra attributes take FP64
throughout).  Surveys on which a bound that takes rounding errors as random, or the slopes
from the energy, does not hold: samples near the Nyquist frequency, whose values cancel
where their slopes do not; geometries that repeat, whose errors add up; windows of one
sample; traces at zero offset, whose traveltimes fall on samples."""
import numpy as np
import pytest

import semb

pytestmark = pytest.mark.gpu


def _arrays(seed, ns, kind, repeat, noise, zero=False, ncdp=6, fold=24):
    """ncdp CDPs 12.5 m apart, `fold` offsets each, every trace `repeat` times."""
    r = np.random.default_rng(seed)
    cdp, off = np.divmod(np.arange(ncdp * fold).repeat(repeat), fold)
    mx = 125 * cdp                      # decimetres
    half = (0 if zero else 200) + 100 * off
    n = len(mx)
    t = np.arange(ns)
    if kind == "nyquist":
        base = (-1.0) ** t * (1.0 + 0.1 * np.sin(0.01 * t))
    else:
        base = sum(np.sin(2 * np.pi * (f * t + r.random())) for f in (0.03, 0.05, 0.08))
    amp = 1.0 + 0.3 * r.standard_normal((n, 1))
    smp = (amp * base + noise * r.standard_normal((n, ns))).astype(np.float32)
    end = (1 + np.arange(ncdp)) * fold * repeat
    z = np.zeros(n, np.int32)
    return semb.GatherArrays(end, ns, 4000, (mx + half).astype(np.int32), z, (mx - half).astype(np.int32), z,
                             np.full(n, -10, np.int32), smp)


def _run(arr, tau, attrs, repick, **grid):
    prm = dict(a0=-1e-4, a1=1e-4, na=5, b0=-1e-8, b1=1e-8, nb=5, c0=4e-7, c1=1.6e-6, nc=5, aph=2000, apm=40,
               tau=tau * 0.004 * 1.0001, azimuth=0.0)
    prm.update(grid)
    with semb.Plan(semb.params(semb.CRS, mode=semb.BATCHED, storage=semb.STORE_F32, attrs=attrs, repick=repick,
                               **prm)) as p:
        p.upload(arr.view())
        p.run()
        assert p.stats()["repicked"] > 0
        return p.download()


@pytest.mark.parametrize("tau", [0, 1, 2])
@pytest.mark.parametrize("kind,repeat,noise,zero", [("nyquist", 1, 0.02, False), ("nyquist", 16, 1e-3, False),
                                                    ("smooth", 16, 1e-3, False), ("smooth", 1, 0.3, True),
                                                    ("nyquist", 8, 1e-4, True), ("smooth", 64, 0.1, False)])
def test_pairs_give_the_fp64_results(kind, repeat, noise, zero, tau):
    for seed in range(4):
        arr = _arrays(seed, 1500, kind, repeat, noise, zero)
        for repick in (semb.REPICK_ALWAYS, semb.REPICK_NEAR_TIES):
            got, ref = (_run(arr, tau, attrs, repick) for attrs in (0, 1))
            for x, y in zip(got, ref):
                assert np.array_equal(x, y), (seed, repick, int((x != y).sum()), x.size)


def _pairs_of_cdps(seed, ns, repeat, npairs=6):
    """CDPs of one trace, each with a neighbour of `repeat` traces of one geometry, and samples
    that alternate: where that geometry's traveltime falls between two of them every value
    cancels, and no slope does."""
    r = np.random.default_rng(seed)
    mx, half, end = [], [], []
    for k in range(npairs):
        mx += [10000 * k] + [10000 * k + 125] * repeat
        half += [3000] + [4000 + 370 * k] * repeat
        end += [len(mx) - repeat, len(mx)]
    mx, half = np.array(mx), np.array(half)
    amp = 1.0 + 0.3 * r.standard_normal((len(mx), 1))
    smp = (amp * (-1.0) ** np.arange(ns)).astype(np.float32)
    z = np.zeros(len(mx), np.int32)
    return semb.GatherArrays(end, ns, 4000, (mx + half).astype(np.int32), z, (mx - half).astype(np.int32), z,
                             np.full(len(mx), -10, np.int32), smp)


@pytest.mark.parametrize("tau", [0, 1, 2])
@pytest.mark.parametrize("repeat", [64, 512])
def test_cancelling_values_of_one_geometry(repeat, tau):
    for seed in range(4):
        arr = _pairs_of_cdps(seed, 1500, repeat)
        got, ref = (_run(arr, tau, attrs, semb.REPICK_ALWAYS, c0=4e-7 + 1e-9 * seed) for attrs in (0, 1))
        for x, y in zip(got, ref):
            assert np.array_equal(x, y), (seed, int((x != y).sum()), x.size)
