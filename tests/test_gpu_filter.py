"""The CRS filter (GPU): the default plans bound every candidate from the moments of whole
B runs and evaluate only the few that can win, with the direct kernels' arithmetic.  The
plain form must then reproduce the oracle's FP32 search, and the batched form the direct
search of a variant without a filter (12: candidates in grid order), at the sizes where
the runs, their padding, the staged chunks and the fallback to the direct kernel change."""
import numpy as np
import pytest

import oracle
import semb
import synth

pytestmark = pytest.mark.gpu


def _arrays(g):
    return semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                             g["scalco"], g["samples"])


def _survey(nb, tau, ns, apm, b1=1e-7, ncdp=9, fold=9, na=3, nc=5, az=0.0, seed=0):
    s = synth.crs_survey(seed=100 + nb + seed, ncdp=ncdp, noffsets=fold, ns=ns, na=na, nb=nb, nc=nc,
                         tau=tau * 0.002 * 1.0001, apm=apm, azimuth=az)
    s.params["b0"], s.params["b1"] = -b1, b1
    return s


# runs of one, full runs, one past a full run, several runs; odd records; every window;
# a B range so wide that most traces leave the expansion; apertures of one CDP, where
# every A and B ties and the lists overflow into the direct kernel; no valid item at all; B
# descending with its index
CASES = [(12, 1, 301, 50, 1e-7, 9), (13, 1, 256, 50, 1e-7, 9), (24, 2, 333, 75, 1e-7, 9), (25, 0, 290, 50, 1e-7, 9),
         (9, 2, 331, 50, 1e-7, 9), (31, 1, 300, 50, 3e-6, 9), (21, 1, 300, 5, 1e-7, 3), (21, 1, 64, 50, 1e-7, 9),
         (21, 1, 300, 50, -1e-7, 9), (15, 2, 300, 50, 1e-7, 9)]


@pytest.mark.parametrize("nb,tau,ns,apm,b1,ncdp", CASES)
@pytest.mark.parametrize("signed", [False, True])
def test_plain_filtered_search_is_the_oracle_s(nb, tau, ns, apm, b1, ncdp, signed):
    s = _survey(nb, tau, ns, apm, b1, ncdp, az=30.0 if signed else 0.0)
    g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float32)
    ref = oracle.crs(g, s.params, "f32", dm_signed=signed)
    with semb.Plan(semb.params(semb.CRS, mode=semb.PLAIN_F32, dm_mode=semb.DM_SIGNED if signed else semb.DM_ABS,
                               **s.params)) as p:
        p.upload(_arrays(g).view())
        p.run()
        ctr, sem, stk = p.download()
    assert np.array_equal(ctr, ref["ctr"])
    np.testing.assert_allclose(sem, ref["str"], rtol=1e-5, atol=1e-7)
    np.testing.assert_allclose(stk, ref["stk"], rtol=1e-5, atol=1e-6)


def test_plain_filtered_search_with_zero_and_non_finite_traces():
    s = _survey(21, 1, 300, 50)
    s.samples[3] = 0.0
    s.samples[20, 100] = np.inf
    s.samples[41, 150] = np.nan
    s.samples[60] *= 1e-12
    g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float32)
    ref = oracle.crs(g, s.params, "f32")
    with semb.Plan(semb.params(semb.CRS, mode=semb.PLAIN_F32, **s.params)) as p:
        p.upload(_arrays(g).view())
        p.run()
        ctr, sem, stk = p.download()
    assert np.array_equal(ctr, ref["ctr"])
    np.testing.assert_allclose(sem, ref["str"], rtol=1e-5, atol=1e-7)
    np.testing.assert_allclose(stk, ref["stk"], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("storage", [semb.STORE_F16, semb.STORE_BF16, semb.STORE_F32])
@pytest.mark.parametrize("nb,tau,ns,apm,b1,ncdp", [c for c in CASES if c[1] > 0])
def test_batched_filtered_search_agrees_with_the_direct_search(nb, tau, ns, apm, b1, ncdp, storage):
    """Up to the order of the FP32 sums of variant 10: semblances within 2e-6, and picks
    that differ only where the two semblances tie within that.  (Variants without B runs
    round the traveltime in another order, which moves a trace in or out of the record
    where it lies exactly on its end, as it does in the nb = 9 case.)"""
    s = _survey(nb, tau, ns, apm, b1, ncdp, na=7)
    g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float64)
    with semb.Plan(semb.params(semb.CRS, mode=semb.BATCHED, storage=storage, repick=semb.REPICK_OFF,
                               **s.params)) as p:
        p.upload(_arrays(g).view())
        p.run()
        ctr, sem, stk = p.download()
        p.set_variant(10)
        p.run()
        c0, s0, k0 = p.download()
    np.testing.assert_allclose(sem, s0, atol=2e-6, rtol=1e-5)
    same = ctr == c0
    np.testing.assert_allclose(stk[same], k0[same], atol=2e-6, rtol=1e-5)
    assert np.mean(same) >= (0.99 if apm > 12 else 0.0)   # one-CDP apertures: every pick is a tie


@pytest.mark.parametrize("nb,tau,ns,apm", [(21, 1, 300, 50), (9, 2, 331, 75), (5, 0, 500, 25), (21, 1, 700, 5)])
def test_certified_repick_gives_the_fp64_picks(nb, tau, ns, apm):
    """The re-pick in pairs of FP32 numbers against the same plan's FP64 re-pick (plans that
    keep the extra attributes take FP64 throughout): same picks, semblances and stacks, bit
    for bit, with few and many traces per aperture (apm 5: one CDP, all A and B tie)."""
    s = _survey(nb, tau, ns, apm, ncdp=9, fold=14, na=4)
    g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float64)
    out = []
    for attrs in (0, 1):
        for repick in (semb.REPICK_NEAR_TIES, semb.REPICK_ALWAYS):
            with semb.Plan(semb.params(semb.CRS, mode=semb.BATCHED, attrs=attrs, repick=repick, **s.params)) as p:
                p.upload(_arrays(g).view())
                p.run()
                out.append(p.download())
                assert p.stats()["repicked"] > 0
    for a, b in ((out[0], out[2]), (out[1], out[3])):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
