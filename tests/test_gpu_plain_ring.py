"""The ring kernels (GPU).  Plain: windows up to 5, candidates in pairs, 8 or 4 per thread, one
to four CTAs per SM.  Every variant must reproduce the oracle's FP32 search, for candidate
counts around its warps' edges, folds around the staged chunk's, odd records, and records
too long for three staged planes (which take the two-barrier kernel)."""
import numpy as np
import pytest

import oracle
import semb
import synth

pytestmark = pytest.mark.gpu


def _arrays(g):
    return semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                             g["scalco"], g["samples"])


def _check(out, ref):
    # where no candidate has a positive semblance the search reports none (-1, CRS 0); of a
    # grid of one candidate the oracle then reports that one
    picked = ref["str"] > 0 if ref["ctr"].max() == 0 else np.ones(ref["str"].shape, bool)
    assert np.array_equal(out[0][picked], ref["ctr"][picked])
    np.testing.assert_allclose(out[1], ref["str"], rtol=1e-5, atol=1e-7)
    np.testing.assert_allclose(out[2], ref["stk"], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("nc,fold,ns,tau", [(1, 3, 97, 0), (31, 20, 301, 1), (104, 33, 257, 2), (105, 127, 300, 1),
                                            (128, 129, 289, 0), (129, 40, 333, 2), (257, 12, 310, 1)])
def test_cmp_plain_variants_match_the_oracle(nc, fold, ns, tau):
    s = synth.cmp_survey(seed=200 + nc, ncmp=5, half_offsets=np.linspace(10.0, 0.9 * ns, fold), ns=ns, nc=nc,
                         tau=tau * 0.002 * 1.0001)
    g = oracle.gather(s.headers, s.samples, "cmp", s.params["aph"])
    ref = oracle.cmp(g, s.params, "f32")
    with semb.Plan(semb.params(semb.CMP, mode=semb.PLAIN_F32, **s.params)) as p:
        p.upload(_arrays(g).view())
        for v in (None, 0, 1, 2):
            if v is not None:
                p.set_variant(v)
            p.run()
            _check(p.download(), ref)


@pytest.mark.parametrize("na,nb,nc,tau,ns", [(1, 1, 1, 1, 200), (2, 3, 5, 2, 231), (3, 2, 7, 0, 250)])
def test_crs_plain_variants_match_the_oracle(na, nb, nc, tau, ns):
    s = synth.crs_survey(seed=300 + nc, ncdp=7, noffsets=11, ns=ns, na=na, nb=nb, nc=nc, tau=tau * 0.002 * 1.0001)
    g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float32)
    ref = oracle.crs(g, s.params, "f32")
    with semb.Plan(semb.params(semb.CRS, mode=semb.PLAIN_F32, **s.params)) as p:
        p.upload(_arrays(g).view())
        for v in (None, 0, 1, 2):
            if v is not None:
                p.set_variant(v)
            p.run()
            _check(p.download(), ref)


@pytest.mark.parametrize("storage", [semb.STORE_F16, semb.STORE_BF16, semb.STORE_F32])
@pytest.mark.parametrize("nc,fold,ns,tau", [(1, 3, 97, 0), (40, 20, 301, 1), (104, 33, 257, 2), (111, 127, 300, 3),
                                            (128, 129, 289, 5), (129, 60, 333, 7), (257, 12, 310, 1)])
def test_cmp_batched_ring_agrees_with_the_two_barrier_kernel(nc, fold, ns, tau, storage):
    """The batched ring variants (30, 31) against variant 0: the same arithmetic per item,
    FP32 sums in another order."""
    s = synth.cmp_survey(seed=500 + nc, ncmp=5, half_offsets=np.linspace(10.0, 0.9 * ns, fold), ns=ns, nc=nc,
                         tau=tau * 0.002 * 1.0001)
    g = oracle.gather(s.headers, s.samples, "cmp", s.params["aph"])
    with semb.Plan(semb.params(semb.CMP, mode=semb.BATCHED, storage=storage, repick=semb.REPICK_OFF,
                               **s.params)) as p:
        p.upload(_arrays(g).view())
        p.set_variant(0)
        p.run()
        ref = p.download()
        for v in (30, 31):
            p.set_variant(v)
            p.run()
            ctr, sem, stk = p.download()
            assert np.mean(ctr == ref[0]) >= 0.995
            np.testing.assert_allclose(sem, ref[1], atol=2e-6, rtol=1e-5)
            same = ctr == ref[0]
            np.testing.assert_allclose(stk[same], ref[2][same], atol=2e-6, rtol=1e-5)


def test_records_too_long_for_the_ring_still_run():
    s = synth.cmp_survey(seed=210, ncmp=1, fold=3, ns=20000, nc=3, tau=0.002)
    g = oracle.gather(s.headers, s.samples, "cmp", s.params["aph"])
    ref = oracle.cmp(g, s.params, "f32")
    with semb.Plan(semb.params(semb.CMP, mode=semb.PLAIN_F32, **s.params)) as p:
        p.upload(_arrays(g).view())
        assert p.stats()["variant"] == 2
        p.run()
        _check(p.download(), ref)
