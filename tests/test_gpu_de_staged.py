"""CRS-DE's staged kernel (GPU): bit for bit the oracle's restatement, for populations around
the lanes' pairs (odd numbers of individuals per lane, fewer than evolution needs, the
largest), every window, apertures of several staged chunks, records that are no multiple of
a CTA's samples, and records too long for staging."""
import numpy as np
import pytest

import oracle
import semb
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb,nc,tau,ns,ncdp,fold,ngen", [
    (1, 3, 1, 1, 61, 3, 5, 2), (2, 2, 1, 0, 90, 3, 7, 3), (3, 11, 1, 2, 123, 5, 9, 4), (4, 4, 4, 1, 100, 9, 16, 3),
    (5, 13, 1, 1, 77, 9, 30, 2), (8, 8, 4, 2, 64, 4, 12, 2), (2, 2, 2, 1, 24000, 1, 2, 1)])
def test_de_matches_the_oracle(na, nb, nc, tau, ns, ncdp, fold, ngen):
    dt_us = 4000 if ns < 1000 else 200
    s = synth.crs_survey(seed=400 + ns, ncdp=ncdp, noffsets=fold, ns=ns, dt_us=dt_us, na=na, nb=nb, nc=nc,
                         tau=tau * dt_us * 1e-6 * 1.0001)
    p = dict(s.params)
    g = oracle.gather(s.headers, s.samples, "crs", p["aph"], p["apm"], real=np.float32)
    ref = oracle.crs_de(g, p, ngen, "f32")
    view = semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                             g["scalco"], g["samples"])
    with semb.Plan(semb.params(semb.CRS, mode=semb.PLAIN_F32, ngen=ngen, **p)) as plan:
        plan.upload(view.view())
        plan.run()
        ctr, sem, stk = plan.download()
        a, b, c = plan.download_abc()
    assert np.array_equal(sem, ref["str"])
    assert np.array_equal(stk, ref["stk"])
    assert np.array_equal(a, ref["a"]) and np.array_equal(b, ref["b"]) and np.array_equal(c, ref["c"])
