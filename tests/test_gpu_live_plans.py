"""Several live plans in one process (GPU).  A kernel's dynamic shared memory limit is one
value per process, and plans of different candidate counts launch the same search kernel
with different amounts (1 to 4 CTAs per SM): each must still run after the others were
uploaded, in turn and from several threads."""
import threading

import numpy as np
import pytest

import oracle
import semb
import synth

pytestmark = pytest.mark.gpu


def _plan(method, nc, tau, **kw):
    """An uploaded plan and its arrays."""
    if method == semb.CMP:
        s = synth.cmp_survey(seed=700 + nc, ncmp=3, half_offsets=np.linspace(10.0, 300.0, 20), ns=320, nc=nc,
                             tau=tau * 0.002 * 1.0001)
        g = oracle.gather(s.headers, s.samples, "cmp", s.params["aph"])
    else:
        s = synth.crs_survey(seed=700 + nc, ncdp=5, noffsets=9, ns=320, na=1, nb=1, nc=nc, tau=tau * 0.002 * 1.0001)
        g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float32)
    arr = semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                            g["scalco"], g["samples"])
    p = semb.Plan(semb.params(method, **s.params, **kw))
    p.upload(arr.view())
    return p


def _run(p):
    p.run()
    return p.download()


CASES = [(semb.CMP, 2, dict(mode=semb.PLAIN_F32), None), (semb.CMP, 1, dict(mode=semb.PLAIN_F32), 1),
         (semb.CRS, 2, dict(mode=semb.PLAIN_F32), None)] + [
    (semb.CMP, tau, dict(mode=semb.BATCHED, storage=st), v)
    for tau in (2, 5) for v in (30, 31) for st in (semb.STORE_F16, semb.STORE_F32)]


@pytest.mark.parametrize("method,tau,kw,variant", CASES)
def test_plans_of_other_sizes_do_not_disturb_each_other(method, tau, kw, variant):
    plans, first = [], []
    for nc in (256, 64, 160, 33):
        p = _plan(method, nc, tau, **kw)
        if variant is not None:
            p.set_variant(variant)
        plans.append(p)
        first.append(_run(p))
    for _ in range(2):
        for p, ref in zip(plans, first):
            for x, y in zip(_run(p), ref):
                assert np.array_equal(x, y)
    for p in plans:
        p.close()


def test_plans_in_threads_of_their_own():
    bad = []

    def work(nc):
        try:
            with _plan(semb.CMP, nc, 2, mode=semb.PLAIN_F32) as p:
                ref = _run(p)
                for _ in range(20):
                    if not all(np.array_equal(x, y) for x, y in zip(_run(p), ref)):
                        bad.append(f"{nc}: results differ")
        except semb.SembError as e:
            bad.append(f"{nc}: {e}")

    threads = [threading.Thread(target=work, args=(nc,)) for nc in (256, 64, 160, 33)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
