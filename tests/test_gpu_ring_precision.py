"""The batched CMP ring kernel's accuracy (GPU): with the FP32 store, where nothing else hides
the order of its sums, its semblances are as near 64 bits as the two-barrier kernel's (whose
chunks, and so whose FP32 chains of energy, are shorter)."""
import numpy as np
import pytest

import oracle
import semb
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau,nc,fold", [(0, 128, 200), (1, 256, 200), (2, 128, 240), (3, 128, 200), (7, 101, 128)])
def test_ring_energy_sums_are_as_accurate(tau, nc, fold):
    """Root mean square error from the FP64 oracle, where both pick its candidate: no more
    than 2% above (about 5000 values: the estimates themselves differ by 1%)."""
    s = synth.cmp_survey(seed=900 + tau, ncmp=6, half_offsets=np.linspace(25.0, 700.0, fold), ns=1000, nc=nc,
                         tau=tau * 0.002 * 1.0001, aph=3200)
    g = oracle.gather(s.headers, s.samples, "cmp", s.params["aph"], real=np.float64)
    ref = oracle.cmp(g, s.params, "f64")
    arr = semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                            g["scalco"], g["samples"])
    got = {}
    with semb.Plan(semb.params(semb.CMP, mode=semb.BATCHED, storage=semb.STORE_F32, repick=semb.REPICK_OFF,
                               **s.params)) as p:
        p.upload(arr.view())
        for v in (0, 30, 31):
            p.set_variant(v)
            p.run()
            got[v] = [x.copy() for x in p.download()]
    same = np.all([x[0] == ref["ctr"] for x in got.values()], axis=0) & (ref["str"] > 1e-3)
    assert same.mean() > 0.8
    rms = {v: np.sqrt(np.mean((x[1].astype(np.float64) - ref["str"])[same] ** 2)) for v, x in got.items()}
    for v in (30, 31):
        assert rms[v] <= 1.02 * rms[0], (rms, int(same.sum()))
