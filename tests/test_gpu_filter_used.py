"""The CRS filter against the search without it (GPU).  Every test asserts that the filter is
attached, turns it off on the same plan and compares the results bit for bit: the refine's
arithmetic is the direct kernel's, and what the filter leaves out must not have won.
Windows, stores, runs of every slot count, several runs per (A, C), padding, descending B,
early samples (whose runs do not expand), records that the traces leave, apertures where
everything ties, streamed, chunked and graph runs."""
import numpy as np
import pytest

import oracle
import semb
import synth

pytestmark = pytest.mark.gpu

STORES = {"f32": semb.STORE_F32, "f16": semb.STORE_F16, "bf16": semb.STORE_BF16}


def _survey(nb, tau, ns=600, apm=50, b1=1e-7, ncdp=9, fold=9, na=5, nc=5, az=0.0, seed=0):
    s = synth.crs_survey(seed=800 + nb + seed, ncdp=ncdp, noffsets=fold, ns=ns, na=na, nb=nb, nc=nc,
                         tau=tau * 0.002 * 1.0001, apm=apm, azimuth=az)
    s.params["b0"], s.params["b1"] = -b1, b1
    return s


def _arrays(s):
    g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float32)
    return semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                             g["scalco"], g["samples"])


def _kw(form, signed=False, **kw):
    kw["dm_mode"] = semb.DM_SIGNED if signed else semb.DM_ABS
    if form == "plain":
        return dict(mode=semb.PLAIN_F32, **kw)
    return dict(mode=semb.BATCHED, storage=STORES[form], repick=semb.REPICK_OFF, attrs=1, **kw)


def _results(p, form):
    p.run()
    out = list(p.download())
    if form != "plain":
        a = p.download_attrs()
        out += [a["sem2"], a["idx2"]]
    return out


def _compare(s, form, overflow=None, variant=None, **kw):
    """Filtered and unfiltered results of one plan; returns the unfiltered ones."""
    arr = _arrays(s)
    with semb.Plan(semb.params(semb.CRS, **_kw(form, **kw), **s.params)) as p:
        p.set_filter(semb.FILTER_ON)
        p.upload(arr.view())
        if variant is not None:
            p.set_variant(variant)
        tasks = p.filter_tasks()[0]
        assert tasks == p.ncdps * ((p.ns + 31) // 32)
        got = _results(p, form)
        direct = p.filter_tasks()[1]
        assert 0 <= direct <= tasks
        if overflow is not None:
            assert (direct > 0) == overflow, (direct, tasks)
        p.set_filter(semb.FILTER_OFF)
        assert p.filter_tasks() == (0, 0)
        ref = _results(p, form)
    for x, y in zip(got, ref):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f"), np.mean(x != y)
    return ref


# slots of 8 to 32 and their neighbours, two and three runs per (A, C)
RUNS = [(2, 1), (12, 1), (13, 1), (16, 1), (17, 1), (21, 1), (22, 1), (23, 1), (31, 1), (32, 1), (33, 1), (45, 1),
        (70, 1), (8, 2), (9, 2), (13, 2), (14, 2), (15, 2), (22, 2), (25, 2), (47, 2)]


@pytest.mark.parametrize("form", ["plain", "f16", "bf16", "f32"])
@pytest.mark.parametrize("nb,tau", RUNS)
def test_runs_of_every_length(nb, tau, form):
    ref = _compare(_survey(nb, tau, ns=601 if nb % 2 else 608, na=3), form)
    assert np.mean(ref[1] > 0) > 0.5


@pytest.mark.parametrize("nb", [3, 12, 31, 40])
def test_one_sample_windows(nb):
    _compare(_survey(nb, 0, ns=610), "plain")


@pytest.mark.parametrize("form", ["plain", "f16", "f32"])
@pytest.mark.parametrize("case", [dict(b1=-1e-7), dict(b1=2e-7), dict(b1=4e-8, ns=300), dict(apm=100, b1=4e-8),
                                  dict(fold=40, ncdp=5, ns=650), dict(ncdp=1, fold=3)],
                         ids=str)
@pytest.mark.parametrize("signed", [False, True])
@pytest.mark.parametrize("tau", [1, 2])
def test_geometries(case, form, signed, tau):
    _compare(_survey(21, tau, az=30.0 if signed else 0.0, **case), form, signed=signed)


def _spikes(r, ns, repeat, ncdp, fold, spacing, noise, early):
    """Traces of isolated spikes in next to no noise, each geometry `repeat` times: where a
    traveltime comes near a spike, the next interval's slopes are all that counts."""
    cdp, off = np.divmod(np.arange(ncdp * fold).repeat(repeat), fold)
    mx, half = np.round(10 * spacing * cdp).astype(int), r.choice([0, 100, 2000]) + 100 * off
    n = len(mx)
    base = np.zeros(ns)
    base[r.integers(0, ns // 3 if early else ns, 12)] = 1.0
    amp = 1.0 + 0.3 * r.standard_normal((n, 1))
    smp = (amp * base + noise * r.standard_normal((n, ns))).astype(np.float32)
    z = np.zeros(n, np.int32)
    return semb.GatherArrays((1 + np.arange(ncdp)) * fold * repeat, ns, 4000, (mx + half).astype(np.int32), z,
                             (mx - half).astype(np.int32), z, np.full(n, -10, np.int32), smp)


@pytest.mark.parametrize("ns,repeat,ncdp,fold,spacing,apm,tau,na,nb,nc,amax,bmax,noise,early", [
    (1500, 128, 5, 2, 5, 11, 1, 4, 9, 5, 3e-4, 1e-8, 1e-5, False),
    (600, 1, 3, 17, 5, 21, 0, 4, 31, 7, 1e-5, 1e-8, 1e-5, False),
    (300, 1, 5, 4, 5, 11, 0, 4, 5, 3, 1e-5, 4e-7, 1e-5, False),
    (1000, 1, 2, 11, 12.5, 51, 0, 7, 31, 9, 1e-6, 1e-7, 1e-5, False),
    (600, 1, 3, 6, 12.5, 13, 0, 4, 9, 12, 1e-5, 1.2e-6, 1e-6, True),
    (600, 1, 5, 19, 12.5, 26, 1, 6, 31, 4, 1e-6, 2.8e-7, 1e-6, True),
    (300, 40, 2, 1, 12.5, 51, 2, 3, 13, 12, 3e-4, 1.4e-8, 1e-5, True)])
@pytest.mark.parametrize("form", ["plain", "f32"])
def test_spikes_next_to_a_traveltime(form, ns, repeat, ncdp, fold, spacing, apm, tau, na, nb, nc, amax, bmax, noise, early):
    if form != "plain":
        tau = max(tau, 1)
    prm = dict(a0=-amax, a1=amax, na=na, b0=-bmax, b1=bmax, nb=nb, c0=4e-7, c1=6e-7, nc=nc, aph=4000, apm=apm,
               tau=tau * 0.004 * 1.0001, azimuth=0.0)
    bad = 0
    with semb.Plan(semb.params(semb.CRS, **_kw(form), **prm)) as p:
        for seed in range(60):
            arr = _spikes(np.random.default_rng(seed), ns, repeat, ncdp, fold, spacing, noise, early)
            p.set_filter(semb.FILTER_ON)
            p.upload(arr.view())
            assert p.filter_tasks()[0] > 0
            got = _results(p, form)
            p.set_filter(semb.FILTER_OFF)
            bad += sum(int((x != y).sum()) for x, y in zip(got, _results(p, form)))
    assert bad == 0


@pytest.mark.parametrize("form", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("tau", [1, 2])
def test_chunks_end_where_the_direct_kernel_s_do(tau, seed, form):
    """Folds of several staged chunks: the refine folds its energies at the same traces."""
    _compare(_survey(21, tau, az=30.0, ncdp=25, fold=17, ns=777, seed=seed), form, signed=True)


class _Scattered:
    """Pairs of CDPs 1 km apart.  The second CDP's traces, `nfar` of them, lie far from its
    first trace's midpoint, with offsets that take them to the record's end: their runs are
    wide, their expansion needs its second order, and no other trace of a chunk does."""

    def __init__(self, seed, npairs=48, nnear=2, nfar=400, ns=300, far=105, spread=0):
        r = np.random.default_rng(seed)
        n = npairs * (nnear + 1 + nfar)
        self.ns, self.ncdp = ns, 2 * npairs
        mx, half = np.empty(n), np.empty(n)
        end, q = [], 0
        for k in range(npairs):
            mx[q:q + nnear] = 1000 * k
            half[q:q + nnear] = 20
            q += nnear
            end.append(q)
            mx[q] = 1000 * k + 49
            half[q] = 20
            mx[q + 1:q + 1 + nfar] = 1000 * k + far + r.integers(-spread, spread + 1, nfar)
            half[q + 1:q + 1 + nfar] = 320 + r.integers(-spread, spread + 1, nfar)
            q += 1 + nfar
            end.append(q)
        self.sx, self.gx = (mx - half).astype(np.int32), (mx + half).astype(np.int32)
        t = np.arange(ns)
        w = sum(np.sin(2 * np.pi * (f * t[None] + r.random((npairs, 1)))) for f in (0.31, 0.37, 0.43))
        pair = np.repeat(np.arange(npairs), nnear + 1 + nfar)
        self.samples = (w[pair] + 0.05 * r.standard_normal((n, ns))).astype(np.float32)
        self.end = end
        self.params = dict(a0=-1e-4, a1=1e-4, na=5, b0=-9e-8, b1=9e-8, nb=21, c0=0.95e-6, c1=1.05e-6, nc=9, aph=1000,
                           apm=50, tau=0.0021, azimuth=0.0)

    def arrays(self):
        z = np.zeros(len(self.sx), np.int32)
        return semb.GatherArrays(self.end, self.ns, 2000, self.gx, z, self.sx, z, z + 1, self.samples)


@pytest.mark.parametrize("form", ["plain", "f32", "f16"])
@pytest.mark.parametrize("seed,spread", [(0, 0), (1, 0), (2, 1), (3, 2)])
def test_wide_runs_at_the_record_s_end(seed, spread, form):
    s = _Scattered(seed, spread=spread)
    with semb.Plan(semb.params(semb.CRS, **_kw(form), **s.params)) as p:
        p.set_filter(semb.FILTER_ON)
        p.upload(s.arrays().view())
        assert p.filter_tasks()[0] > 0
        got = _results(p, form)
        p.set_filter(semb.FILTER_OFF)
        ref = _results(p, form)
    for x, y in zip(got, ref):
        assert np.array_equal(x, y), np.mean(x != y)


@pytest.mark.parametrize("variant", [10, 13, 14, 28, 30, 31, 32, 33])
def test_every_filtered_variant(variant):
    s = _survey(21, 1)
    arr = _arrays(s)
    with semb.Plan(semb.params(semb.CRS, **_kw("f16"), **s.params)) as p:
        p.set_filter(semb.FILTER_ON)
        p.upload(arr.view())
        p.set_variant(variant)
        if p.filter_tasks()[0] == 0:
            assert variant == 10   # a kernel without the pipelined staging
            return
    _compare(s, "f16", variant=variant)


@pytest.mark.parametrize("tau,variant", [(1, 16), (1, 17), (1, 18), (2, 16)])
@pytest.mark.parametrize("form", ["f16", "f32"])
def test_variants_that_do_not_stage_whole_windows_have_no_filter(form, tau, variant):
    """Their long windows come from the FP32 store and end no chunk, which the refine does not
    repeat: forced, they evaluate every candidate."""
    s = synth.crs_survey(seed=72, ncdp=8, noffsets=24, ns=1500, dt_us=4000, na=1, nb=21, nc=5,
                         tau=tau * 0.004 * 1.0001, aph=2600, apm=50)
    s.params["c1"] *= 30.0   # a pass spans hundreds of samples
    arr = _arrays(s)
    with semb.Plan(semb.params(semb.CRS, **_kw(form), **s.params)) as p:
        p.set_filter(semb.FILTER_ON)
        p.upload(arr.view())
        p.set_staging(128)
        assert p.filter_tasks()[0] > 0
        p.set_variant(variant)
        got = _results(p, form)
        assert p.filter_tasks() == (0, 0)
        p.set_filter(semb.FILTER_OFF)
        ref = _results(p, form)
    for x, y in zip(got, ref):
        assert np.array_equal(x, y), (np.mean(x != y), np.abs(x - y).max())


@pytest.mark.parametrize("form", ["plain", "f16", "bf16", "f32"])
def test_apertures_of_one_cdp_overflow_into_the_direct_kernel(form):
    """Every A and B ties: no list holds them all."""
    _compare(_survey(21, 1, apm=5, ncdp=3, na=9), form, overflow=True)


@pytest.mark.parametrize("form", ["plain", "f16", "f32"])
def test_no_valid_candidate(form):
    s = _survey(21, 1)
    s.params["c0"] *= 400.0
    s.params["c1"] *= 400.0
    ref = _compare(s, form, overflow=False)
    assert np.any(ref[1] == 0)


@pytest.mark.parametrize("form", ["plain", "f32"])
def test_zero_and_non_finite_traces(form):
    s = _survey(21, 1)
    s.samples[3] = 0.0
    s.samples[20, 100] = np.inf
    s.samples[41, 150] = np.nan
    s.samples[60] *= 1e-12
    s.samples[:, 400:430] = 0.0
    _compare(s, form)


@pytest.mark.parametrize("form", ["f16", "f32"])
@pytest.mark.parametrize("tau", [1, 2])
def test_streamed_chunked_and_graph_runs(form, tau):
    s = _survey(21, tau, ncdp=14)
    arr = _arrays(s)
    with semb.Plan(semb.params(semb.CRS, **_kw(form), **s.params)) as p:
        p.set_filter(semb.FILTER_OFF)
        p.upload(arr.view())
        ref = _results(p, form)[:3]

        def same():
            assert p.filter_tasks()[0] > 0
            for x, y in zip(p.download(), ref):
                assert np.array_equal(x, y)

        p.set_filter(semb.FILTER_ON)
        for _ in range(2):   # captured, replayed
            p.use_graph(True)
            p.run()
            same()
        p.use_graph(False)
        for _ in range(2):
            p.set_chunks(4)
            p.run()
            same()
        p.set_chunks(0)
        p.stream(arr.view(), 3)
        same()


@pytest.mark.parametrize("form", ["plain", "f16"])
def test_default_use(form):
    """Where it pays: the 21 x 21 x 21 grid, not a 3 x 3 x 3 one or one B value, never CMP."""
    def tasks(signed=False, azimuth=0.0, **kw):
        s = _survey(ns=600, tau=1, ncdp=3, **kw)
        s.params["azimuth"] = azimuth
        with semb.Plan(semb.params(semb.CRS, **_kw(form, signed), **s.params)) as p:
            p.upload(_arrays(s).view())
            return p.filter_tasks()[0]

    assert tasks(na=21, nb=21, nc=21) > 0
    assert tasks(na=3, nb=3, nc=3) == 0
    assert tasks(na=21, nb=1, nc=21) == 0
    # apertures in which no traveltime depends on A (batched form): one CDP; a line across the
    # azimuth
    pays = form == "plain"
    assert (tasks(na=21, nb=21, nc=21, apm=5) > 0) == pays
    assert (tasks(na=21, nb=21, nc=21, azimuth=90.0, signed=True) > 0) == pays
    assert tasks(na=21, nb=21, nc=21, azimuth=30.0, signed=True) > 0
    assert tasks(na=1, nb=21, nc=441, apm=5) > 0
    s = synth.cmp_survey(seed=1, ncmp=2, half_offsets=np.linspace(10.0, 300.0, 20), ns=320, nc=64, tau=0.0021)
    g = oracle.gather(s.headers, s.samples, "cmp", s.params["aph"])
    arr = semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                            g["scalco"], g["samples"])
    with semb.Plan(semb.params(semb.CMP, mode=semb.PLAIN_F32, **s.params)) as p:
        with pytest.raises(semb.SembError):
            p.filter_tasks()   # before the upload
        with pytest.raises(semb.SembError):
            p.set_filter(3)
        p.set_filter(semb.FILTER_ON)
        p.upload(arr.view())
        assert p.filter_tasks() == (0, 0)
