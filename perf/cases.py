"""The searches that users of this framework run, as timed cases.

A case is one kind of call over a seeded synthetic survey (25 Hz events on the search
operator's traveltimes plus noise, as field data looks to the search): the method (CMP or
CRS), the form (the plain single-precision search that the command lines run, or the
batched search with a 16-bit or FP32 trace store), the grid, the window, the record, and
how the call is made:

    resident   the survey is on the device; a pass searches it and reads the picks back
               (velocity analysis over several grids, re-runs, the benchmark's step)
    upload     a pass takes a host gather through upload, search and download
    su         a pass takes SU bytes through grouping, upload, search and download
    stream     a pass takes a host gather through the streamed upload-and-search

Inputs and results live in page-locked host memory, as a program that streams surveys
keeps them.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ipdps-crs-cmp-code_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import semb  # noqa: E402
import synth  # noqa: E402

_STORE = {"f32": semb.STORE_F32, "f16": semb.STORE_F16, "bf16": semb.STORE_BF16}


def _case(**kw):
    c = dict(method="cmp", form="plain", store="f16", call="resident", ncdp=1, fold=60, fold_lo=0, fold_hi=0, ns=1000,
             dt_us=2000, tau=1, na=0, nb=0, nc=101, apm=0, signed=False, ngen=0, chunks=0)
    c.update(kw)
    return c


def listed():
    return [
        # One CMP gather from SU bytes to picks, as an interactive velocity-analysis tool
        # does for each gather it shows: launches, copies and set-up count.
        _case(name="cmp-gather-su", call="su"),
        # The 200-CMP, 60-fold line with 101 velocities in the command line's form.
        _case(name="cmp-line-plain", ncdp=200),
        # The same line, batched with the FP16 store.
        _case(name="cmp-line-f16", ncdp=200, form="batched"),
        # A stretch of the 4096-CMP line (fold 12 to 240, 256 velocities, w = 5), host
        # gather to picks with the copies overlapped: production velocity analysis.
        _case(name="cmp-uneven-stream", form="batched", call="stream", chunks=4, ncdp=256, fold_lo=12, fold_hi=240,
              ns=2000, tau=2, nc=256),
        # The same kind of line in the command line's form.
        _case(name="cmp-uneven-plain", ncdp=160, fold_lo=12, fold_hi=240, ns=2000, tau=2, nc=256),
        # A wide window (w = 11) on an odd record length: low-frequency data, BF16 store.
        _case(name="cmp-wide-bf16", form="batched", store="bf16", ncdp=75, fold=37, ns=751, tau=5, nc=90),
        # The 48-offset CRS line with the 21 x 21 x 21 grid, command line's form.
        _case(name="crs-line-plain", method="crs", ncdp=12, fold=48, na=21, nb=21, nc=21, apm=50),
        # The same line, batched with the FP16 store.
        _case(name="crs-line-f16", method="crs", form="batched", ncdp=64, fold=48, na=21, nb=21, nc=21, apm=50),
        # Blocks of the 20,000-CDP survey with apertures of 50 to 2000 traces: the
        # production CRS search.
        _case(name="crs-uneven-f16", method="crs", form="batched", ncdp=128, fold_lo=50, fold_hi=2000, ns=1500,
              dt_us=4000, na=21, nb=21, nc=21, apm=150),
        # Blocks of the 100,000-CDP survey: BF16 store and the 31 x 31 x 31 grid.
        _case(name="crs-uneven31-bf16", method="crs", form="batched", store="bf16", ncdp=48, fold_lo=50, fold_hi=2000,
              ns=1500, dt_us=4000, na=31, nb=31, nc=31, apm=150),
        # A refinement search: small ragged grid, w = 5, signed midpoint displacement and
        # the FP32 store, host gather to picks.
        _case(name="crs-refine-w5-f32", method="crs", form="batched", store="f32", call="upload", ncdp=24, fold=28,
              ns=601, tau=2, na=9, nb=13, nc=5, apm=75, signed=True),
        # CRS by differential evolution, the optimiser that replaces the grid.
        _case(name="crs-de", method="crs", ncdp=8, fold=24, ns=500, na=6, nb=5, nc=6, apm=50, ngen=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cmp", "cmp", "cmp-uneven", "crs", "crs", "crs-uneven", "crs-de"])
    most = 1.6e11   # trace-evaluations: well below the largest listed case
    for _ in range(1000):
        c = _case(form=rng.choice(["plain", "batched"]), store=rng.choice(["f16", "f16", "bf16", "f32"]),
                  call=rng.choice(["resident", "resident", "upload"]), ns=_log(rng, 300, 2000),
                  dt_us=rng.choice([2000, 2000, 4000]), tau=rng.choice([0, 1, 1, 1, 2, 2]))
        if kind == "cmp":
            c.update(ncdp=_log(rng, 1, 300), fold=_log(rng, 6, 200), nc=_log(rng, 20, 300))
            if rng.random() < 0.2:
                c["tau"] = rng.randint(3, 7)
        elif kind == "cmp-uneven":
            lo = _log(rng, 4, 40)
            c.update(ncdp=_log(rng, 20, 300), fold_lo=lo, fold_hi=lo * rng.randint(2, 12), nc=_log(rng, 40, 300))
        elif kind == "crs-de":
            c.update(method="crs", form="plain", ncdp=_log(rng, 1, 12), ns=_log(rng, 300, 600),
                     na=rng.randint(3, 6), nb=rng.randint(3, 6), nc=rng.randint(3, 7), apm=rng.choice([25, 50, 75]),
                     ngen=rng.randint(5, 25))
            c["fold"] = _log(rng, 6, int(24e-6 * c["ns"] * c["dt_us"]))
        else:
            c.update(method="crs", ncdp=_log(rng, 4, 96), na=rng.randint(5, 31), nb=rng.randint(5, 31),
                     nc=rng.randint(5, 31), signed=rng.random() < 0.2)
            if kind == "crs":
                c.update(fold=_log(rng, 6, int(24e-6 * c["ns"] * c["dt_us"])), apm=rng.choice([25, 50, 75, 100]))
            else:
                c.update(fold_lo=50, fold_hi=_log(rng, 200, 2000), apm=150)
        if c["form"] == "batched" and rng.random() < 0.2:
            c.update(call="stream", chunks=rng.randint(2, 8))
        if 2e6 <= _trace_evals(c) * (1 if c["form"] == "batched" and not c["ngen"] else 3) <= most:
            return c
    return _case(ncdp=rng.randint(20, 200), fold=rng.randint(10, 80))


def _fold(c):
    """Mean traces of a CDP and mean aperture."""
    if c["method"] == "cmp":
        lo, hi = c["fold_lo"], c["fold_hi"]
        f = (hi - lo) / math.log(hi / lo) if lo else c["fold"]
        return f, f
    if c["fold_lo"]:
        ap = (c["fold_hi"] - c["fold_lo"]) / math.log(c["fold_hi"] / c["fold_lo"])
        return max(2.0, ap / 9.0), ap
    nn = sum(1 for d in range(-c["ncdp"], c["ncdp"] + 1) if abs(d) * 12.5 <= c["apm"])
    nn = min(nn, c["ncdp"])
    return float(c["fold"]), float(c["fold"] * nn)


def _ncand(c):
    return c["nc"] if c["method"] == "cmp" else c["na"] * c["nb"] * c["nc"]


def _trace_evals(c):
    return float(c["ncdp"]) * c["ns"] * _ncand(c) * _fold(c)[1] * (1 + c["ngen"])


def work(case):
    """Each sample of the gather read once and each result written once; the operations
    of the semblance definition (traveltime, interpolation, numerators, energy, linear
    sum per trace and window sample)."""
    c = case
    f, ap = _fold(c)
    w = 2 * c["tau"] + 1
    evals = float(c["ncdp"]) * c["ns"] * _ncand(c) * (1 + c["ngen"])
    t = 5 if c["method"] == "cmp" else 10
    return {"bytes": 4.0 * c["ncdp"] * c["ns"] * f + 12.0 * c["ncdp"] * c["ns"],
            "flops": evals * (ap * (t + 7 * w) + 2 * w + 2)}


def _survey(c, seed):
    # the spread grows with the record, as in the field: most traveltimes stay inside it
    dt = c["dt_us"] * 1e-6
    rec = c["ns"] * dt
    kw = dict(seed=seed, ns=c["ns"], dt_us=c["dt_us"], nc=c["nc"], tau=c["tau"] * dt * (1 + 1e-4))
    if c["method"] == "cmp":
        if c["fold_lo"]:
            return synth.cmp_survey(ncmp=c["ncdp"], fold_range=(c["fold_lo"], c["fold_hi"]), hmax=750.0 * rec, aph=3200,
                                    nevents=8, **kw)
        return synth.cmp_survey(ncmp=c["ncdp"], half_offsets=np.linspace(25.0, 381.0 * rec, c["fold"]), aph=3200, **kw)
    kw.update(na=c["na"], nb=c["nb"], apm=c["apm"], ncdp=c["ncdp"])
    if c["fold_lo"]:
        return synth.crs_survey(aperture_range=(c["fold_lo"], c["fold_hi"]), block=16,
                                aph=int(433.0 * rec), azimuth=90.0, nevents=6, **kw)
    return synth.crs_survey(noffsets=min(c["fold"], int(24 * rec)), aph=1300, **kw)


class _State:
    """A survey in page-locked host memory, the plan that searches it and the buffers of
    its results."""

    def __init__(self, c, seed):
        s = _survey(c, seed)
        self.c = c
        h = s.headers
        n = c["ncdp"] * c["ns"]
        kw = {} if c["method"] == "cmp" else dict(dm_mode=semb.DM_SIGNED if c["signed"] else semb.DM_ABS, ngen=c["ngen"])
        mode = semb.BATCHED if c["form"] == "batched" else semb.PLAIN_F32
        p = {k: v for k, v in s.params.items()}
        self.plan = semb.Plan(semb.params(semb.CMP if c["method"] == "cmp" else semb.CRS, mode=mode,
                                          storage=_STORE[c["store"]], **p, **kw))
        self.aph = int(p["aph"])
        self.out = [self._pin(n, torch.int32), self._pin(n, torch.float32), self._pin(n, torch.float32)]
        if c["call"] == "su":
            raw = _su_bytes(h, s.samples)
            self.bytes = self._pin(len(raw), torch.uint8)
            self.bytes[:] = np.frombuffer(raw, np.uint8)
        else:
            smp = self._pin(s.samples.size, torch.float32).reshape(s.samples.shape)
            smp[:] = s.samples
            end = np.cumsum(np.bincount(h["cdp"] - 1, minlength=c["ncdp"]))
            self.gather = semb.GatherArrays(end, c["ns"], c["dt_us"], h["gx"], h["gy"], h["sx"], h["sy"], h["scalco"],
                                            smp)
            self.view = self.gather.view()
            if c["call"] == "resident":
                self.plan.upload(self.view)

    @staticmethod
    def _pin(n, dtype):
        return torch.empty(n, dtype=dtype, pin_memory=True).numpy()

    def __del__(self):
        if getattr(self, "plan", None) is not None:
            self.plan.close()


def _su_bytes(headers, samples):
    rows = np.empty((len(headers), 240 + 4 * samples.shape[1]), np.uint8)
    rows[:, :240] = np.ascontiguousarray(headers).view(np.uint8).reshape(len(headers), 240)
    rows[:, 240:] = np.ascontiguousarray(samples, np.float32).view(np.uint8)
    return rows.tobytes()


def prepare(case, seed):
    return _State(dict(case), int(seed) % (1 << 31))


def run(state):
    c, plan = state.c, state.plan
    if c["call"] == "su":
        s = semb.Survey.from_bytes(state.bytes, semb.CMP if c["method"] == "cmp" else semb.CRS, state.aph)
        plan.upload(s.view())
        plan.run()
        s.close()
    elif c["call"] == "stream":
        plan.stream(state.view, c["chunks"])
    else:
        if c["call"] == "upload":
            plan.upload(state.view)
        plan.run()
    ctr, sem, stk = plan.download(*state.out)
    if c["ngen"]:
        a, b, cc = plan.download_abc()
        return {"a": a, "b": b, "c": cc, "sem": sem, "stk": stk}
    return {"ctr": ctr, "sem": sem, "stk": stk}


def exact(case, seed):
    """Semblance and stack of the best candidate per (CDP, t0) in 64 bits, straight from
    the definition."""
    c = dict(case)
    if c["ngen"] or _trace_evals(c) > 1.2e10:
        return None
    s = _survey(c, int(seed) % (1 << 31))
    dev = "cuda"
    h = s.headers
    f8 = np.float64
    sc = np.where(h["scalco"] == 0, 1.0, np.where(h["scalco"] < 0, 1.0 / np.minimum(h["scalco"], -1).astype(f8), h["scalco"]))
    gx, gy, sx, sy = (h[k].astype(f8) for k in ("gx", "gy", "sx", "sy"))
    hh = 0.25 * (((gx - sx) * sc) ** 2 + ((gy - sy) * sc) ** 2) / 1e6
    mx, my = (gx + sx) * sc * 0.5, (gy + sy) * sc * 0.5
    end = np.cumsum(np.bincount(h["cdp"] - 1, minlength=c["ncdp"]))
    beg = np.concatenate([[0], end[:-1]])
    dt = c["dt_us"] / 1e6
    ns, tau, w = c["ns"], c["tau"], 2 * c["tau"] + 1
    p = s.params
    if c["method"] == "cmp":
        c0, c1 = float(np.float32(p["c0"])) * 1e6, float(np.float32(p["c1"])) * 1e6
        A = B = np.zeros(c["nc"])
        C = c0 + (c1 - c0) * (1.0 / c["nc"]) * np.arange(c["nc"])
    else:
        ia, ib, ic = np.meshgrid(np.arange(c["na"]), np.arange(c["nb"]), np.arange(c["nc"]), indexing="ij")
        A = (p["a0"] + (p["a1"] - p["a0"]) / c["na"] * ia).ravel()
        B = (p["b0"] + (p["b1"] - p["b0"]) / c["nb"] * ib).ravel()
        C = (p["c0"] * 1e6 + (p["c1"] - p["c0"]) * 1e6 / c["nc"] * ic).ravel()
    ncand = len(C)
    tens = lambda v: torch.tensor(np.ascontiguousarray(v, f8), device=dev)  # noqa: E731
    T = tens(np.arange(ns) * dt)[None, :]
    smp = torch.tensor(s.samples, device=dev).double()
    az = math.radians(float(p.get("azimuth", 0.0)))
    fsc = np.float32(1.0) / np.float32(-100.0)
    fm = [((np.float32(1) * fsc) * (h["gx"][beg] + h["sx"][beg]).astype(np.float32)) * np.float32(0.5),
          ((np.float32(1) * fsc) * (h["gy"][beg] + h["sy"][beg]).astype(np.float32)) * np.float32(0.5)]
    sem_o, stk_o = np.zeros((c["ncdp"], ns)), np.zeros((c["ncdp"], ns))
    per = max(1, min(ncand, 3_000_000 // ns))
    for i in range(c["ncdp"]):
        if c["method"] == "cmp":
            tr = np.arange(beg[i], end[i])
            dm, dm2 = np.zeros(len(tr)), np.zeros(len(tr))
        else:
            dx, dy = fm[0] - fm[0][i], fm[1] - fm[1][i]
            near = np.nonzero(dx * dx + dy * dy <= np.float32(c["apm"] * c["apm"]))[0]
            tr = np.concatenate([np.arange(beg[j], end[j]) for j in near])
            ddx, ddy = mx[tr] - mx[beg[i]], my[tr] - my[beg[i]]
            if c["signed"]:
                dm = ddx * math.cos(az) + ddy * math.sin(az)
                dm2 = dm * dm
            else:
                dm2 = ddx * ddx + ddy * ddy
                dm = np.sqrt(dm2)
        best = torch.zeros(ns, dtype=torch.float64, device=dev)
        bstk = torch.zeros_like(best)
        stt00 = 0.0
        for q in range(0, ncand, per):
            a, b, cc = (tens(v[q:q + per])[:, None] for v in (A, B, C))
            num = [torch.zeros((a.shape[0], ns), dtype=torch.float64, device=dev) for _ in range(w)]
            den, mm = torch.zeros_like(num[0]), torch.zeros_like(num[0])
            for k, m, m2 in zip(tr, dm, dm2):
                t2 = (T + a * float(m)) ** 2 + b * float(m2) + cc * float(hh[k])
                t = torch.where(t2 < 0, -1.0, t2.clamp(min=0).sqrt()) / dt
                it = t.clamp(-2, ns + 2).to(torch.int64)
                ok = (t >= tau) & (it + tau + 1 < ns)
                x = torch.where(ok, t - it, 0.0)
                it = torch.where(ok, it - tau, 0)
                okd = ok.double()
                s0 = smp[k][it]
                for j in range(w):
                    s1 = smp[k][it + j + 1] if ns > w else s0
                    v = ((s1 - s0) * x + s0) * okd
                    num[j] += v
                    den += v * v
                    s0 = s1
                mm += okd
            good = (den > 1e-13) & (mm > 0) & (len(tr) - mm < 2)
            dm_ = torch.where(good, den * mm, 1.0)
            sem = torch.where(good, sum(n * n for n in num) / dm_, -1.0)
            stk = torch.where(good, sum(num) / (w * mm.clamp(min=1)), 0.0)
            if q == 0:
                stt00 = float(stk[0, 0])
            v, at = sem.max(dim=0)
            won = v > best
            bstk = torch.where(won, stk.gather(0, at[None])[0], bstk)
            best = torch.where(won, v, best)
        if c["method"] == "crs":
            bstk = torch.where(best > 0, bstk, torch.full_like(bstk, stt00))
        sem_o[i], stk_o[i] = best.cpu().numpy(), bstk.cpu().numpy()
    return {"ctr": None, "sem": sem_o, "stk": stk_o}
