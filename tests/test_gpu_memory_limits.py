"""A plan near the end of the device's memory (GPU).  The CRS filter's lists and the re-pick's
paired geometry are optional: what a plan needs later (the chunk table, another variant's
candidate table, an autotuner's sample, a second upload) takes their place where nothing
else is left.  The limit is one that a cudaMalloc in front of CUDA's sets in a child
process: it refuses what would go beyond it."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r'''
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdio.h>
#define N 65536
static struct { void* p; size_t n; } held[N];
static size_t total, limit = (size_t)-1;
static int refused;
/* the library's own CUDA runtime, which is not in the global scope */
static void* of_cudart(const char* name) {
  void* lib = dlopen("libcudart.so.13", RTLD_LAZY);
  return lib ? dlsym(lib, name) : 0;
}
size_t shim_total(void) { return total; }
int shim_refused(void) { return refused; }
void shim_limit(size_t n) { limit = n; refused = 0; }
int cudaMalloc(void** p, size_t n) {
  static int (*real)(void**, size_t);
  if (!real) real = (int (*)(void**, size_t))of_cudart("cudaMalloc");
  if (total + n > limit) {
    ++refused;
    return 2;   /* cudaErrorMemoryAllocation */
  }
  int rc = real(p, n);
  for (int i = 0; rc == 0 && i < N; ++i)
    if (!held[i].p) {
      held[i].p = *p;
      held[i].n = n;
      total += n;
      break;
    }
  return rc;
}
int cudaFree(void* p) {
  static int (*real)(void*);
  if (!real) real = (int (*)(void*))of_cudart("cudaFree");
  for (int i = 0; p && i < N; ++i)
    if (held[i].p == p) {
      held[i].p = 0;
      total -= held[i].n;
      break;
    }
  return real(p);
}
'''

CHILD = r'''
import ctypes, sys
import numpy as np
import oracle, semb, synth
shim = ctypes.CDLL(sys.argv[1])
shim.shim_total.restype = ctypes.c_size_t
shim.shim_limit.argtypes = [ctypes.c_size_t]
what, form = sys.argv[2], sys.argv[3]

def arrays(ncdp):
    s = synth.crs_survey(seed=5, ncdp=ncdp, noffsets=9, ns=600, na=9, nb=21, nc=9, tau=0.0021)
    g = oracle.gather(s.headers, s.samples, "crs", s.params["aph"], s.params["apm"], real=np.float32)
    return s, semb.GatherArrays(g["ntraces_by_cdp_id"], g["ns"], g["dt_us"], g["gx"], g["gy"], g["sx"], g["sy"],
                                g["scalco"], g["samples"])

s, arr = arrays(12)
kw = dict(mode=semb.PLAIN_F32) if form == "plain" else dict(mode=semb.BATCHED)
with semb.Plan(semb.params(semb.CRS, **kw, **s.params)) as p:
    p.upload(arr.view())
    p.run()
    ref = [x.copy() for x in p.download()]
    assert p.filter_tasks()[0] > 0
    if what == "graph":
        p.use_graph(True)
        p.run()
    if what == "reupload":
        p.close()
        p = semb.Plan(semb.params(semb.CRS, **kw, **s.params))
        small = arrays(8)[1]
        p.upload(small.view())
        p.run()
    shim.shim_limit(shim.shim_total() + (0 if what != "reupload" else 250000))
    if what in ("chunks", "graph"):
        p.set_chunks(5) if what == "chunks" else p.set_variant(p.stats()["variant"])
    elif what == "variant":
        p.set_variant(1 if form == "plain" else 13)
    elif what == "autotune":
        p.autotune()
    elif what == "reupload":
        p.upload(arr.view())
    assert shim.shim_refused() > 0 or what == "chunks"
    for _ in range(2):
        p.run()
        assert shim.shim_refused() > 0
        ctr, sem, stk = p.download()
        if what == "autotune" and form != "plain":
            continue   # whichever variant was fastest
        same = ctr == ref[0]
        assert np.mean(same) > 0.999, np.mean(same)
        np.testing.assert_allclose(sem, ref[1], rtol=1e-5, atol=2e-6)
        np.testing.assert_allclose(stk[same], ref[2][same], rtol=1e-5, atol=2e-6)
    p.close()
print("ok")
'''


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    d = tmp_path_factory.mktemp("shim")
    (d / "shim.c").write_text(SHIM)
    subprocess.run([cc, "-shared", "-fPIC", "-O1", "-o", str(d / "shim.so"), str(d / "shim.c"), "-ldl"], check=True)
    return str(d / "shim.so")


@pytest.mark.parametrize("what,form", [("chunks", "f16"), ("variant", "f16"), ("variant", "plain"), ("autotune", "f16"),
                                       ("autotune", "plain"), ("graph", "f16"), ("reupload", "f16"),
                                       ("reupload", "plain")])
def test_optional_buffers_give_way(shim, what, form):
    path = os.pathsep.join(os.path.join(ROOT, d) for d in ("ipdps-crs-cmp-code_gb300", "oracle", "tests"))
    env = dict(os.environ, LD_PRELOAD=shim, PYTHONPATH=path)
    r = subprocess.run([sys.executable, "-c", CHILD, shim, what, form], env=env, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
