"""CUDA calls that fail once while a step graph is set up or captured (a shim
preloaded into a child process returns the error, on the host): the run
returns an error, and the next one gives what a fresh context gives."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>
static int armed, seen;
/* the nth call of that name from now on fails, once */
static char name[64];
static int nth;
void shim_arm(const char* which, int n) { strncpy(name, which, sizeof name - 1); nth = n; seen = 0; armed = 1; }
int shim_fired(void) { return !armed; }
static int due(const char* which)
{
    if (!armed || strcmp(which, name) || ++seen != nth) return 0;
    armed = 0;
    return 1;
}
static void* real(const char* which) { return dlsym(dlopen("libcudart.so.13", RTLD_NOW), which); }
int cudaStreamCreateWithFlags(void** s, unsigned f)
{
    if (due("cudaStreamCreateWithFlags")) return 2;
    return ((int (*)(void**, unsigned))real("cudaStreamCreateWithFlags"))(s, f);
}
int cudaEventCreateWithFlags(void** e, unsigned f)
{
    if (due("cudaEventCreateWithFlags")) return 2;
    return ((int (*)(void**, unsigned))real("cudaEventCreateWithFlags"))(e, f);
}
int cudaEventRecord(void* e, void* s)
{
    if (due("cudaEventRecord")) return 2;
    return ((int (*)(void*, void*))real("cudaEventRecord"))(e, s);
}
int cudaStreamWaitEvent(void* s, void* e, unsigned f)
{
    if (due("cudaStreamWaitEvent")) return 2;
    return ((int (*)(void*, void*, unsigned))real("cudaStreamWaitEvent"))(s, e, f);
}
"""

CHILD = r"""
import ctypes, sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import numpy as np
import systems as S
nbg = S.nbg
shim = ctypes.CDLL(sys.argv[2])
sim = S.water_box(11, seed=3, thermostat=nbg.BerendsenThermostat(300.0, 0.1))
desc, keep = nbg.system_descriptor(sim)
u, v = S.state(sim)
ref = nbg.Engine(desc, 0).run(u, v, 5e-4, 37, 0)
eng = nbg.Engine(desc, 0)
shim.shim_arm(sys.argv[3].encode(), int(sys.argv[4]))
try:
    eng.run(u, v, 5e-4, 37, 0)
    raised = False
except nbg.EngineError as e:
    raised = True
    print(e)
assert shim.shim_fired() and raised
got = eng.run(u, v, 5e-4, 37, 0)
for k in range(2):
    np.testing.assert_array_equal(got[k], ref[k])
print("ok")
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    src, lib = d / "shim.c", d / "libshim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(lib), "-ldl"], check=True)
    return str(lib)


# setting up: the side stream and the two events of the fork and the join;
# capturing: calls of the first steps' forks and joins (the first record is
# the run's own)
@pytest.mark.parametrize("call,nth", [("cudaStreamCreateWithFlags", 1), ("cudaEventCreateWithFlags", 1),
                                      ("cudaEventCreateWithFlags", 2), ("cudaEventRecord", 2), ("cudaEventRecord", 3),
                                      ("cudaEventRecord", 4), ("cudaEventRecord", 5), ("cudaStreamWaitEvent", 1),
                                      ("cudaStreamWaitEvent", 2), ("cudaStreamWaitEvent", 3)])
def test_next_run_after_a_failed_call(gpu, shim, call, nth):
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, shim, call, str(nth)], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": shim})
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
