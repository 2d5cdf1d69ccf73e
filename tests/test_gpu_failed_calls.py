"""A force call that fails after its charges were spread leaves no charge and
no pair force behind: the call after it gives the forces of a fresh context.
The failure is made on the host, by a library preloaded before cuFFT whose
execution entry returns an error once."""

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
int fail_r2c = 0, fail_c2r = 0;
typedef int (*exec_fn)(int, void *, void *);
static int run(const char *name, int *fail, int plan, void *in, void *out) {
  if (*fail > 0) { --*fail; return 6; }  /* CUFFT_EXEC_FAILED */
  void *cufft = dlopen("libcufft.so.11", RTLD_LAZY | RTLD_NOLOAD);  /* the one that is loaded */
  exec_fn f = cufft ? (exec_fn)dlsym(cufft, name) : 0;
  return f ? f(plan, in, out) : 5;  /* CUFFT_INTERNAL_ERROR */
}
int cufftExecR2C(int plan, void *in, void *out) { return run("cufftExecR2C", &fail_r2c, plan, in, out); }
int cufftExecC2R(int plan, void *in, void *out) { return run("cufftExecC2R", &fail_c2r, plan, in, out); }
"""

CHILD = r"""
import ctypes, os, sys
import torch
from mdir_b200 import NonbondedTerm, systems
from mdir_b200._lib import NativeError
shim = ctypes.CDLL(os.environ["LD_PRELOAD"])
deterministic, waters = sys.argv[1] == "1", int(sys.argv[2])
s = systems.tip3p(waters=waters, seed=2)
x = torch.tensor(s["positions"], device="cuda")
t = NonbondedTerm(len(s["charges"]))
t.set_particles(s["charges"], s["types"], s["sigma"], s["epsilon"])
t.set_exclusions(pairs=s["excluded_pairs"])
t.set_interaction(s["cutoff"], s["reach"], s["beta"])
t.set_pme(s["grid"], 4)
t.set_tuning(pme_fft="cufft")
t.set_deterministic(deterministic)
t.build(x, s["box"])
for energy in (False, True):
    want = t.force(x, energy=energy).clone()
    for entry in ("fail_r2c", "fail_c2r"):
        ctypes.c_int.in_dll(shim, entry).value = 1
        try:
            t.force(x, energy=energy)
            raise SystemExit("the call did not fail")
        except NativeError:
            pass
        assert ctypes.c_int.in_dll(shim, entry).value == 0
        got = t.force(x, energy=energy)
        # f32 sums in another order at most: 2e-6 of the norm (twice the pairs' forces or the charges: some 0.1 to 1)
        off = float((got - want).norm() / want.norm())
        assert off <= 2e-6, (entry, energy, off)
print("as a fresh context's")
"""


# the chain on the call's stream and beside the pairs
@pytest.mark.parametrize("waters", [600, 2200])
@pytest.mark.parametrize("deterministic", [False, True])
def test_a_failed_transform_leaves_no_charge(cuda, tmp_path, waters, deterministic):
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib))
    p = subprocess.run([sys.executable, "-c", CHILD, "1" if deterministic else "0", str(waters)], env=env, text=True,
                       capture_output=True, timeout=300, cwd=Path(__file__).resolve().parent.parent)
    assert p.returncode == 0 and "as a fresh context's" in p.stdout, p.stdout[-2000:] + p.stderr[-4000:]
