"""A batch whose streams could not all be created (the failure made on the host,
by a stand-in for the call that reports an error once): the run fails with an
error, the next one sets up what is missing and gives the usual result."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

STAND_IN = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int calls;
int cudaStreamCreateWithFlags(void **s, unsigned flags) {
    static int (*real)(void **, unsigned);
    if (!real) real = (int (*)(void **, unsigned))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD),
                                                        "cudaStreamCreateWithFlags");
    return ++calls == FAIL_AT ? 2 : real(s, flags);  /* cudaErrorMemoryAllocation */
}
"""

RUN = """
import numpy as np
from cumc3d_b200 import models
from cumc3d_b200.engine import BatchSolver, CumcError
def solver():
    probs = [models.riemann_1d(n, p["left"], p["right"], p["bx"], t_end=0.02)
             for n, p in zip((40, 300, 900), models.batch_problems(3, seed=4))]
    b = BatchSolver([p[0] for p in probs])
    for i, (_, prim, eps) in enumerate(probs):
        b.set_state(i, prim, eps)
    return b
b = solver()                      # creates one stream
try:
    b.run(5, check=False)
    raise SystemExit("the failing call went unnoticed")
except CumcError:
    pass
b.run(5, check=False)
c = solver()
c.run(5, check=False)
for i in range(3):
    for x, y in zip(b.get_state(i), c.get_state(i)):
        assert np.array_equal(x, y)
print("same")
"""


@pytest.mark.parametrize("fail_at", [2, 4, 7])
def test_run_after_a_failed_setup(tmp_path, fail_at):
    src, so = str(tmp_path / "s.c"), str(tmp_path / "s.so")
    with open(src, "w") as f:
        f.write(STAND_IN)
    subprocess.run(["gcc", "-shared", "-fPIC", "-DFAIL_AT=%d" % fail_at, src, "-o", so, "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", RUN], cwd=ROOT, env=dict(os.environ, LD_PRELOAD=so), capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
