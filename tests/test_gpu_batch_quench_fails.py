"""A quench that ends half-way (its graph cannot be made: cudaGraphInstantiate
is faked to fail once) leaves the batch as it has to be: the next evaluations
and the next quench are those of a batch that never saw the failure."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

FAKE = r"""
#include <dlfcn.h>
extern "C" int cudaGraphInstantiate(void **exec, void *graph, unsigned long long flags) {
    static int calls = 0;
    typedef int (*fn)(void **, void *, unsigned long long);
    static fn real = (fn)dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaGraphInstantiate");
    return calls++ == 0 ? 2 : real(exec, graph, flags);   // cudaErrorMemoryAllocation
}
"""

CHILD = """
import numpy as np
from moldy_b200 import MoldyBatch, workloads as wl
from moldy_b200._lib import MoldyError
ws = [wl.make_workload(n, sigma=0.1, temperature=0.0, ivol=1, seed=n) for n in (4, 6, 5, 7)]
new = np.concatenate([wl.make_workload(n, sigma=0.1, temperature=0.0, ivol=1, seed=90 + n).x0 for n in (4, 6, 5, 7)])
new = (new + 0.17) % 1.0 - 0.5                # every list is due again
res = []
for fail in (True, False):
    b = MoldyBatch.from_workloads(ws)
    if fail:
        try:
            b.quench(maxfn=20)
            raise SystemExit("the quench did not fail")
        except MoldyError as e:
            print(e)
    b.set_state(x0=new)
    out, f = b.force(), b.forces()
    q = b.quench(maxfn=20)
    res.append((out, f, q, b.get_state()))
    b.close()
for a, c in zip(*res):
    for p, q in (zip(a.values(), c.values()) if isinstance(a, dict) else [(a, c)]):
        assert np.array_equal(p, q)
print("as if nothing had failed")
"""


def test_batch_after_a_quench_that_failed(gpu_lib, tmp_path):
    src, so = tmp_path / "fake.cpp", tmp_path / "fake.so"
    src.write_text(FAKE)
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([gxx, "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=dict(os.environ, LD_PRELOAD=str(so)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "as if nothing had failed" in r.stdout, r.stdout + r.stderr
