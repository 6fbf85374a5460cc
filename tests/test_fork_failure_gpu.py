"""A (+-1') class that fails while its pencil's reduction is still under way on the
helper thread: nvpt_qdnevpt returns the error, and the next call on the same context is
right.  The failure is made on the host: a preloaded cublasDgemm refuses the product that
follows the start of the reduction, for the classes with as many labels as virtual
orbitals.  Runs in a child process (the preloaded library belongs to one).  The good
calls are held to the energies' tolerance, 1e-9."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

SHIM = r"""
#include <dlfcn.h>
typedef int (*gemm_t)(void *, int, int, int, int, int, const double *, const double *, int, const double *, int,
                      const double *, double *, int);
static int order, labels, refused;
void shim_refuse(int n3, int l) { order = n3; labels = l; refused = 0; }
int shim_refused(void) { return refused; }
int cublasDgemm_v2(void *h, int ta, int tb, int m, int n, int k, const double *al, const double *a, int lda,
                   const double *b, int ldb, const double *be, double *c, int ldc) {
    static gemm_t real;
    if (!real) real = (gemm_t)dlsym(dlopen("libcublas.so.13", RTLD_LAZY), "cublasDgemm_v2");
    if (order && m == order && k == order && n == labels) {
        __sync_fetch_and_add(&refused, 1);
        return 3; /* CUBLAS_STATUS_ALLOC_FAILED */
    }
    return real(h, ta, tb, m, n, k, al, a, lda, b, ldb, be, c, ldc);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, {root!r})
from nevpt2_gb300 import koopro, qdnevpt as gq, synth
from nevpt2_gb300._native import NvptError
shim = ctypes.CDLL({shim!r})
n, metat, nvirt = {n}, {metat}, 11
p = synth.make_problem(n, n, 3, nvirt, metat=metat, seed=31, with_trdm=metat > 1)
koop = koopro.koopro4QD(p)
run = lambda: gq.qdnevpt(p, koop, transition=p.trdm if metat > 1 else None)
ref = run()
for _ in range(4):
    shim.shim_refuse(n**3, nvirt)
    try:
        run()
        raise SystemExit("the refused product was not reported")
    except NvptError as e:
        assert e.status == 2, e
    assert shim.shim_refused() >= metat
    shim.shim_refuse(0, 0)
    got = run()
    for k in ("e2mpp", "e2enp", "e2mp", "e2en"):
        np.testing.assert_allclose(getattr(got, k), getattr(ref, k), rtol=1e-9, atol=1e-9)
print("recovered")
"""


@pytest.mark.parametrize("n,metat", [(5, 1), (5, 2), (6, 3)])
def test_class_that_fails_before_its_join(tmp_path, n, metat):
    src, shim = tmp_path / "shim.c", tmp_path / "libshim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(shim), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=str(ROOT), shim=str(shim), n=n, metat=metat)],
                       env=dict(os.environ, LD_PRELOAD=str(shim)), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "recovered" in r.stdout, r.stdout[-500:] + r.stderr[-2000:]
