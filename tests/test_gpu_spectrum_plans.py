"""FP64 handles that solve around the line pass plan the full transforms at the
first power spectrum only, in the gradient mesh's memory."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

COUNT = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int plans = 0;
int cufftMakePlanMany(int h, int r, int *n, int *ie, int is, int id, int *oe, int os, int od, int t, int b, size_t *w) {
    int (*real)(int, int, int *, int *, int, int, int *, int, int, int, int, size_t *) =
        dlsym(dlopen("libcufft.so.11", RTLD_NOW | RTLD_NOLOAD), "cufftMakePlanMany");
    ++plans;
    return real(h, r, n, ie, is, id, oe, os, od, t, b, w);
}
"""

CHILD = r"""
import ctypes, sys
import conan_b200 as cb
plans = ctypes.c_int.in_dll(ctypes.CDLL(sys.argv[1]), "plans")
for dim, n, gradient, made, later in ((2, 64, "fd4", 2, 2), (3, 64, "fd4", 2, 2), (2, 32, "fd4", 2, 0),
                                      (2, 64, "spectral", 2, 0)):
    plans.value = 0
    g = cb.Gravity(dim, n, 1, 100.0, precision="fp64", gradient=gradient)
    assert plans.value == made, (dim, n, gradient, plans.value)
    for _ in range(2):
        g.power_spectrum()
    assert plans.value == made + later
    g.close()
"""


def test_handles_plan_one_pair(gpu, conan, tmp_path):
    src, lib = tmp_path / "count.c", tmp_path / "count.so"
    src.write_text(COUNT)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(lib)], cwd=ROOT, env={**os.environ, "LD_PRELOAD": str(lib)},
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("dim,Nm,f", [(2, 64, 1), (2, 512, 2), (3, 64, 1), (3, 32, 4)])
def test_spectra_between_steps(gpu, conan, dim, Nm, f):
    """The spectrum against numpy's, and a run with spectra in between against one without: the same bits."""
    L, nf, a, da = 100.0, Nm * f, 0.1, 0.02
    phi = np.random.default_rng(dim + Nm).normal(size=Nm ** dim) * 20
    g, h = (conan.Gravity(dim, Nm, f, L, precision="fp64") for _ in range(2))
    for s in (g, h):
        s.init(phi, a, a + da / 2)
    for i in range(3):
        if i < 2:
            k, P, cnt = g.power_spectrum()
        for s in (g, h):
            s.drift(a, da)
        if i:
            g.power_spectrum()
        for s in (g, h):
            s.kick(a + da / 2, da)
        a += da
    g.power_spectrum()
    for x, y in zip(g.state(), h.state()):
        assert np.array_equal(x, y)
    d = h.density().reshape((nf,) * dim)
    W = np.abs(np.fft.fftn(d)) ** 2
    i = np.indices(W.shape)
    i = np.where(i > nf // 2, i - nf, i)
    b = np.floor(np.sqrt((i ** 2).sum(0)) + 0.5).astype(int)
    k, P, cnt = h.power_spectrum(8)
    for j in range(1, 8):
        sel = W[b == j]
        assert cnt[j] == sel.size and abs(P[j] - sel.mean() * L ** dim / nf ** (2 * dim)) < 1e-10 * P[j]
    g.close()
    h.close()
