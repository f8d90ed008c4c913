"""Copies of pageable host arrays through the shared staging lanes against
page-locked ones (which go to the driver as they are): sizes below, at and
beyond the four chunks where the lanes start, a last chunk that is not full,
several host threads at once, and after the caches were given back. The same
bytes either way."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


# states of n^dim x dim doubles: 0.4, 8 (four chunks), 50.3, 5.6 and 33.6 MB
@pytest.mark.parametrize("dim,Nm", [(3, 32), (1, 1 << 20), (3, 128), (2, 512), (2, 2048 // 2)])
def test_pageable_and_page_locked_copies_agree(gpu, conan, dim, Nm):
    rng = np.random.default_rng(3)
    phi = rng.normal(size=Nm ** dim)
    out = []
    for pin in (False, True):
        g = conan.Gravity(dim, Nm, 1, 100.0, precision="fp64")
        g.init(_pinned(phi) if pin else phi, 0.1, 0.1)
        # an array that starts 8 bytes into its pages
        X, P = (np.empty(Nm ** dim * dim + 1)[1:].reshape(-1, dim) for _ in range(2))
        if pin:
            X, P = _pinned(X), _pinned(P)
        g.state_into(X, P)
        h = conan.Gravity(dim, Nm, 1, 100.0, precision="fp64")
        h.set_state(X, P, 0.1, 0.1)
        d = h.density()
        out.append((X.copy(), P.copy(), d))
        g.close()
        h.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.isfinite(out[0][0]).all() and np.abs(out[0][1]).max() > 0


def test_threads_share_the_lanes(gpu, conan):
    H = {"dim": 3, "mbits": 7, "size": 100.0}
    rng = np.random.default_rng(4)
    fields = [rng.normal(size=128 ** 3) for _ in range(4)]
    ref = [conan.compute_potential(H, f) for f in fields]
    L = conan._lib.lib()
    assert L.conan_release_caches() == 0
    got, errs = [[None] * 3 for _ in fields], []

    def work(i):
        try:
            for j in range(3):
                got[i][j] = conan.compute_potential(H, fields[i])
        except Exception as e:  # noqa: BLE001
            errs.append(e)

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(fields))]
    for t in th:
        t.start()
    assert L.conan_release_caches() == 0  # while calls are under way
    for t in th:
        t.join()
    assert not errs
    for r, g in zip(ref, got):
        for x in g:
            assert np.array_equal(r, x)
