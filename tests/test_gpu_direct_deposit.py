"""The FP64 direct deposit (small lattices) against the counting sort, bit for
bit: densities of spread and of crowded particles (more than 2^12 in one cell,
where the sorted deposit's third word is used), whole runs, and the largest
lattice that takes it and the next one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,Nm,f", [(1, 64, 1), (1, 256, 4), (2, 16, 1), (2, 64, 1), (2, 256, 2), (2, 1024, 1),
                                      (3, 8, 1), (3, 16, 2), (3, 64, 1), (3, 32, 4)])
def test_direct_deposit_equals_sorted(gpu, conan, dim, Nm, f):
    L = 50.0
    rng = np.random.default_rng(Nm)
    q = np.stack(np.meshgrid(*[np.arange(Nm)] * dim, indexing="ij"), -1).reshape(-1, dim)[:, ::-1] * (L / Nm)
    for crowd in (False, True):
        X = q + rng.uniform(-3, 3, size=q.shape) * (L / (Nm * f))
        if crowd:
            X[: len(X) // 2] = L / 2 + rng.uniform(0, 1e-3, size=(len(X) // 2, dim)) * (L / (Nm * f))
        X = np.ascontiguousarray(X)
        out = []
        for mode in (None, "sorted"):
            g = conan.Gravity(dim, Nm, f, L, precision="fp64")
            if mode:
                g.deposit_mode = mode
            assert g.deposit_mode == "sorted"
            g.set_state(X, np.zeros_like(X), 0.3, 0.3)
            d = g.density()
            g.run(None, 0.3, 0.01, 3)
            g.drift(0.33, 0.01)  # a fused deposit that a new state makes stale
            g.set_state(X, np.zeros_like(X), 0.3, 0.3)
            out.append((d, g.density(), *g.state()))
            g.close()
        for a, b in zip(*out):
            assert np.array_equal(a, b)
        assert np.array_equal(out[0][0], out[0][1])


@pytest.mark.parametrize("dim,Nm", [(2, 64), (3, 32)])
def test_switching_the_deposit_mid_run(gpu, conan, dim, Nm):
    L = 50.0
    rng = np.random.default_rng(1)
    phi = rng.normal(size=Nm ** dim) * 1e-2
    ref = conan.Gravity(dim, Nm, 1, L, precision="fp64")
    ref.run(phi, 0.1, 0.02, 6)
    g = conan.Gravity(dim, Nm, 1, L, precision="fp64")
    g.run(phi, 0.1, 0.02, 3)
    g.drift(0.16, 0.02)
    g.deposit_mode = "sorted"  # with a fused deposit pending
    g.kick(0.17, 0.02)
    a = 0.16 + 0.02
    g.run(None, a, 0.02, 2)
    for x, y in zip(ref.state(), g.state()):
        assert np.allclose(x, y, rtol=0, atol=1e-12 * L)  # the scale factors accumulate differently
    ref.close()
    g.close()
