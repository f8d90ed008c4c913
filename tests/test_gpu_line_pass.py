"""The FP64 Poisson solve around the line pass (2D meshes of 64 to 1024 cells
per side, 3D of 64 to 512), every transform length, against the same solve by
full transforms in numpy: the density that the handle deposits, its potential
within FP64 rounding of two transforms (log2(cells) levels of 2^-53, a
hundredfold margin)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,Nm,f", [(2, 64, 1), (2, 128, 1), (2, 256, 1), (2, 512, 1), (2, 512, 2), (2, 64, 4),
                                      (3, 64, 1), (3, 64, 2), (3, 64, 4), (3, 64, 8), (2, 32, 1), (2, 2048, 1)])
def test_potential_matches_full_transforms(gpu, conan, dim, Nm, f):
    L, a, nf = 80.0, 0.4, Nm * f
    rng = np.random.default_rng(Nm + f)
    q = np.stack(np.meshgrid(*[np.arange(Nm)] * dim, indexing="ij"), -1).reshape(-1, dim)[:, ::-1] * (L / Nm)
    X = np.ascontiguousarray(q + rng.uniform(-3, 3, size=q.shape) * (L / nf))
    g = conan.Gravity(dim, Nm, f, L, precision="fp64")
    g.set_state(X, np.zeros_like(X), a, a)
    delta = g.density().reshape((nf,) * dim)
    g.kick(a, 0.01)
    phi = g.potential().reshape((nf,) * dim)
    g.close()
    k2 = 0.0
    for ax in range(dim):
        w = np.arange(nf // 2 + 1) if ax == dim - 1 else np.where(np.arange(nf) > nf // 2, np.arange(nf) - nf, np.arange(nf))
        k2 = k2 + (w.astype(float) ** 2).reshape([-1 if i == ax else 1 for i in range(dim)])
    k2.flat[0] = np.inf
    G = 1.5 * 68.5 ** 2
    axes = tuple(range(dim))
    spec = np.fft.rfftn(delta, axes=axes) * (-(G / a) * (L / (2 * np.pi)) ** 2 / k2)
    ref = np.fft.irfftn(spec, s=delta.shape, axes=axes)
    scale = np.sqrt(np.mean(ref ** 2))
    assert np.max(np.abs(phi - ref)) < 100 * np.log2(nf ** dim) * 2.0 ** -53 * np.max(np.abs(ref)) + 1e-13 * scale
