"""The sorted deposit's small tiles and the two-launch scan at the edges of
their ranges: the smallest meshes that hold a tile, meshes one size below
and above the switch to the large tiles (148 tiles), block counts of the scan
around 256, and batches of small boxes, against md_cic (FP64 rounding of sums
of 2^-52 weights)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,Nm,f", [(1, 128, 2), (1, 256, 1), (2, 16, 1), (2, 32, 1), (2, 256, 1), (2, 512, 1),
                                      (2, 512, 2), (3, 8, 1), (3, 16, 1), (3, 32, 2), (3, 64, 2)])
def test_sorted_deposit_small_tiles(gpu, conan, oracle, dim, Nm, f):
    L = 40.0
    rng = np.random.default_rng(Nm * f)
    q = np.stack(np.meshgrid(*[np.arange(Nm)] * dim, indexing="ij"), -1).reshape(-1, dim)[:, ::-1]
    X = q * (L / Nm) + rng.uniform(-3, 3, size=q.shape) * (L / (Nm * f))
    X[: len(X) // 4] = L / 3 + rng.uniform(0, L / (Nm * f), size=(len(X) // 4, dim))  # a crowded cell
    X = np.ascontiguousarray(X)
    g = conan.Gravity(dim, Nm, f, L, precision="fp64")
    g.set_state(X, np.zeros_like(X), 0.1, 0.1)
    ref = oracle.md_cic(dim, Nm * f, L, X, float(f) ** dim) - 1
    got = g.density()
    assert np.max(np.abs(got - ref)) < 1e-11 * max(1.0, np.max(np.abs(ref)))
    assert np.array_equal(got, g.density())  # the counts were cleared
    g.close()
