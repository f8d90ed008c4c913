"""Friends-of-friends rows at the lengths where the row sorts and the shared
candidate lists change their form: quarter warps (8), warps (32), one warp in
shared memory (512), one CTA (4096), the radix sort beyond, and counts that
leave the last warp nearly empty. Whole numbers against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("m", [1, 7, 8, 9, 32, 33, 512, 513, 4096, 4097])
def test_row_lengths(gpu, conan, oracle, dim, m):
    L, ll = 100.0, 0.9
    rng = np.random.default_rng(m)
    rows = [np.column_stack([rng.uniform(-3, L + 3, m)] + [rng.uniform(50.0, 50.9, m)] * (dim - 1))]
    # a second row beside it, short rows elsewhere, unwrapped coordinates
    rows.append(np.column_stack([rng.uniform(0, L, max(1, m // 2))] + [rng.uniform(51.0, 51.8, max(1, m // 2))] * (dim - 1)))
    rows.append(rng.uniform(-L / 2, 1.5 * L, size=(77, dim)))
    X = np.ascontiguousarray(rng.permutation(np.concatenate(rows)))
    X[: len(X) // 8] = X[len(X) // 2: len(X) // 2 + len(X) // 8]  # equal positions: ties in x
    ref = oracle.fof(dim, L, ll, X)
    ref = ref[0] if isinstance(ref, tuple) else ref
    for _ in range(3):
        tags, ng = conan.fof(X, dim, L, ll)
        assert np.array_equal(tags, ref)
        assert ng == ref.max()
