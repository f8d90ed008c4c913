"""The initial conditions' filters around the size where they come from tables
(3D, 32 cells per side), with row lengths (n/2 + 1 modes) that four modes per
thread do not divide, against the CPU oracle in FP64 (rounding of the FFTs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,mbits", [(1, 5), (2, 1), (2, 6), (3, 1), (3, 4), (3, 5), (3, 6)])
@pytest.mark.parametrize("scale_free,smooth", [(True, False), (True, True), (False, False)])
def test_filters_match_the_oracle(gpu, conan, oracle, dim, mbits, scale_free, smooth):
    L, ns = 70.0, -1.7
    noise = oracle.noise_mt19937(5, 1 << (mbits * dim))
    H = {"dim": dim, "mbits": mbits, "size": L, "ns": ns, "smooth": smooth, "scale-free": scale_free, "scale": 3.0,
         "sigma": 0.83, "Omega0": 0.32, "H0": 69.0}
    if scale_free:
        ref = oracle.grf_scale_free(dim, mbits, L, ns, smooth, 3.0, 0.83, noise)
    else:
        ref = oracle.grf_cdm(dim, mbits, L, 0.32, 69.0, ns, noise)
    got = conan.generate_random_field(H, noise=noise)
    assert np.max(np.abs(got - ref)) < 1e-11 * np.max(np.abs(ref))
    pref = oracle.potential(dim, mbits, L, ref)
    assert np.max(np.abs(conan.compute_potential(H, ref) - pref)) < 1e-11 * np.max(np.abs(pref))
