"""The error of the FP64 Poisson solve around the line pass against long double,
beside that of the same solve by library transforms (torch.fft): no larger. The
measure is the rms over all modes of |k| times the potential's error, the
error of the force, pooled over several fields: restated in numpy, the ratio is
0.97 to 1.00 with correctly rounded twiddles and 1.05 to 1.08 with those of the
rounded angles, so 1.03 tells them apart."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
sf = pytest.importorskip("scipy.fft")


@pytest.mark.parametrize("n,fields", [(128, 16), (256, 12), (512, 8)])
def test_error_is_the_librarys(gpu, conan, n, fields):
    LD, L, a = np.longdouble, 80.0, 0.4
    kx = np.arange(n // 2 + 1).astype(float)
    ky = np.where(np.arange(n) > n // 2, np.arange(n) - n, np.arange(n)).astype(float)
    k2 = ky[:, None] ** 2 + kx[None] ** 2
    k2i = k2.copy()
    k2i[0, 0] = np.inf
    gs = -(1.5 * 68.5 ** 2) / (a * n ** 2) * (L / (2 * np.pi)) ** 2
    weight = k2 * np.where((kx == 0) | (kx == n // 2), 1, 2)[None]
    q = np.stack(np.meshgrid(*[np.arange(n)] * 2, indexing="ij"), -1).reshape(-1, 2)[:, ::-1] * (L / n)
    green = torch.tensor(gs / k2i, device="cuda")
    here = lib = 0.0
    g = conan.Gravity(2, n, 1, L, precision="fp64")
    for i in range(fields):
        rng = np.random.default_rng(100 * n + i)
        X = q + rng.uniform(-3, 3, size=q.shape) * (L / n)
        g.set_state(X, np.zeros_like(X), a, a)
        d = g.density().reshape(n, n)
        g.kick(a, 0.01)
        phi = g.potential().reshape(n, n)
        t = torch.fft.irfft2(torch.fft.rfft2(torch.tensor(d, device="cuda")) * green, s=(n, n), norm="forward")
        ref = sf.irfft2(sf.rfft2(d.astype(LD)) * (LD(gs) / k2i.astype(LD)), s=(n, n), norm="forward")
        err = lambda x: np.sum(np.abs(sf.rfft2((x - ref).astype(np.float64))) ** 2 * weight)  # noqa: E731
        here += err(phi)
        lib += err(t.cpu().numpy())
    g.close()
    assert np.sqrt(here / lib) < 1.03
