"""The z-marching gradient mesh at its smallest mesh, on both sides of its
default's threshold and in both precisions, bit for bit against one thread per
cell (the same operations on the same values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nm,f,prec", [(32, 1, "fp32"), (16, 2, "fp64"), (64, 1, "fp64"), (128, 1, "fp64"),
                                       (64, 4, "fp32")])
def test_marching_gradient_mesh(gpu, conan, monkeypatch, Nm, f, prec):
    L = 100.0
    rng = np.random.default_rng(Nm)
    q = np.stack(np.meshgrid(*[np.arange(Nm)] * 3, indexing="ij"), -1).reshape(-1, 3)[:, ::-1] * (L / Nm)
    X = np.ascontiguousarray(q + rng.uniform(-2, 2, size=q.shape) * (L / (Nm * f)))
    out = []
    for kern in ("cell", "zm", None):
        if kern:
            monkeypatch.setenv("CONAN_GRAD_KERNEL", kern)
        else:
            monkeypatch.delenv("CONAN_GRAD_KERNEL")
        g = conan.Gravity(3, Nm, f, L, precision=prec)
        g.set_state(X, np.zeros_like(X), 0.4, 0.4)
        g.kick(0.4, 0.01)
        out.append(g.state()[1])
        g.close()
    assert np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
