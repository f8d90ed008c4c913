"""The adjoint's size-dependent kernels: the merging vector deposit (2^18
particles and more, 2D and 3D), the z-marching divergence (3D meshes of 32
cells per side and more) with the plane transforms' solve (FP32, 64 cells and
more), the last step alone (no vector deposit), and checkpoints at every step
and at none. In FP64 against the CPU adjoint (the bar of the suite's other
FP64 adjoint tests); in FP32, where positions pass CIC kinks and no bar per
component follows from the rounding, through two exact properties: reruns
give the same bits, and so does a density gradient times a power of two (the
fixed-point exponent follows the largest |pbar|).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASES = [  # dim, mbits, f, L, ns, a0, da, n, checkpoint
    (3, 6, 1, 60.0, -2.0, 0.05, 0.08, 4, 3),   # smallest merging lattice; z pass
    (2, 9, 1, 60.0, -1.5, 0.05, 0.08, 4, 2),   # the same in 2D
    (3, 5, 1, 40.0, -2.0, 0.05, 0.1, 4, 1),    # smallest z-marching mesh, 3D transforms
    (3, 5, 2, 40.0, -1.5, 0.05, 0.1, 3, 8),    # mesh finer than the lattice
    (3, 4, 2, 25.0, -2.0, 0.05, 0.1, 1, 1),    # one step: rhobar is zero
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_adjoint_kernels(gpu, conan, oracle, case, prec):
    from conan_b200.autograd import DiffPM
    dim, mbits, f, L, ns, a0, da, n, every = case
    rng = np.random.default_rng(23)
    w = rng.normal(size=(1 << mbits) ** dim)
    dt = torch.float64 if prec == "fp64" else torch.float32
    m = DiffPM(dim=dim, mbits=mbits, L_box=L, ns=ns, a0=a0, da=da, n=n, checkpoint_every=every, f=f, precision=prec)
    out = torch.empty(m.ncells, dtype=dt, device="cuda")
    wt = torch.tensor(w, dtype=dt, device="cuda")
    dbar = rng.normal(size=m.ncells) / m.ncells
    gd = torch.tensor(dbar, dtype=dt, device="cuda")
    g = torch.empty_like(wt)
    m.forward_raw(wt, out)
    m.backward_raw(gd, g)
    if prec == "fp64":
        dref, gref = oracle.diff_adjoint(dim, mbits, f, L, ns, False, 8.0, 0.83, a0, da, n, w, dbar)
        assert np.max(np.abs(out.cpu().numpy() - dref)) < 1e-10 * max(1.0, np.max(np.abs(dref)))
        assert np.max(np.abs(g.cpu().numpy() - gref)) < 1e-8 * np.max(np.abs(gref))
    for scale in (1.0, 16.0, 2.0 ** -20):
        h = torch.empty_like(g)
        m.forward_raw(wt, out)
        m.backward_raw(gd * scale, h)
        assert torch.equal(h, g * scale)
    m.close()
