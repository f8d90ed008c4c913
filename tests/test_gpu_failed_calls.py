"""What a call that failed on the host leaves behind: the next calls are right.
The failures are made on the host (an error code in place of the call's own)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# A run of 14 steps is four graphs of 4, 4, 4 and 2; the third is an update of
# the second, so the graphs made anew are 0 (first), 1 (a middle one), 2 (last).
# Lagrangian accumulator (FP32), two-word accumulator (FP64), sorted (FP64).
@pytest.mark.parametrize("fail", [0, 1, 2])
@pytest.mark.parametrize("prec,mode", [("fp32", None), ("fp64", None), ("fp64", "sorted")])
def test_run_that_fails_between_its_graphs(gpu, conan, prec, mode, fail):
    from conan_b200 import _lib as L
    Nm, a0, da, n = 32, 0.05, 0.02, 14
    phi = np.random.default_rng(1).normal(size=Nm ** 3) * 50

    def handle():
        g = conan.Gravity(3, Nm, 1, 100.0, precision=prec)
        if mode:
            g.deposit_mode = mode
        return g

    fresh = handle()
    g = handle()
    try:
        L.lib().conan_selftest_fail_graph(fail)
        with pytest.raises(conan.ConanError):
            g.run(phi, a0, da, n)
    finally:
        L.lib().conan_selftest_fail_graph(-1)
    # the state is that of the graphs before (up to the rounding of a kick and a
    # drift in one kernel or two), and its density holds its mass once
    a = a0
    done = (0, 4, 12)[fail]
    for _ in range(done):
        a += da
    X, P = g.state()
    assert abs(g.density().mean()) < 1e-5
    if done:
        assert g.scale_factors() == pytest.approx((a, a - da / 2), abs=1e-12)
        fresh.run(phi, a0, da, done)
        fresh.drift(a, da)
    else:
        assert g.scale_factors() == (a0, a0 + da / 2)
        fresh.init(phi, a0, a0 + da / 2)
    Xf, Pf = fresh.state()
    tol = 1e-5 if prec == "fp32" else 1e-11
    assert np.max(np.abs(X - Xf)) < tol * 100 and np.max(np.abs(P - Pf)) < tol * np.max(np.abs(Pf))
    # set anew, it runs as a fresh handle does
    g.init(phi, a0, a0 + da / 2)
    fresh.init(phi, a0, a0 + da / 2)
    assert np.array_equal(g.density(), fresh.density())
    g.run(phi, a0, da, n)
    fresh.run(phi, a0, da, n)
    for a, b in zip(g.state(), fresh.state()):
        assert np.array_equal(a, b)
    g.close()
    fresh.close()


# the model's second pass makes its graphs: the steps, the last step, the adjoint
@pytest.mark.parametrize("fail", [0, 1, 2])
@pytest.mark.parametrize("prec,mbits,plane", [("fp32", 5, "0"), ("fp64", 5, "0"), ("fp32", 8, "2")])
def test_model_pass_that_fails(gpu, conan, monkeypatch, prec, mbits, plane, fail):
    from conan_b200 import _lib as L
    from conan_b200.autograd import DiffPM
    monkeypatch.setenv("CONAN_PLANE_PASS", plane)
    dt = torch.float32 if prec == "fp32" else torch.float64
    m = DiffPM(dim=3, mbits=mbits, L_box=100.0, ns=-2.0, a0=0.05, da=0.05, n=3, checkpoint_every=2, precision=prec)
    gen = torch.Generator(device="cuda").manual_seed(11)
    noise = torch.randn(m.nnoise, device="cuda", dtype=dt, generator=gen)
    gd = torch.randn(m.ncells, device="cuda", dtype=dt, generator=gen) / m.ncells
    ref, gref = torch.empty_like(gd), torch.empty_like(noise)
    m.forward_raw(noise, ref)
    m.backward_raw(gd, gref)
    out, g = torch.empty_like(ref), torch.empty_like(gref)
    try:
        L.lib().conan_selftest_fail_graph(fail)
        with pytest.raises(conan.ConanError):
            m.forward_raw(noise, out)
            m.backward_raw(gd, g)
    finally:
        L.lib().conan_selftest_fail_graph(-1)
    if fail < 2:  # no forward to go with
        with pytest.raises(conan.ConanError):
            m.backward_raw(gd, g)
    else:
        m.backward_raw(gd, g)
        assert torch.equal(g, gref)
    for _ in range(2):
        m.forward_raw(noise, out)
        m.backward_raw(gd, g)
        assert torch.equal(out, ref) and torch.equal(g, gref)
    m.close()


def test_ensemble_run_after_a_failed_pass(gpu, conan, monkeypatch):
    """The run is one graph that is replayed: the deposit that the failed pass left
    for its plane transform is gone before."""
    from conan_b200 import _lib as L
    from conan_b200.ensemble import Ensemble
    monkeypatch.setenv("CONAN_PLANE_PASS", "2")
    e = Ensemble([(8, 100.0, -2.0, 1)], a0=0.05, a_end=0.15, steps=2, autotune=False)
    e.init()
    e.run()
    want = [x.copy() for x in e.state(0)]
    try:
        L.lib().conan_selftest_fail_graph(1)  # the model's second pass: its last step's graph
        with pytest.raises(conan.ConanError):
            e.forward_adjoint()
    finally:
        L.lib().conan_selftest_fail_graph(-1)
    e.run()
    for a, b in zip(e.state(0), want):
        assert np.array_equal(a, b)
    e.close()


def test_handles_get_the_memory_that_calls_without_one_keep(gpu, conan):
    """A friends-of-friends handle of 0.6 GB and the autotuner's copy of a state
    beside an array that leaves less free than they need: what a field call of
    256^3 kept idle (up to 0.5 GB) is given back for them."""
    conan.release_caches()
    g = conan.Gravity(3, 128, 1, 100.0, precision="fp32")
    g.init(np.zeros(128 ** 3), 0.05, 0.06)
    torch.cuda.empty_cache()
    H = {"dim": 3, "mbits": 8, "size": 100.0}
    conan.compute_potential(H, np.zeros(256 ** 3))
    MB = 1 << 20
    kept = torch.cuda.mem_get_info()[0]
    conan.release_caches()
    kept = torch.cuda.mem_get_info()[0] - kept
    assert 300 * MB < kept < 600 * MB  # it can be given back
    conan.compute_potential(H, np.zeros(256 ** 3))
    n = 6_000_000  # 24 + 24 + 24 + 4 + 4 + 4 + 8 bytes and more per particle
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 320 * MB, dtype=torch.uint8, device="cuda")
    fof = conan.FoF(3, n, 100.0, 0.1)
    fof.close()
    conan.release_caches()
    conan.compute_potential(H, np.zeros(256 ** 3))
    del fill
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 20 * MB, dtype=torch.uint8, device="cuda")
    g.autotune(0.05, 0.01)  # copies 50 MB
    del fill
    torch.cuda.empty_cache()
    conan.release_caches()
    g.close()
