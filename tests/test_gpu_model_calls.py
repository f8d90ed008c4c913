"""Calls of the differentiable model: buffers, repeated passes, stream capture."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# 64: the density is copied out of the mesh; 256 with the cluster plane pass: it
# is written into the caller's array by a kernel, as on 512^3 meshes by default
@pytest.mark.parametrize("mbits,plane", [(6, "0"), (8, "2")])
def test_density_arrays_need_no_more_than_a_floats_alignment(gpu, conan, monkeypatch, mbits, plane):
    from conan_b200.autograd import DiffPM
    monkeypatch.setenv("CONAN_PLANE_PASS", plane)
    m = DiffPM(dim=3, mbits=mbits, L_box=100.0, ns=-2.0, a0=0.05, da=0.05, n=1)
    gen = torch.Generator(device="cuda").manual_seed(3)
    noise = torch.randn(m.nnoise, device="cuda", generator=gen)
    ref = torch.empty(m.ncells, device="cuda")
    m.forward_raw(noise, ref)
    for skip in (1, 2, 3, 4):
        buf = torch.full((m.ncells + 8,), 7.0, device="cuda")
        m.forward_raw(noise, buf[skip:skip + m.ncells])
        torch.cuda.synchronize()
        assert torch.equal(buf[skip:skip + m.ncells], ref)
        assert (buf[:skip] == 7).all() and (buf[skip + m.ncells:] == 7).all()
    m.close()


# the last checkpoint at the initial state, one step and several before the end
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("mbits,n,every", [(4, 3, 8), (5, 5, 2), (6, 4, 2), (6, 1, 1)])
def test_a_further_gradient_of_one_forward(gpu, conan, prec, mbits, n, every):
    from conan_b200.autograd import DiffPM
    dt = torch.float32 if prec == "fp32" else torch.float64
    m = DiffPM(dim=3, mbits=mbits, L_box=60.0, ns=-2.0, a0=0.05, da=0.08, n=n, checkpoint_every=every, precision=prec)
    gen = torch.Generator(device="cuda").manual_seed(7)
    noise = torch.randn(m.nnoise, device="cuda", dtype=dt, generator=gen)
    losses = [torch.randn(m.ncells, device="cuda", dtype=dt, generator=gen) / m.ncells for _ in range(3)]
    out, g = torch.empty_like(losses[0]), torch.empty_like(noise)
    want = []
    for gd in losses:  # one forward each
        m.forward_raw(noise, out)
        m.backward_raw(gd, g)
        want.append(g.clone())
    m.forward_raw(noise, out)
    for gd, w in list(zip(losses, want)) + [(losses[0], want[0])]:  # one forward for all
        m.backward_raw(gd, g)
        assert torch.equal(g, w)
    # through torch.autograd: two losses of one density
    x = noise.clone().requires_grad_(True)
    delta = m(x)
    for gd, w in zip(losses[:2], want):
        assert torch.equal(torch.autograd.grad(delta, x, gd, retain_graph=True)[0], w)
    m.close()


@pytest.mark.parametrize("prec,mbits,n,every", [("fp32", 6, 5, 2), ("fp64", 5, 3, 8)])
def test_captured_calls(gpu, conan, prec, mbits, n, every):
    from conan_b200.autograd import DiffPM
    dt = torch.float32 if prec == "fp32" else torch.float64
    m = DiffPM(dim=3, mbits=mbits, L_box=60.0, ns=-2.0, a0=0.05, da=0.08, n=n, checkpoint_every=every, precision=prec)
    gen = torch.Generator(device="cuda").manual_seed(9)
    fields = [torch.randn(m.nnoise, device="cuda", dtype=dt, generator=gen) for _ in range(3)]
    gd = torch.randn(m.ncells, device="cuda", dtype=dt, generator=gen) / m.ncells
    noise, out, g = fields[0].clone(), torch.empty_like(gd), torch.empty_like(fields[0])
    want = []
    for f in fields:  # uncaptured, one forward each
        noise.copy_(f)
        m.forward_raw(noise, out)
        m.backward_raw(gd, g)
        want.append((out.clone(), g.clone()))

    def check(i, density=True):
        torch.cuda.synchronize()
        assert torch.equal(g, want[i][1]) and (not density or torch.equal(out, want[i][0]))
        g.zero_()
        out.zero_()

    graphs = []
    for calls in ("fb", "f", "b"):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            if "f" in calls:
                m.forward_raw(noise, out)
            if "b" in calls:
                m.backward_raw(gd, g)
    both, fwd, bwd = graphs
    g.zero_()
    for i in (1, 2):  # one graph
        noise.copy_(fields[i])
        both.replay()
        check(i)
    noise.copy_(fields[0])  # a graph each, and a further gradient
    fwd.replay()
    bwd.replay()
    check(0)
    bwd.replay()
    check(0, density=False)
    noise.copy_(fields[1])  # a captured forward, uncaptured gradients
    fwd.replay()
    for density in (True, False):
        m.backward_raw(gd, g)
        check(1, density)
    noise.copy_(fields[2])  # the other way, then a further gradient
    m.forward_raw(noise, out)
    bwd.replay()
    check(2)
    m.backward_raw(gd, g)
    check(2, density=False)
    noise.copy_(fields[0])  # and uncaptured again
    m.forward_raw(noise, out)
    m.backward_raw(gd, g)
    check(0)
    torch.cuda.synchronize()
    del graphs, both, fwd, bwd
    m.close()


def test_checkpoint_memory(gpu, conan):
    """A slot per kept state and no more: 16 steps with a checkpoint every 8 keep two, as 15 steps do."""
    from conan_b200.autograd import DiffPM
    used = []
    for n, every in ((8, 8), (15, 8), (16, 8), (16, 16), (8, 16), (16, 4)):  # the first loads the kernels
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        m = DiffPM(dim=3, mbits=7, L_box=60.0, ns=-2.0, a0=0.05, da=0.01, n=n, checkpoint_every=every)
        used.append(before - torch.cuda.mem_get_info()[0])
        m.close()
    slot = 6 * 4 * 128 ** 3
    used = used[1:]
    assert abs(used[1] - used[0]) < slot / 4 and abs(used[2] - used[3]) < slot / 4
    assert abs(used[4] - used[1] - 2 * slot) < slot / 4 and abs(used[1] - used[2] - slot) < slot / 4
