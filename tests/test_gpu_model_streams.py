"""The differentiable model is ordered after the caller's stream: inputs that a
slow kernel is still producing when the call returns control to the host, on
the default stream and on one of the caller's own."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("own", [False, True])
def test_calls_wait_for_their_inputs(gpu, conan, own):
    from conan_b200.autograd import DiffPM
    m = DiffPM(dim=3, mbits=6, L_box=60.0, ns=-2.0, a0=0.05, da=0.05, n=3, checkpoint_every=2)
    gen = torch.Generator(device="cuda").manual_seed(5)
    noise = torch.randn(m.nnoise, device="cuda", generator=gen)
    gd = torch.randn(m.ncells, device="cuda", generator=gen) / m.ncells
    A = torch.randn(4096, 4096, device="cuda", generator=gen)
    ref, gref = torch.empty(m.ncells, device="cuda"), torch.empty(m.nnoise, device="cuda")
    torch.cuda.synchronize()
    m.forward_raw(noise, ref)
    m.backward_raw(gd, gref)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if own else torch.cuda.default_stream()
    with torch.cuda.stream(stream):
        for _ in range(3):
            n2, g2 = torch.zeros_like(noise), torch.zeros_like(gd)
            out, gn = torch.empty_like(ref), torch.empty_like(gref)
            slow = A
            for _ in range(8):  # a millisecond or more of work ahead of the input
                slow = slow @ A
            n2.copy_(noise + 0 * slow[0, 0].clamp(0, 0))
            m.forward_raw(n2, out)
            for _ in range(8):
                slow = slow @ A
            g2.copy_(gd + 0 * slow[0, 0].clamp(0, 0))
            m.backward_raw(g2, gn)
            stream.synchronize()
            assert torch.equal(out, ref) and torch.equal(gn, gref)
    m.close()
