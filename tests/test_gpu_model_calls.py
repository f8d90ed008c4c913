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
