"""conan_deposit_static on its small tiles: the smallest lattice that holds
one and the lattices around the 2D switch, on an output that is not 16-byte
aligned, called back to back without waiting (each call clears what the one
before left) and from a CUDA graph. Against a double-precision CIC deposit of
the same displacements; positions are rounded to 2^-21 cell and weights to
2^-23 per particle, so a cell of m particles is within m (6 2^-21 + 8 2^-23)
plus the rounding of the float result."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _cic(d, dim, n, f):
    nf = n * f
    i = np.arange(n ** dim)
    rho, cnt = np.zeros(nf ** dim), np.zeros(nf ** dim)
    org, fr = [], []
    for k in range(dim):
        x = d[k].astype(np.float64)
        fl = np.floor(x)
        org.append((i // n ** k) % n * f + fl.astype(np.int64))
        fr.append(x - fl)
    for b in range(1 << dim):
        idx, w = 0, 1.0
        for k in range(dim - 1, -1, -1):
            idx = idx * nf + (org[k] + ((b >> k) & 1)) % nf
            w = w * (fr[k] if (b >> k) & 1 else 1 - fr[k])
        np.add.at(rho, idx, w)
        np.add.at(cnt, idx, 1.0)
    mass = float(f) ** dim
    return rho * mass - 1, (cnt * (6 * 2.0 ** -21 + 8 * 2.0 ** -23)) * mass


@pytest.mark.parametrize("dim,n,f", [(3, 16, 1), (3, 32, 1), (3, 64, 1), (3, 32, 2), (3, 128, 1), (2, 16, 1),
                                     (2, 256, 1), (2, 512, 1), (2, 256, 2), (1, 128, 1)])
def test_static_deposit_small_tiles(gpu, conan, dim, n, f):
    lib = conan._lib.lib()
    rng = np.random.default_rng(n)
    sets = []
    for amp in (0.3, 6.0):
        d = rng.uniform(-amp, amp, size=(dim, n ** dim)).astype(np.float32)
        d[:, : n ** dim // 16] = -(np.arange(n ** dim // 16) % 7)  # on cell faces
        buf = torch.full(((n * f) ** dim + 1,), 7.0, device="cuda")
        sets.append((d, torch.from_numpy(d).cuda(), buf))

    def call(dev, out, stream):
        p = [C.c_void_p(dev[k].data_ptr()) if k < dim else None for k in range(3)]
        conan._lib.check(lib.conan_deposit_static(dim, n, f, p[0], p[1], p[2], C.c_void_p(out.data_ptr()),
                                                  C.c_void_p(stream)))

    def good():
        for d, _, buf in sets:
            ref, bar = _cic(d, dim, n, f)
            got = buf[1:].cpu().numpy().astype(np.float64)
            assert np.all(np.abs(got - ref) <= bar + np.abs(ref) * 2.0 ** -23 + 2.0 ** -23)

    s = torch.cuda.current_stream().cuda_stream
    for _ in range(3):
        for _, dev, buf in sets:
            call(dev, buf[1:], s)
    torch.cuda.synchronize()
    good()
    for _, _, buf in sets:
        buf.fill_(7.0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _, dev, buf in sets:
            call(dev, buf[1:], torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    good()
