"""The cache of idle FFT plans, on the host: the library's cuFFT calls go to a
stand-in that counts plans and fails where it is told to. A pair that could not
be planned is destroyed and never handed to a later call; one that finds no
memory is planned again once the idle pairs are given back."""
import os
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

FAKE = r"""
#include <stddef.h>
int handles = 0, planned[64], live = 0, fail_at = -1, fail_code = 5, calls = 0;
int cufftCreate(int *h) { *h = ++handles; ++live; return 0; }
int cufftDestroy(int h) { --live; planned[h] = 0; return 0; }
int cufftSetAutoAllocation(int h, int on) { return 0; }
int cufftMakePlanMany(int h, int rank, int *n, int *ie, int is, int id, int *oe, int os, int od, int type, int batch,
                      size_t *work) {
    if (calls++ == fail_at) return fail_code;
    planned[h] = 1;
    *work = 16;
    return 0;
}
"""

CHILD = r"""
import ctypes as C, sys
lib, fake = C.CDLL(sys.argv[1]), C.CDLL(sys.argv[2])
var = lambda n: C.c_int.in_dll(fake, n)
planned = (C.c_int * 64).in_dll(fake, "planned")

class Mesh(C.Structure):  # common.cuh
    _fields_ = [("R", C.c_int), ("n", C.c_int), ("shift", C.c_int), ("cells", C.c_size_t), ("nh", C.c_int),
                ("spec", C.c_size_t), ("cshift", C.c_int), ("mspec", C.c_size_t), ("batch", C.c_int),
                ("inv_nh", C.c_double)]

class Pair(C.Structure):  # fft.cuh
    _fields_ = [("r2c", C.c_int), ("c2r", C.c_int), ("work_bytes", C.c_size_t), ("dbl", C.c_bool)]

m = Mesh(3, 32, 5, 32 ** 3, 17, 17 * 1024, 15, 17 * 1024, 1, 1 / 17)
take = lambda p: lib._ZN5conan9plan_takeERKNS_4MeshEbPNS_7FFTPairE(C.byref(m), C.c_bool(True), C.byref(p))
give = lambda p: lib._ZN5conan11plan_returnERKNS_4MeshEbPNS_7FFTPairE(C.byref(m), C.c_bool(True), C.byref(p))
for at in (0, 1):  # the forward, then the inverse plan cannot be made
    var("calls").value, var("fail_at").value = 0, at
    p = Pair()
    assert take(p) != 0
    give(p)  # as the scope that took it does
    var("fail_at").value = -1
    assert var("live").value == 0
    q = Pair()
    assert take(q) == 0 and planned[q.r2c] and planned[q.c2r] and q.work_bytes == 16
    give(q)
    r = Pair()  # the same pair again
    assert take(r) == 0 and (r.r2c, r.c2r) == (var("handles").value - 1, var("handles").value)
    give(r)
    assert lib.conan_release_caches() == 0 and var("live").value == 0
# no memory (CUFFT_ALLOC_FAILED): the idle pair goes, and planning succeeds
p = Pair()
assert take(p) == 0
give(p)
m.n, m.shift, m.cshift = 64, 6, 18
var("calls").value, var("fail_at").value, var("fail_code").value = 0, 1, 2
q = Pair()
assert take(q) == 0 and planned[q.r2c] and planned[q.c2r] and not planned[p.r2c] and var("live").value == 2
give(q)
assert lib.conan_release_caches() == 0 and var("live").value == 0
"""


def test_a_pair_that_was_not_planned_is_not_kept(conan, tmp_path):
    src, fake = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(fake), str(src)], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(ROOT / "conan_b200/lib/libconan_pm.so"), str(fake)],
                       env={**os.environ, "LD_PRELOAD": str(fake)}, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
