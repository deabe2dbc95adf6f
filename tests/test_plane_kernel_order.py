"""The plane kernel (k_yz: y backward, z and y forward passes of an x plane in
one block) under every order of its threads that its barriers allow: compiled
for the host, where the block's threads take turns in ascending or in
descending order (host_emulation/emulate.h), it gives the same bits in both and
the values of the same passes in numpy's FP64.  At n = 8 and 16 a thread holds
a whole column and the lanes past the last column repeat it, so a missing
barrier between the reads and the in-place stores shows as a column transformed
twice."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HERE = os.path.join(ROOT, "tests", "host_emulation")
CSRC = os.path.join(ROOT, "dns_b200", "csrc")
SU, SV, SDWDY, SOMZ, SDWDX, SW, NWORK = 0, 1, 2, 3, 4, 5, 6  # kernels.cuh's work slots


@pytest.fixture(scope="module")
def plane(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("plane")
    src = open(os.path.join(CSRC, "kernels.cuh")).read()
    # the two instructions of the asynchronous copies
    src, a = re.subn(r"(void copy16\(void \*dst, const void \*src\) \{)[^}]*\}", r"\1 emu_copy16(dst, src); }", src)
    src, b = re.subn(r'asm volatile\("cp\.async\.wait_all;" ::: "memory"\);', "emu_copies_wait();", src)
    assert a == 1 and b >= 1
    (tmp / "kernels.cuh").write_text(src)
    (tmp / "fft_core.cuh").write_text(open(os.path.join(CSRC, "fft_core.cuh")).read())
    so = str(tmp / "plane.so")
    # no contraction: as on the device, only what is written as fma is one
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-ffp-contract=off", "-shared", "-fPIC",
                        f"-I{HERE}", f"-I{tmp}", os.path.join(HERE, "plane.cc"), "-o", so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    lib = ctypes.CDLL(so)
    lib.plane_run.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p] * 3 + [ctypes.c_int] * 4
    return lib


def expected(work, stale, n, kind, p):
    """N_x, N_y, N_z of plane p, and its real velocity."""
    nf = n // 2 + 1
    ky = (np.fft.fftfreq(n) * n)[:, None]
    kz = np.arange(nf)
    f = [work[s, p, :, :nf].astype(np.complex128) for s in range(NWORK)]
    back = lambda X: np.fft.ifft(X, axis=0) * n  # noqa: E731
    u, v, w, dwdx = (back(f[s]) for s in (SU, SV, SW, SDWDX))
    oz = back(f[SOMZ] - 1j * ky * f[SU])
    ox = back(1j * ky * f[SW]) - 1j * kz * v
    oy = 1j * kz * u - dwdx
    real = lambda X: np.fft.irfft(X, n, axis=1) * n / n ** 3  # noqa: E731
    vel = stale[:, p].astype(np.float64) if kind == 0 else np.array([real(a) for a in (u, v, w)])
    om = np.array([real(a) for a in (ox, oy, oz)])
    N = np.cross(vel, om, axis=0)
    return np.fft.fft(np.fft.rfft(N, axis=2), axis=1), vel


@pytest.mark.parametrize("n,fp64", [(8, 1), (8, 0), (16, 1), (16, 0), (32, 1), (32, 0), (64, 1), (64, 0)])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_order_of_threads_does_not_matter(plane, n, fp64, kind):
    R, C = (np.float64, np.complex128) if fp64 else (np.float32, np.complex64)
    W = 8 if fp64 else 16
    nf, nfp = n // 2 + 1, (n // 2 + 1 + W - 1) // W * W
    kcut = max(k for k in range(n) if k < 2.0 / 3.0 * (n // 2 + 1))
    rng = np.random.default_rng(n + kind)
    shape = (NWORK, n, n, nfp)
    work = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(C)
    stale = rng.standard_normal((3, n, n, n)).astype(R)
    tw = np.exp(-2j * np.pi * np.arange(n) / n).astype(C)
    p = n - 1
    out = []
    for descending in (0, 1):
        a, s = work.copy(), stale.copy()
        assert plane.plane_run(fp64, n, kind, a.ctypes.data, s.ctypes.data, tw.ctypes.data, nfp, kcut, p,
                               descending) == 1
        out.append((a, s))
    assert np.array_equal(out[0][0].view(R), out[1][0].view(R))
    assert np.array_equal(out[0][1], out[1][1])
    # a value passes some 3 log2(n) <= 18 butterflies and 20 pointwise
    # operations, each of one rounding: 64 of them bound the relative error
    tol = 64 * (2.0 ** -53 if fp64 else 2.0 ** -24)
    want, vel = expected(work, stale, n, kind, p)
    rows = [k % n for k in range(-kcut, kcut + 1)]
    got = np.array([out[0][0][s, p, :, :nf] for s in (0, 1, 2)])[:, rows, :kcut + 1]
    want = want[:, rows, :kcut + 1]
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
    if kind == 2:
        assert np.linalg.norm(out[0][1][:, p] - vel) <= tol * np.linalg.norm(vel)
    assert np.array_equal(out[0][0][:, :p].view(R), work[:, :p].view(R))  # the other planes are left alone
