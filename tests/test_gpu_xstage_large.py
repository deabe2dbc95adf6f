"""The x pass at the tiles that only the large grids have (n = 256: FP64 rows
of 64 bytes; n = 512: one block of some 200 KB, in FP32 of 1024 threads), on
white noise, which fills the modes outside the 2/3 rule too: n = 256 against
the CPU oracle, n = 512 against the step written with torch's FP64 FFTs, and at
n = 512 the bits of one call against those of two."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# as in test_gpu_xstage.py: single steps, FP64 rounding of a few transforms,
# FP32 rounding of some 30 operations a value
TOL = {0: 1e-13, 1: 1e-5}
DT = 2e-3


def white_field(n, seed):
    rng = np.random.default_rng(seed)
    return [0.1 * rng.standard_normal((n, n, n)) for _ in range(3)]


def nu_for(n):
    """nu dt |k|^2 up to 1 at the corner: the modes outside the rule decay
    visibly and stay stable."""
    return 1.0 / (DT * 3 * (n / 2) ** 2)


def outside_rule(n):
    k = np.abs(np.fft.fftfreq(n, 1.0 / n))
    kz = np.arange(n // 2 + 1)
    kmax = 2.0 / 3.0 * (n // 2 + 1)
    return (k[:, None, None] >= kmax) | (k[None, :, None] >= kmax) | (kz[None, None, :] >= kmax)


@pytest.fixture(scope="module")
def oracle_256(oracle_lib):
    n = 256
    U = white_field(n, n)
    o = oracle_lib.Oracle(n)
    o.set_velocity(*U)
    o.step(nu_for(n), DT, 2)
    return U, o.get_spectral(), o.dump_fields()[3]


@pytest.mark.parametrize("prec", [0, 1])
def test_white_noise_steps_match_oracle_256(dns_lib, oracle_256, prec):
    import dns_b200 as dns

    n = 256
    U, want, Po = oracle_256
    with dns.Context(n, prec, dns.DNS_FLAG_PRESSURE) as c:
        c.set_velocity(*U)
        c.step(nu_for(n), DT, 2)
        got = c.get_spectral()
        P = c.get_fields(pressure=True)[3]
    assert np.linalg.norm(got - want) <= TOL[prec] * np.linalg.norm(want)
    out = outside_rule(n)
    assert np.linalg.norm((got - want)[:, out]) <= TOL[prec] * np.linalg.norm(want[:, out])
    assert np.linalg.norm(P - Po) <= TOL[prec] * np.linalg.norm(Po)


def torch_step(U, nu, dt):
    """main.c:334-414 from the initial state (whose stale velocity is U
    itself), in torch's float64 on the GPU."""
    import torch

    n = U[0].shape[0]
    dev = torch.device("cuda")
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev)
    ks = (k.view(n, 1, 1), k.view(1, n, 1),
          torch.arange(n // 2 + 1, dtype=torch.float64, device=dev).view(1, 1, -1))
    kk = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    kmax = 2.0 / 3.0 * (n // 2 + 1)
    mask = (ks[0].abs() < kmax) & (ks[1].abs() < kmax) & (ks[2] < kmax)

    def back(X):  # FFTW's c2r over n^3: complex over x and y, real along z
        return torch.fft.irfft(torch.fft.ifft(torch.fft.ifft(X, dim=0), dim=1), n=n, dim=2)

    u = [torch.from_numpy(a).to(dev) for a in U]
    u0 = [torch.fft.rfftn(a) for a in u]
    us, acc = u0, [a.clone() for a in u0]
    for s in range(4):
        if s > 0:
            u = [back(a) for a in us]
        w = [back(1j * (ks[(f + 1) % 3] * us[(f + 2) % 3] - ks[(f + 2) % 3] * us[(f + 1) % 3])) for f in range(3)]
        d = [torch.fft.rfftn(u[(f + 1) % 3] * w[(f + 2) % 3] - u[(f + 2) % 3] * w[(f + 1) % 3]) * mask * dt
             for f in range(3)]
        del w
        p = (ks[0] * d[0] + ks[1] * d[1] + ks[2] * d[2]) / torch.where(kk > 0, kk, torch.ones_like(kk))
        for f in range(3):
            d[f] = d[f] - p * ks[f] - nu * dt * kk * us[f]
            acc[f] += (1 / 6, 1 / 3, 1 / 3, 1 / 6)[s] * d[f]
        if s < 3:
            us = [u0[f] + (0.5, 0.5, 1.0)[s] * d[f] for f in range(3)]
    return [a.cpu().numpy() for a in acc]


@pytest.fixture(scope="module")
def step_512():
    import torch

    n = 512
    U = white_field(n, n)
    want = torch_step(U, nu_for(n), DT)
    torch.cuda.empty_cache()
    return U, want


@pytest.mark.parametrize("prec", [0, 1])
def test_white_noise_step_512(dns_lib, step_512, prec):
    import dns_b200 as dns

    n = 512
    U, want = step_512
    with dns.Context(n, prec) as c:
        c.set_velocity(*U)
        c.step(nu_for(n), DT, 1)
        got = c.get_spectral()
    out = outside_rule(n)
    e = w = eo = wo = 0.0
    for f in range(3):
        d = got[f] - want[f]
        e += np.linalg.norm(d) ** 2
        w += np.linalg.norm(want[f]) ** 2
        eo += np.linalg.norm(d[out]) ** 2
        wo += np.linalg.norm(want[f][out]) ** 2
    assert e <= TOL[prec] ** 2 * w
    assert eo <= TOL[prec] ** 2 * wo


@pytest.mark.parametrize("prec", [0, 1])
def test_steps_in_one_call_equal_single_steps_512(dns_lib, prec):
    import dns_b200 as dns

    def digest(a):
        return hashlib.blake2b(np.ascontiguousarray(a).data).hexdigest()

    out = []
    for calls in ((3,), (1, 2)):
        with dns.Context(512, prec) as c:
            c.set_perturbed_tgv(5, 0.1)
            for k in calls:
                c.step(0.01, 0.002, k)
            out.append((digest(c.get_spectral()), digest(c.get_stale())))
    assert out[0] == out[1]
