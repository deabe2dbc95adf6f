"""The x pass (RK update between the x transforms) where it can go wrong:
the smallest and largest plans, tiles that straddle the 2/3 rule and the
Nyquist column, modes outside the rule, and the two forms of the last
stage (with and without the next step's transform)."""
import numpy as np
import pytest

from conftest import random_field

pytestmark = pytest.mark.gpu

# single steps: the tolerances of the other step tests (FP64 rounding of a
# few transforms; FP32 rounding, 2^-24 = 6e-8, of some 30 operations a value)
TOL = {0: 1e-13, 1: 1e-5}


@pytest.fixture(scope="module")
def dns(dns_lib):
    import dns_b200

    return dns_b200


def white_field(n, seed):
    """White noise: every mode of the grid, outside the 2/3 rule too."""
    rng = np.random.default_rng(seed)
    return [0.1 * rng.standard_normal((n, n, n)) for _ in range(3)]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [8, 16, 32, 64, 128])
def test_white_noise_steps_match_oracle(dns, oracle_lib, n, prec):
    """nu large enough that the modes outside the rule decay visibly
    (nu dt |k|^2 up to ~1 at the corner) but stay stable."""
    dt = 2e-3
    nu = 1.0 / (dt * 3 * (n / 2) ** 2)
    U, V, W = white_field(n, n)
    o = oracle_lib.Oracle(n)
    o.set_velocity(U, V, W)
    o.step(nu, dt, 2)
    want = o.get_spectral()
    with dns.Context(n, prec, dns.DNS_FLAG_PRESSURE) as c:
        c.set_velocity(U, V, W)
        c.step(nu, dt, 2)
        got = c.get_spectral()
        P = c.get_fields(pressure=True)[3]
    assert np.linalg.norm(got - want) <= TOL[prec] * np.linalg.norm(want)
    k = np.abs(np.fft.fftfreq(n, 1.0 / n))
    kz = np.arange(n // 2 + 1)
    kmax = 2.0 / 3.0 * (n // 2 + 1)
    out = (k[:, None, None] >= kmax) | (k[None, :, None] >= kmax) | (kz[None, None, :] >= kmax)
    assert np.linalg.norm((got - want)[:, out]) <= TOL[prec] * np.linalg.norm(want[:, out])
    Po = o.dump_fields()[3]
    assert np.linalg.norm(P - Po) <= TOL[prec] * np.linalg.norm(Po)


@pytest.mark.parametrize("n,prec", [(8, 0), (16, 1), (64, 1), (128, 0), (256, 0), (256, 1), (512, 1)])
def test_steps_in_one_call_equal_single_steps(dns, n, prec):
    """A call's last step ends without the next step's x transform, its
    others with it: the bits are the same."""
    if n == 512:
        out = []
        for calls in ((3,), (1, 2)):
            with dns.Context(n, prec) as c:
                c.set_perturbed_tgv(5, 0.1)
                for k in calls:
                    c.step(0.01, 0.002, k)
                out.append(c.diagnostics_dd())
        assert out[0] == out[1]
        return
    U, V, W = random_field(n, 11) if n < 256 else dns.perturbed_tgv(n, 5, 0.1)
    out = []
    for calls in ((3,), (1, 1, 1), (2, 1)):
        with dns.Context(n, prec) as c:
            c.set_velocity(U, V, W)
            for k in calls:
                c.step(0.01, 0.002, k)
            out.append((c.get_spectral(), c.get_stale()))
    for uh, stale in out[1:]:
        assert np.array_equal(uh.view(np.float64), out[0][0].view(np.float64))
        assert np.array_equal(stale, out[0][1])
