"""The adjoint's fused z part at its smallest plan, at n = 64 (8 values per
thread) and at n = 128 in FP32 (16 values): FP64 against central finite
differences (eps = 1e-6: truncation ~1e-12, rounding of J ~1e-16 / 1e-6, so
1e-6 relative leaves a margin of 1e3), mixed against FP64 (FP32 rounding of
some 20 transforms a step, 1e-4 as in the other adjoint tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 64])
def test_gradient_matches_finite_differences(dns_lib, n):
    import dns_b200 as dns

    nu, dt, steps = 0.02, 0.005, 3
    u0 = dns.perturbed_tgv(n, seed=9, amplitude=0.3)
    J, g, gnu = dns.adjoint_energy(*u0, nu, dt, steps, snapshots=2)
    assert J == pytest.approx(dns.final_energy(*u0, nu, dt, steps), rel=1e-15)
    # a direction along the field itself plus a solenoidal one: dJ is not small
    d = [a + b for a, b in zip(u0, dns.solenoidal_perturbation(n, seed=4))]
    eps = 1e-6
    Jp = dns.final_energy(*(u + eps * q for u, q in zip(u0, d)), nu, dt, steps)
    Jm = dns.final_energy(*(u - eps * q for u, q in zip(u0, d)), nu, dt, steps)
    fd, ad = (Jp - Jm) / (2 * eps), float(sum(np.sum(a * b) for a, b in zip(g, d)))
    assert abs(fd - ad) <= 1e-6 * abs(ad), (fd, ad)


@pytest.mark.parametrize("n", [8, 64, 128])
def test_mixed_gradient_against_fp64(dns_lib, n):
    import dns_b200 as dns

    nu, dt, steps = 0.02, 0.005, 3
    u0 = dns.perturbed_tgv(n, seed=9, amplitude=0.3)
    J, g, gnu = dns.adjoint_energy(*u0, nu, dt, steps, snapshots=2)
    J32, g32, gnu32 = dns.adjoint_energy(*u0, nu, dt, steps, snapshots=2,
                                         precision=dns.DNS_PREC_MIXED)
    e = np.sqrt(sum(np.sum((a - b) ** 2) for a, b in zip(g32, g)) / sum(np.sum(b ** 2) for b in g))
    assert abs(J32 - J) <= 1e-5 * J and e <= 1e-4 and abs(gnu32 - gnu) <= 1e-4 * abs(gnu)
