"""dns_time_kernels times the step that dns_step repeats: the passes that
share a kernel get equal shares of it, the last stage's E1 and E2 with the next
step's A among them, and the state advances as by dns_step."""
import numpy as np
import pytest

from conftest import random_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,prec", [(8, 1), (32, 0), (64, 0), (128, 1)])
def test_shares_of_fused_kernels_and_state(dns_lib, n, prec):
    import dns_b200 as dns

    U = random_field(n, 5)
    with dns.Context(n, prec) as c, dns.Context(n, prec) as d:
        for x in (c, d):
            x.set_velocity(*U)
        ms = c.time_kernels(0.01, 0.002, 3)
        d.step(0.01, 0.002, 3)
        assert np.array_equal(c.get_spectral().view(np.float64), d.get_spectral().view(np.float64))
        assert np.array_equal(c.get_stale(), d.get_stale())
    assert ms.shape == (24,) and np.all(ms > 0)
    p = ms.reshape(4, 6)
    for s in range(4):
        assert p[s, 4] == p[s, 5] == p[(s + 1) % 4, 0]
        if n <= 32:
            assert p[s, 1] == p[s, 2] == p[s, 3]
