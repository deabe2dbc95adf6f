"""bench.py's byte model of a step (kernel_units: what its roofline and
step_hbm fields are computed from) against counts made from the fields
themselves: every array that a kernel has to read or write, with its modes
counted one by one from main.c's 2/3 rule (main.c:231-238)."""
import pytest


def counted(n, size):
    """[stage][B, C, D, X] bytes."""
    kmax = 2.0 / 3.0 * (n // 2 + 1)
    nz_in = sum(1 for k in range(n // 2 + 1) if k < kmax)
    nx_in = sum(1 for i in range(n) if abs(i if i < n // 2 else i - n) < kmax)
    c = 2 * size
    full = n * n * (n // 2 + 1) * c        # a field after any pass
    real = n ** 3 * size
    n_z = n * n * nz_in * c                # N after the z pass
    n_y = n * nx_in * nz_in * c            # N after the y forward pass
    packed = nx_in * nx_in * nz_in * c     # a stage input inside the rule
    out = []
    for s in range(4):
        first, last = s == 0, s == 3
        read = {"u": full, "v": full, "w": full, "dv/dx": full, "dw/dx": full}
        write = {"u": full, "v": full, "omega_z": full, "dw/dx": full, "dw/dy": full}
        if not first:
            write["w"] = full
        B = sum(read.values()) + sum(write.values())
        C = sum(write.values()) + 3 * n_z + (3 * real if first or last else 0)
        D = 3 * n_z + 3 * n_y
        kept = {0: 0, 1: 1, 2: 1, 3: 3}[s]  # U_0 is the state; stage 3 reads U_1, U_2 and U_3
        X = 3 * n_y + 3 * full + kept * 3 * packed + 5 * full + (3 * full if last else 3 * packed)
        out.append([B, C, D, X])
    return out


@pytest.mark.parametrize("n,size", [(8, 8), (32, 8), (64, 4), (256, 8), (256, 4), (512, 8)])
def test_kernel_bytes_match_counted_fields(n, size):
    import bench

    want = counted(n, size)
    got = bench.kernel_bytes(n, size)
    for s in range(4):
        assert got[s] == pytest.approx(want[s], rel=1e-12), s
    assert bench.step_bytes(n, size) == pytest.approx(sum(map(sum, want)), abs=8)


def test_step_bytes_256_fp64():
    import bench

    assert abs(bench.step_bytes(256) / 1e9 - 19.04) < 0.01


def test_kernel_times_sum_to_the_step():
    """Every pass of dns_time_kernels is counted in exactly one kernel."""
    import numpy as np

    import bench

    kms = np.arange(1.0, 25.0).reshape(4, 6)
    kt = np.array(bench.kernel_times(kms))
    assert kt.shape == (4, 4) and kt.sum() == kms.sum()


def test_reference_arm_without_the_reference(monkeypatch, capsys, tmp_path):
    """Without the reference's binary the arm reports no figure of its own."""
    import argparse
    import json

    import bench
    import oracle

    monkeypatch.setattr(oracle, "REF_DNS", str(tmp_path / "dns"))
    args = argparse.Namespace(n=16, gpus=1, steps=1, warmup=3)
    assert bench.run_reference_arm(args, 1, 0) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "unavailable" in line and "value" not in line
