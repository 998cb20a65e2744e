"""The entries of the bond-order table (csrc/bond_table.cuh) on the host: every accepted entry, evaluated in FP32 as the
kernels do (plain and fine), against b and b' in long double, for 401 values of beta and beta s from 0.05 to 8.

Bounds: b to 7e-8 of its size (one FP32 rounding, 6e-8, and what the polynomial adds, less than 1e-8); b' to 2e-7 of the
entry's largest (6e-8 of interpolation; FP32 coefficients and the last of the FMAs, two roundings), fine 1.3e-7 (without
the coefficient's), or of 1e-3 / s.
Up to n = 5 every entry is accepted, so ordinary sets never leave the table."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("bond") / "bond_table_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "bond_table_check.cpp")], check=True)

    def run(*args):
        out = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, check=True).stdout.split()
        return int(out[0]), int(out[1]), *map(float, out[2:])
    return run


@pytest.mark.parametrize("n", [0.3, 0.5, 0.787, 1, 1.5, 2, 3, 4, 5, 6, 8, 10, 12, 16, 22.956, 35, 50])
def test_accepted_entries_are_exact(check, n):
    total, accepted, eb, ed, eb_fine, ed_fine, _ = check(n, 0.05, 8)
    assert max(eb, eb_fine) <= 7e-8 and ed <= 2e-7 and ed_fine <= 1.3e-7
    assert accepted == total if n <= 5 else 0.8 * total <= accepted < total


def test_small_arguments(check):
    """Down to where b = 1 and b' = 0, and below the FP32 range of the powers of 1 / h."""
    for n in (0.5, 1, 4):
        total, accepted, eb, ed, *_ = check(n, 1e-14, 1e-8)
        assert accepted > 0 and eb <= 7e-8 and ed <= 2e-7


@pytest.mark.parametrize("n", [0.3, 0.787, 1.5, 3, 5])
def test_no_bias_within_an_entry(check, n):
    """The bonds of a crystal share few entries: in the fine evaluation the mean error of b' over an entry, 1024 roundings of up to 6e-8 that
    average out (five standard deviations: 6e-9), stays below 1e-8 where a rounded first coefficient alone has up to 6e-8."""
    assert check(n, 0.05, 8)[6] <= 1e-8
