"""The gradient's sums in three floats (kpt_sum.h) at every size of the terms
that floats have, on the CPU, denormals flushed as the kernels' build does."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "kittlespt_gb300", "csrc")


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("sum") / "float_sum")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", f"-I{CSRC}", os.path.join(HERE, "float_sum.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    return {int(line.split()[0]): float(line.split()[1]) for line in out.splitlines()}


@pytest.mark.parametrize("size", [-120, -110, -100, -90, -80, -70, -40, 0, 40, 80, 92])
def test_as_near_as_a_double(errors, size):
    # 200 terms: the value's rounding to double; that of mid + lo (mid below 200 * 2^-24); lo's, each 2^-24 of at
    # most 200 * 2^-48
    assert errors[size] <= 2.0 ** -53 * (1 + 200 * 2.0 ** -24) + 200 * 200 * 2.0 ** -72


@pytest.mark.parametrize("size", [98, 104, 120])
def test_sums_that_spill(errors, size):
    # up to 200 times to a double: two roundings of the value, one of its sum with the term, one of the double's
    assert errors[size] <= 4 * 200 * 2.0 ** -53
