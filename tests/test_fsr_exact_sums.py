"""The float forms of EASU's weights, stretch and lobe and of the tonemap's
Yxy -> XYZ against the reference's double-precision expressions, on the CPU
(tests/fsr_exact_sums.c, the same float operations in the same order): every
input that the float form decides has to give the double form's float."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fsr") / "fsr_exact_sums")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", os.path.join(HERE, "fsr_exact_sums.c"), "-o", exe, "-lm", "-lpthread"],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {line.split()[0]: tuple(int(v) for v in line.split()[1:]) for line in out.splitlines()}


@pytest.mark.parametrize("form", ["lobe", "half", "luma", "weight00", "weight10", "stretch", "xyy"])
def test_float_form_gives_the_double_forms_float(counts, form):
    n, different, undecided = counts[form]
    assert n > 1e7 and different == 0 and undecided < n
