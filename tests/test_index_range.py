"""Index arithmetic at the ends of the 32-bit range (kpt_index.h), on the CPU:
every index that a thread takes lies in its array, and each is taken once."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "kittlespt_gb300", "csrc")


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("index") / "index_range")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", os.path.join(HERE, "index_range.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    return {line.split()[0]: tuple(int(v) for v in line.split()[1:]) for line in out.splitlines()}


@pytest.mark.parametrize("walk", ["sky", "queue", "refit"])
def test_every_index_is_taken_once_and_in_range(counts, walk):
    places, wrong = counts[walk]
    assert places > 1000 and wrong == 0
