"""The rules of the memory kept between calls (asr_b200/csrc/devmem.h) on a made-up device: what stays, what is given back
and when, without a GPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("devmem") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(HERE, "fake_cuda"),
                    os.path.join(HERE, "devmem_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("case", ["reuse", "many", "scarce", "scarce_later", "contexts", "lasting", "planned", "limit"])
def test_devmem(check, case):
    r = subprocess.run([check, case], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
