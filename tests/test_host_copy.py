"""The threaded host copy (potreeconverter_b200/csrc/host_copy.h), built for
the host: the same bytes with all the threads it asks for, with some and with
none, at sizes around the 8 MiB from which another thread is used."""

import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("copy") / "host_copy_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", "-I" + os.path.join(REPO, "potreeconverter_b200", "csrc"),
                    os.path.join(REPO, "tests", "cpp", "host_copy_check.cpp"), "-o", exe, "-ldl", "-pthread"], check=True)
    return exe


@pytest.mark.parametrize("threads", [0, 1, 3, 100])
@pytest.mark.parametrize("size", [0, 1, (16 << 20) - 1, 16 << 20, (24 << 20) + 7, (80 << 20) + 1])
def test_copy_with_as_many_threads_as_there_are(check, threads, size):
    r = subprocess.run([check, str(threads), str(size)], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "same\n"), r.stderr
