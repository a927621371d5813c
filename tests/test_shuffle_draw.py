"""How the shuffle takes its engine's draws (csrc/shuffle_draw.h), built for the
host, against libstdc++: up to as many values as there are draws, and one more,
the last step of 2^31 - 1 elements, where no draw is enough by itself."""

import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_draws_are_libstdcxxs(tmp_path):
    exe = str(tmp_path / "shuffle_draw_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(REPO, "potreeconverter_b200", "csrc"),
                    os.path.join(REPO, "tests", "cpp", "shuffle_draw_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "20000"], capture_output=True, text=True, timeout=120)
    assert (r.returncode, r.stdout) == (0, "same\n"), r.stdout
