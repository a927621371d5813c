"""The hierarchy writer (potreeconverter_b200/csrc/writers.cpp), built for the
host, against the oracle's hierarchy.bin at the depths where the form of a
node's number changes: names of up to 21, 42 and more levels. A header box that
is long in one axis makes such trees: the cube takes that axis' size, the
points keep the others' scale."""

import os
import struct
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "potreeconverter_b200", "csrc")


def long_box(length, n=24_000, along=2_000):
    """n points within 10 m in y and z at one end of a header box `length` m
    long in x, and `along` more along it."""
    from potreeconverter_b200 import synth
    las = bytearray(synth.terrain(n + along, 5))
    off, rec = struct.unpack_from("<I", las, 96)[0], struct.unpack_from("<H", las, 105)[0]
    points = np.frombuffer(las, dtype=np.uint8)[off:].reshape(n + along, rec).copy()
    rng = np.random.default_rng(3)
    xyz = rng.integers(0, 10_000, (n + along, 3)).astype("<i4")
    xyz[:n, 0] = 0
    xyz[n:, 0] = rng.integers(0, 10 ** 9, along)
    points[:, :12] = xyz.view(np.uint8).reshape(n + along, 12)
    struct.pack_into("<12d", las, 131, length / 1e9, 0.001, 0.001, *[0.0] * 3, length, 0.0, 10.0, 0.0, 10.0, 0.0)
    las[off:] = points.tobytes()
    return bytes(las)


@pytest.fixture(scope="module")
def hierarchy(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("hierarchy") / "hierarchy_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(REPO, "include"),
                    os.path.join(REPO, "tests", "cpp", "hierarchy_check.cpp"), os.path.join(CSRC, "writers.cpp"),
                    os.path.join(CSRC, "setup.cpp"), "-o", exe], check=True)

    def build(nodes):
        text = "".join(f"{name} {offset} {size} {points}\n" for name, offset, size, points in nodes)
        return subprocess.run([exe], input=text.encode(), check=True, capture_output=True).stdout

    return build


@pytest.mark.parametrize("length,levels", [(1e3, 8), (1e7, 21), (2e7, 22), (2e13, 42), (4e13, 43), (1e15, 48), (1e18, 58)])
def test_deep_trees(hierarchy, oracle, length, levels):
    want = oracle.convert(long_box(length), "poisson")
    assert max(len(name) for name, *_ in want["nodes"]) - 1 == levels
    assert hierarchy(want["nodes"]) == want["hierarchy.bin"]
