"""The warp decoder of LAZ chunks against the scalar decoder of laz.cuh built
for the host: coded flight segments of every point format at chunk sizes
around the 32 records that leave together, and chunks of random bytes, which
reach every model, class and GPS-time path (with and without extra bytes).
Malformed chunks are refused by both."""

import os
import struct
import subprocess

import numpy as np
import pytest

import potreeconverter_b200 as pc
from perf import cases
from potreeconverter_b200 import synth

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def host_decode(tmp_path_factory):
    d = tmp_path_factory.mktemp("laz")
    exe = str(d / "laz_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + os.path.join(REPO, "potreeconverter_b200", "csrc"),
                    os.path.join(REPO, "tests", "cpp", "laz_check.cpp"), "-o", exe], check=True)

    def decode(laz):
        (d / "in.laz").write_bytes(laz)
        r = subprocess.run([exe, str(d / "in.laz"), str(d / "out.bin")], capture_output=True)
        return (d / "out.bin").read_bytes() if r.returncode == 0 else None

    return decode


def device_decode(ctx, laz):
    try:
        return ctx.laz_decode(laz)
    except pc.PcgError as e:
        assert e.status == 1, e
        return None


def image(chunks, counts, chunk_size, pdrf, extra):
    """A LAZ image of the given chunk bytes."""
    rec = cases.REC_LEN[pdrf] + extra
    items = [(6, 20)] + [(7, 8)] * (pdrf in (1, 3)) + [(8, 6)] * (pdrf in (2, 3)) + [(0, extra)] * (extra > 0)
    vlr = struct.pack("<HHBBHIIqqH", 2, 0, 3, 4, 3, 0, chunk_size, -1, -1, len(items)) + b"".join(struct.pack("<HHH", t, s, 2) for t, s in items)
    record = bytearray(54)
    record[2:16] = b"laszip encoded"
    struct.pack_into("<HH", record, 18, 22204, len(vlr))
    head = bytearray(synth.las_header(sum(counts), pdrf=pdrf, version_minor=2, record_length=rec, vlrs=bytes(record) + vlr, has_extra=True,
                                      scale=(0.001,) * 3, offset=(0.0,) * 3, bbox=(1, 0, 1, 0, 1, 0), by_return=np.array([sum(counts), 0, 0, 0, 0])))
    head[104] |= 0x80
    table, sizes, last = cases._Encoder(), cases._Residuals(32, 2), 0
    for c in chunks:
        sizes.code(table, last, len(c), 1)
        last = len(c)
    body = b"".join(chunks)
    return bytes(head) + struct.pack("<q", len(head) + 8 + len(body)) + body + struct.pack("<II", 0, len(chunks)) + table.finish() + bytes(8)


@pytest.mark.parametrize("pdrf", [0, 1, 2, 3])
@pytest.mark.parametrize("points,chunk", [(2, 1), (97, 32), (100, 33), (12_345, 4_000), (30_000, 30_000)])
def test_coded_segments(gpu_ctx, host_decode, pdrf, points, chunk):
    laz = cases._laz(dict(points=points, chunk=chunk, pdrf=pdrf), 11 + pdrf)
    want = host_decode(laz)
    assert want is not None
    assert gpu_ctx.laz_decode(laz) == want


@pytest.mark.parametrize("pdrf", [0, 1, 2, 3])
@pytest.mark.parametrize("extra", [0, 1, 7, 64])
def test_random_chunks(gpu_ctx, host_decode, pdrf, extra):
    decoded = refused = 0
    for seed in range(12):
        rng = np.random.default_rng([seed, pdrf, extra])
        count = int(rng.integers(2, 900))
        rec = cases.REC_LEN[pdrf] + extra
        size = rec + 4 + count * (rec + 24) if seed % 4 else int(rng.integers(rec, rec + 40 + 8 * count))
        data = rng.integers(0, 256, size, dtype=np.uint8)
        if seed % 3 == 0:  # long runs drive the coder into its first and last symbols
            data[rec:] = np.repeat(rng.choice([0, 255, 128, 1], size - rec), 1)
        laz = image([data.tobytes()], [count], count, pdrf, extra)
        want = host_decode(laz)
        got = device_decode(gpu_ctx, laz)
        assert (got is None) == (want is None), seed
        if want is None:
            refused += 1
        else:
            decoded += 1
            assert got == want, seed
    assert decoded + refused == 12
