"""Several contexts in several threads of one process: their kernels are the
same functions, so what one thread asks of a function (how much shared memory
a launch may take) must not take it away from another."""

import threading

import numpy as np
import pytest

import potreeconverter_b200 as pc
from perf import cases
from tests.test_gpu_accept import OFFSET, SCALE, SIDE, node

pytestmark = pytest.mark.gpu
THREADS = 8


def all_equal(calls, repeats):
    """Every thread makes its own call `repeats` times on its own context and
    compares what it gets with what the call gave alone."""
    with pc.Context() as ctx:
        alone = [c(ctx) for c in calls]
    failures, start = [], threading.Barrier(THREADS)

    def work(k):
        call, want = calls[k % len(calls)], alone[k % len(calls)]
        try:
            with pc.Context() as ctx:
                start.wait()
                for _ in range(repeats):
                    if call(ctx) != want:
                        failures.append(f"thread {k}: another result")
                        return
        except Exception as e:  # noqa: BLE001 - reported below
            failures.append(f"thread {k}: {e}")
            start.abort()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(THREADS)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_acceptance_of_nodes_of_different_sizes():
    # a node's batch, and with it the shared memory of its block, grows up to
    # 81,920 candidates: 40,000 and 60,000 are decided by one kernel, 70,000 and
    # 150,000 by another
    def call(n):
        q, child = node("sheet", n, 5)
        return lambda ctx: ctx.accept("poisson", q[:, 0], q[:, 1], q[:, 2], child, SCALE, OFFSET, np.zeros(3), np.full(3, SIDE), 1.0, None)[0].tobytes()

    all_equal([call(n) for n in (40_000, 60_000, 70_000, 150_000)], 150)


def test_laz_files_of_different_chunk_counts():
    # 8, 200, 400 and 550 chunks: one to four blocks an SM share its memory
    images = [cases._laz(dict(points=p, chunk=c, pdrf=3), 7) for p, c in ((160, 20), (4_000, 20), (8_000, 20), (11_000, 20))]
    all_equal([lambda ctx, z=z: ctx.laz_decode(z) for z in images], 300)
