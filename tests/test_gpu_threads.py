"""Stand-alone transforms of short and long lines called from several host threads at once (they hold no
handle): the kernels' shared-memory limits belong to the process."""
import threading

import numpy as np
import pytest

import mwf_gb300 as mwf
from mwf_gb300 import solver

pytestmark = pytest.mark.gpu


def test_short_and_long_lines_side_by_side(built_lib):
    long_p = mwf.RunParams(K0=4, MM=2, NN=648, alpha=0.3, gamma=0.2)       # more than 70 KB of shared memory a CTA
    short_p = mwf.RunParams(K0=4, MM=2, NN=2, alpha=0.3, gamma=0.2)
    rng = np.random.default_rng(1)
    field = {p.NN: rng.standard_normal((p.NN, p.M, p.KK)) + 1j * rng.standard_normal((p.NN, p.M, p.KK)) for p in (long_p, short_p)}
    want = {p.NN: solver.spec2phys(p, field[p.NN]) for p in (long_p, short_p)}
    wrong, done = [], threading.Event()

    def call(p):
        try:
            if not np.array_equal(solver.spec2phys(p, field[p.NN]), want[p.NN]):
                wrong.append(f"NN = {p.NN}: another result")
        except mwf.MwfError as e:
            wrong.append(f"NN = {p.NN}: {e}")

    def short():
        while not done.is_set():
            call(short_p)

    threads = [threading.Thread(target=short) for _ in range(3)]
    for t in threads:
        t.start()
    try:
        for _ in range(2000):
            call(long_p)
    finally:
        done.set()
        for t in threads:
            t.join()
    assert not wrong, (len(wrong), wrong[0])
