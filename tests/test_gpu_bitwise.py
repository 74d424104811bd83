"""FP32 (and FP64) runs keep their bits whatever else is in their handle: the columns and lines of a work item
depend on how full its launch is, and the results do not."""
import numpy as np
import pytest

import mwf_gb300 as mwf

pytestmark = pytest.mark.gpu

BATCHED = [(K0, N) for K0 in (4, 6) for N in (32, 48, 64, 96, 128, 192, 256) if not (K0 == 6 and N > 128)]


def run_params(K0, MM, NN, prec="fp32", **kw):
    return mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=3.0 / MM, gamma=3.0 / NN, dt=0.01, theta=0.3, precision=prec, **kw)


def stepped(p, c0, n=1, persistent=False):
    with mwf.Ensemble([p] * n) as ens:
        if persistent:
            ens.set_persistent(True)
        for i in range(n):
            ens.set_state(i, c0)
        ens.step(3)
        return ens.get_state(n - 1)


@pytest.mark.parametrize("K0,N", BATCHED)
def test_every_item_width_gives_the_same_bits(built_lib, K0, N):
    """Each width is a kernel body of its own; the knobs choose it."""
    p = run_params(K0, N, N)
    c0 = mwf.ic.gaussian_ic(p, seed=3)
    one = dict(xf_cols=1, xi_cols=1, z_lines=1)
    want = stepped(p.with_(**one), c0)
    assert np.array_equal(stepped(p, c0), want)
    assert np.array_equal(stepped(p, c0, persistent=True), want)
    for knob in one:
        for width in range(2, 33):
            q = p.with_(**{**one, knob: width})
            try:
                mwf.describe_run(q)
            except mwf.MwfError:                        # wider than any item of this length
                break
            assert np.array_equal(stepped(q, c0), want), (knob, width)


@pytest.mark.parametrize("prec,K0,MM,NN", [("fp32", 4, 32, 32), ("fp32", 4, 96, 48), ("fp32", 6, 64, 128), ("fp32", 4, 27, 36),
                                           ("fp32", 6, 72, 18), ("fp32", 4, 64, 54), ("fp32", 4, 162, 96), ("fp32", 4, 9, 768),
                                           ("fp64", 4, 32, 32), ("fp64", 6, 27, 48), ("fp64", 4, 6, 864)])
def test_a_checkpoint_continues_bitwise_in_another_handle(built_lib, prec, K0, MM, NN):
    """Alone; among as many of its kind as fill the chip; and moved from the one to the other after three steps."""
    p = run_params(K0, MM, NN, prec)
    c0 = mwf.ic.gaussian_ic(p, seed=3)
    other = run_params(4, 48, 48)
    with mwf.Ensemble([p]) as alone, mwf.Ensemble([other] + [p] * 40 + [other]) as full:
        alone.set_state(0, c0)
        full.set_state(7, c0)
        alone.step(3)
        full.step(3)
        ckpt = alone.checkpoint(0)
        assert all(np.array_equal(a, b) for a, b in zip(ckpt, full.checkpoint(7)))
        full.restore(30, ckpt)
        alone.step(4)
        full.step(4)
        want = alone.get_state(0)
        assert np.array_equal(full.get_state(7), want) and np.array_equal(full.get_state(30), want)
