"""The FP32 passes with a warp per line (mwf_zwarp.cuh, mwf_xwarp.cuh) against the FP64 oracle, and
against the kernels with run-time plans that a radix cap selects."""
import numpy as np
import pytest

from oracle import mwf_oracle as O
import mwf_gb300 as mwf
from test_gpu_parity import oracle_params

# Every radix (2, 3, 4, 6, 8, 9, 12, 16) first and last, padded and unpadded lines, one to four stages,
# odd lengths, several short lines per warp, last items with fewer lines or columns, the three
# subsets at once and in turn, a team of two warps per line, one pass batched beside the other
SHAPES = [(4, 2, 2), (4, 3, 9), (6, 9, 2), (4, 16, 16), (4, 27, 6), (4, 12, 27), (6, 24, 36), (4, 54, 81), (6, 18, 54),
          (6, 12, 192), (6, 8, 256), (4, 6, 384), (4, 4, 512), (6, 4, 512), (6, 4, 864), (4, 4, 972), (4, 3, 1024), (4, 1024, 3),
          (4, 768, 4), (4, 64, 36), (4, 36, 64)]


def norm(a):
    return np.sqrt((np.abs(a) ** 2).sum())


@pytest.mark.gpu
@pytest.mark.parametrize("K0,MM,NN", SHAPES)
def test_nonlinear_term_and_step_against_the_oracle(built_lib, K0, MM, NN):
    """One Euler step; the history it leaves is the projected nonlinear term.  FP32 rounds at 6e-8; a
    few tens of operations deep, and with derivatives up to the largest wavenumber, the term
    is held to 1e-5 of its norm and the state (one rounding plus dt times that) to 1e-6."""
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=3.0 / MM, gamma=3.0 / NN, Re=200, dt=0.01, theta=0.3, precision="fp32")
    c0 = mwf.ic.gaussian_ic(p, seed=1)
    s = O.Solver(oracle_params(p), c0)
    s.step(1)
    with mwf.Ensemble([p]) as ens:
        ens.set_state(0, c0)
        ens.step(1)
        h, _ = ens.get_history(0)
        g = ens.get_state(0)
    assert norm(h - s.onl) <= 1e-5 * norm(s.onl)
    assert norm(g - s.c) <= 1e-6 * norm(s.c)


@pytest.mark.gpu
@pytest.mark.parametrize("K0,MM,NN", [(4, 27, 36), (6, 54, 24), (4, 96, 162), (6, 256, 256)])
def test_same_steps_as_the_run_time_plan_kernels(built_lib, K0, MM, NN):
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=3.0 / MM, gamma=3.0 / NN, Re=200, dt=0.01, precision="fp32")
    c0 = mwf.ic.gaussian_ic(p, seed=4)
    with mwf.Ensemble([p, p.with_(z_radix=8, x_radix=8), p]) as ens:
        for i in range(3):
            ens.set_state(i, c0)
        ens.set_active(2, False)
        ens.step(5)
        a, b, c = (ens.get_state(i) for i in range(3))
    assert norm(a - b) <= 2e-6 * norm(b)          # five roundings of the state on either side
    assert np.array_equal(c, c0.astype(np.complex64))


@pytest.mark.gpu
def test_a_non_finite_run_fails_alone(built_lib):
    p = mwf.RunParams(K0=4, MM=27, NN=36, alpha=0.3, gamma=0.2, Re=200, dt=0.01, precision="fp32")
    good = mwf.ic.gaussian_ic(p, seed=1)
    with mwf.Ensemble([p, p, p]) as ens:
        bad = good.copy()
        bad[3, 5, 2] = np.nan
        ens.set_state(1, bad)
        ens.set_state(2, good)
        ens.step(2)
        assert np.all(ens.get_state(0) == 0)
        with pytest.raises(mwf.MwfError):
            ens.energy(1)
        both = ens.get_state(2)
    with mwf.Ensemble([p]) as ens:
        ens.set_state(0, good)
        ens.step(2)
        assert np.array_equal(ens.get_state(0), both)


def test_plans_fit_the_kernels():
    smooth = sorted(2 ** a * 3 ** b for a in range(11) for b in range(7) if 2 <= 2 ** a * 3 ** b <= 1024)
    for K0 in (4, 6):
        for N in smooth:
            if K0 == 6 and N == 1024:        # no z kernel holds it: refused when the handle is made
                continue
            d = mwf.describe_run(mwf.RunParams(K0=K0, MM=N, NN=N, alpha=0.1, gamma=0.1, precision="fp32"))
            assert max(d["xf_smem"], d["z_smem"], d["xi_smem"]) <= 232448
            assert d["z_items"] == -(-3 * N // d["z_lines"])
            if not d["batched_x"]:
                assert d["xf_items"] == -(-N // d["xf_cols"]) * K0 and d["xi_items"] == -(-N // d["xi_cols"]) * K0


@pytest.mark.gpu
@pytest.mark.parametrize("K0,MM,NN", [(4, 32, 32), (6, 64, 48), (4, 27, 36), (6, 72, 18), (4, 64, 54), (4, 128, 2)])
def test_a_run_alone_and_among_many(built_lib, K0, MM, NN):
    """A launch that its runs do not fill takes narrower items: the same sums in the same order for each
    line, so a run steps alike alone and among as many as fill the launch, to the rounding of differently
    contracted products (a few 6e-8 of the state's norm in three steps)."""
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=3.0 / MM, gamma=3.0 / NN, dt=0.01, precision="fp32")
    c0 = mwf.ic.gaussian_ic(p, seed=3)
    out = []
    for n in (1, 5, 40):
        with mwf.Ensemble([p] * n) as ens:
            for i in range(n):
                ens.set_state(i, c0)
            ens.step(3)
            out += [ens.get_state(0), ens.get_state(n - 1)]
    for g in out[1:]:
        assert np.linalg.norm(g - out[0]) <= 1e-6 * np.linalg.norm(out[0])
