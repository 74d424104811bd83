"""The FP64 passes in 64-bit fixed point (mwf_fx.cuh, mwf_fxpass.cuh) against the oracle and against
the FP64-arithmetic kernels, which any tuning knob selects."""
import numpy as np
import pytest

from oracle import mwf_oracle as O
import mwf_gb300 as mwf
from test_gpu_parity import oracle_params

# Shapes where the passes change: the shortest lines, odd ones, one line longer and shorter than a
# warp's butterflies, last blocks of columns and lines that are narrower, radix 9 and 3 stages, the
# longest z lines of the fixed-point pass for each model, and the next one, which FP64 arithmetic keeps
SHAPES = [(4, 2, 2), (4, 3, 9), (6, 9, 2), (4, 16, 16), (4, 12, 27), (6, 16, 24), (6, 27, 32), (4, 81, 54),
          (4, 6, 243), (6, 4, 486), (6, 8, 512), (4, 4, 768), (4, 4, 864), (4, 1024, 4)]


def norm(a):
    return np.sqrt((np.abs(a) ** 2).sum())


def state(p, kind):
    c = mwf.ic.gaussian_ic(p, seed=1)
    if kind == "white":                       # every retained coefficient alike: the widest lines
        rng = np.random.default_rng(2)
        w = rng.standard_normal(p.shape) + 1j * rng.standard_normal(p.shape)
        w[0] = c[0]
        c = w
    return c * (1e-8 if kind == "tiny" else 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["gauss", "white", "tiny"])
@pytest.mark.parametrize("K0,MM,NN", SHAPES)
def test_nonlinear_term_and_step_against_the_oracle(built_lib, K0, MM, NN, kind):
    """One Euler step: the AB2 history it leaves is the projected nonlinear term itself.  Both sides
    round a few hundred operations per coefficient at 1.1e-16 of the term's norm, so 1e-13 of it is two
    orders of headroom; the tiny state checks that the O(1) base flow does not set the scale of
    the perturbation's derivatives."""
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=3.0 / MM, gamma=3.0 / NN, Re=200, dt=0.01, theta=0.3)
    c0 = state(p, kind)
    s = O.Solver(oracle_params(p), c0)
    s.step(1)
    with mwf.Ensemble([p]) as ens:
        ens.set_state(0, c0)
        ens.step(1)
        h, euler = ens.get_history(0)
        g = ens.get_state(0)
    assert not euler
    assert norm(h - s.onl) <= 1e-13 * norm(s.onl)
    assert norm(g - s.c) <= 1e-13 * norm(s.c)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [{}, {"theta": 0.7, "dragall": False}, {"hypo": 1e-3, "vdrag": 0.02},
                                {"reflect": True}, {"uvreflect": True, "wreflect": True}])
def test_same_steps_as_the_fp64_arithmetic_kernels(built_lib, kw):
    p = mwf.RunParams(K0=4, MM=18, NN=27, alpha=0.3, gamma=0.2, Re=200, dt=0.01, **kw)
    c0 = mwf.ic.gaussian_ic(p, seed=4)
    with mwf.Ensemble([p, p.with_(z_radix=8)]) as ens:
        for i in range(2):
            ens.set_state(i, c0)
        ens.step(5)
        a, b = ens.get_state(0), ens.get_state(1)
    assert norm(a - b) <= 1e-12 * norm(b)


@pytest.mark.gpu
def test_zero_and_non_finite_states(built_lib):
    """The laminar state stays exactly laminar; a NaN or an infinity anywhere makes its own run
    non-finite and no other."""
    p = mwf.RunParams(K0=6, MM=12, NN=18, alpha=0.3, gamma=0.2, Re=200, dt=0.01)
    good = mwf.ic.gaussian_ic(p, seed=1)
    with mwf.Ensemble([p, p, p, p]) as ens:
        for i, v in ((1, np.nan), (2, np.inf)):
            c = good.copy()
            c[3, 5, 2] = v
            ens.set_state(i, c)
        ens.set_state(3, good)
        ens.step(2)
        assert np.all(ens.get_state(0) == 0)
        for i in (1, 2):
            with pytest.raises(mwf.MwfError):
                ens.energy(i)
        alone = ens.get_state(3)
        assert np.isfinite(ens.energy(3))
    with mwf.Ensemble([p]) as ens:
        ens.set_state(0, good)
        ens.step(2)
        assert np.array_equal(ens.get_state(0), alone)


def test_plans_fit_the_kernels():
    """Every FP64 size: items cover the grid, column blocks are powers of two (host only)."""
    smooth = sorted(2 ** a * 3 ** b for a in range(11) for b in range(7) if 2 <= 2 ** a * 3 ** b <= 1024)
    for K0 in (4, 6):
        for N in smooth:
            if N > 512 and K0 == 6:
                continue
            d = mwf.describe_run(mwf.RunParams(K0=K0, MM=N, NN=N, alpha=0.1, gamma=0.1))
            assert max(d["xf_smem"], d["z_smem"], d["xi_smem"]) <= 232448 - 1024
            assert d["xf_items"] == -(-N // d["xf_cols"]) * 2 * (3 * K0 - 1)
            assert d["xi_items"] == -(-N // d["xi_cols"]) * K0
            assert d["z_items"] == -(-3 * N // d["z_lines"]) * 3
            if N <= 512:
                assert d["xf_cols"] in (1, 2, 4, 8) and d["xi_cols"] in (1, 2, 4, 8)
