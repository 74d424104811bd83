"""Lines transformed on their own in fixed point (mwf_fxlines.cuh): the stand-alone transforms against
the oracle, the physical field and the diagnostics of a run against the FP64-arithmetic kernels,
which any tuning knob selects."""
import numpy as np
import pytest

from oracle import mwf_oracle as O
import mwf_gb300 as mwf
from mwf_gb300 import solver
from test_gpu_parity import oracle_params

pytestmark = pytest.mark.gpu

# the shortest lines, odd ones, last blocks of columns and pairs that are narrower, a warp per subset
# (N > 85) and per line, few pairs to a CTA, the longest z lines, and the next one, which FP64
# arithmetic keeps; for the diagnostics the lines on both sides of what fits a CTA (M4: 648, 729)
SHAPES = [(4, 2, 2), (4, 3, 9), (6, 9, 2), (4, 16, 16), (6, 81, 96), (4, 96, 81), (6, 4, 486), (6, 3, 512), (4, 2, 648),
          (4, 2, 729), (4, 2, 768), (4, 2, 864), (4, 1024, 3)]


@pytest.mark.parametrize("scale", [1.0, 1e-200, 1e200])
@pytest.mark.parametrize("K0,MM,NN", SHAPES)
def test_transforms_against_the_oracle(built_lib, K0, MM, NN, scale):
    """Both sides round log2(3N) stages at 1.1e-16 of the line's norm: 1e-13 of the field's norm is two
    orders of headroom.  One field is 1e-12 of the others, and its partner in the pair must not cost it
    more than its own line's rounding at the pair's scale."""
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=0.3, gamma=0.45)
    op = oracle_params(p)
    rng = np.random.default_rng(K0 * 1000 + MM + NN)
    s = rng.standard_normal((NN, p.M, p.KK)) + 1j * rng.standard_normal((NN, p.M, p.KK))
    s[..., 3] *= 1e-12
    s *= scale

    def norm(a):
        return np.sqrt((np.abs(a / scale) ** 2).sum())
    ph, ref = solver.spec2phys(p, s), O.spec2phys(op, s)
    assert norm(ph - ref) <= 1e-13 * norm(ref)
    back, ref_back = solver.phys2spec(p, ref), O.phys2spec(op, ref)
    assert norm(back - ref_back) <= 1e-13 * norm(ref_back)


@pytest.mark.parametrize("K0,MM,NN", SHAPES)
def test_field_and_diagnostics_against_fp64_arithmetic(built_lib, K0, MM, NN):
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=0.3, gamma=0.2, Re=200, dt=0.01)
    c0 = mwf.ic.gaussian_ic(p, seed=5)
    with mwf.Ensemble([p, p.with_(z_radix=8)]) as ens:
        for i in range(2):
            ens.set_state(i, c0)
        a, b = ens.get_phys(0), ens.get_phys(1)
        assert np.abs(a - b).max() <= 1e-13 * np.abs(b).max()
        ep = np.sort(O.epos(K0, b).ravel())
        k = int(0.7 * ep.size)
        ct = 0.5 * (ep[k] + ep[k + 1])
        (ca, ea), (cb, eb) = ens.phys_diagnostics(0, ct), ens.phys_diagnostics(1, ct)
        assert ca == cb and abs(ea - eb) <= 1e-13 * eb


def test_non_finite_and_zero_fields(built_lib):
    """A NaN or an infinity stays in its lines and makes all of them NaN; zeros stay zeros."""
    p = mwf.RunParams(K0=4, MM=9, NN=16, alpha=0.3, gamma=0.2)
    s = np.zeros((p.NN, p.M, p.KK), complex)
    assert not solver.spec2phys(p, s).any()
    s[3, 2, 10] = np.nan
    s[:, :, 4] = 1.0
    ph = solver.spec2phys(p, s)
    assert np.isnan(ph[..., 10]).all() and np.isfinite(ph[..., :10]).all()
    ph = np.zeros((p.X, p.Z, p.KK))
    ph[4, 5, 10] = np.inf
    back = solver.phys2spec(p, ph)
    assert np.isnan(back[..., 10]).all() and not back[..., :10].any()
