"""State copies through pinned arrays, which the device accesses in place, and through pageable ones,
which are staged: the same values; and the energy call's non-finite check."""
import numpy as np
import pytest

import mwf_gb300 as mwf

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("K0,MM,NN", [(4, 2, 2), (6, 27, 16), (4, 48, 32)])
def test_pinned_and_pageable_copies_agree(built_lib, K0, MM, NN, prec):
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=0.3, gamma=0.2, dt=0.01, precision=prec)
    rng = np.random.default_rng(1)
    n = p.dof
    with mwf.Ensemble([p, p]) as ens:
        block = pinned(2 * n + 3)                       # views inside one pinned allocation, odd offset
        re, im = block[1:n + 1], block[n + 2:2 * n + 2]
        re[:], im[:] = rng.standard_normal(n), rng.standard_normal(n)
        ens.set_state_ref(0, re, im)                    # both pinned
        ens.set_state_ref(1, re.copy(), im.copy())      # both pageable
        a, b = ens.get_state(0), ens.get_state(1)
        want = (re + 1j * im).reshape(p.shape)
        assert np.array_equal(a, want if prec == "fp64" else want.astype(np.complex64))
        assert np.array_equal(a, b)
        ens.set_state_ref(1, re, im.copy())             # one of each: staged
        assert np.array_equal(ens.get_state(1), a)
        ens.step(2)
        out = pinned(2 * n)
        out[:] = -1.0
        ens.get_state_ref(0, out[:n], out[n:])
        g = ens.get_state(0)
        assert np.array_equal(out[:n], g.real.ravel()) and np.array_equal(out[n:], g.imag.ravel())


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_energy_checks_every_coefficient(built_lib, prec):
    """Also the coefficients that no velocity field reads, and again after a failed call."""
    p = mwf.RunParams(K0=4, MM=9, NN=16, alpha=0.3, gamma=0.2, dt=0.01, precision=prec)
    good = mwf.ic.gaussian_ic(p, seed=2)
    with mwf.Ensemble([p]) as ens:
        ens.set_state(0, good)
        e = ens.energy(0)
        for at, v in (((0, 0, 0), np.nan), ((15, 16, 6), np.inf), ((3, 8, 4), -np.inf)):
            bad = good.copy()
            bad[at] = v
            ens.set_state(0, bad)
            with pytest.raises(mwf.MwfError):
                ens.energy(0)
        ens.set_state(0, good)
        assert ens.energy(0) == e
