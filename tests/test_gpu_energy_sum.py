"""The energy's sum over the blocks' partial sums is compensated: small terms beside one large one count."""
import numpy as np
import pytest

import mwf_gb300 as mwf

pytestmark = pytest.mark.gpu

THREADS, BLOCKS = 64, 2432            # of the energy kernel on a state this large


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_small_partials_are_not_lost(built_lib, prec):
    """One coefficient in (nearly) every block's points, all terms of the energy exact powers of two times
    integers: one of 2^73 to 2^75 and some 2400 below half its last bit, 2^20, each.  A plain running sum drops those
    that follow the large one (4.9 units in the last place here); a compensated one rounds at the end."""
    p = mwf.RunParams(K0=4, MM=256, NN=324, alpha=1.0, gamma=1.0, precision=prec)
    c = np.zeros(p.shape, complex)
    exact = 0                                             # in units of 2^-20
    for b in range(BLOCKS):
        n, ms = divmod(THREADS * b, p.M)
        if n == 0:
            continue
        m = ms if ms < p.MM else ms - p.M
        h = 2 * (n * n + m * m)                           # the energy of psi_0 = 1
        if b == 16:
            e = 73 - h.bit_length() + 1                   # h 2^e in [2^73, 2^75)
            e += e % 2
        else:
            e = 20 - h.bit_length()                       # h 2^e in [2^18, 2^20)
            e -= e % 2
        c[n, ms, 0] = 2.0 ** (e // 2)
        exact += h * 2 ** (e + 20)
    with mwf.Ensemble([p]) as ens:
        ens.set_state(0, c)
        got = ens.energy(0)
    err = abs(int(np.ldexp(got, 20)) - exact) / 2 ** 20
    assert err <= np.spacing(got), err / np.spacing(got)
