"""The nonlinear term of the fixed-point FP64 passes against extended-precision arithmetic, measured by the
error of the FP64-arithmetic kernels, which any tuning knob selects."""
import numpy as np
import pytest

import mwf_gb300 as mwf

sf = pytest.importorskip("scipy.fft")
pytestmark = pytest.mark.gpu

REAL, CPLX = np.longdouble, np.clongdouble


def nonlinear_term(p, c):
    """The projected nonlinear term of state c in long double: velocities and gradients on the dealiased grid, the
    products on eight points in y (exact for these wall-normal modes), and back."""
    K0, M, MM, NN, X, Z = p.K0, p.M, p.MM, p.NN, p.X, p.Z
    ms = np.arange(M)
    m = np.where(ms < MM, ms, ms - M)
    m1, n1 = REAL(p.alpha) * m[None, :], REAL(p.gamma) * np.arange(NN)[:, None]
    h = m1 ** 2 + n1 ** 2
    beta = 2 * np.arctan(REAL(1))                          # pi/2
    kap = [(-k if k % 2 else k) * beta for k in range(K0)]
    c = c.astype(CPLX)
    i = CPLX(1j)
    psi = [c[..., k] for k in range(K0)]
    phi = [0 * c[..., 0]] + [c[..., K0 + k] for k in range(K0 - 1)]
    u = [-i * n1 * psi[k] + i * kap[k] * m1 * phi[k] for k in range(K0)]
    w = [i * m1 * psi[k] + i * kap[k] * n1 * phi[k] for k in range(K0)]
    v = [h * phi[k] for k in range(1, K0)]
    for k in range(K0):
        u[k][0, 0], w[k][0, 0] = psi[k][0, 0], phi[k][0, 0]
    u[0][0, 0] = 0
    u[1][0, 0] += REAL(np.cos(p.theta))
    w[1][0, 0] += REAL(np.sin(p.theta))

    def physical(s):
        a = np.zeros((NN, X), CPLX)
        a[:, m % X] = s
        t = sf.ifft(a, axis=1, norm="forward")
        t[0] = t[0].real
        b = np.zeros((Z // 2 + 1, X), CPLX)
        b[:NN] = t
        return sf.irfft(b, n=Z, axis=0, norm="forward")

    s = u + v + w
    F, Fx, Fz = ([physical(f * q) for q in s] for f in (REAL(1), i * m1, i * n1))
    y = (np.arange(8).astype(REAL) + REAL(0.5)) / 4 - 1
    k = np.arange(K0)
    ky = k[:, None] * beta
    odd = (k % 2 == 1)[:, None]
    sn, cs = np.sin(ky * y), np.cos(ky * y)
    Eu, dEu = np.where(odd, sn, cs), np.where(odd, ky * cs, -ky * sn)
    Ev, dEv = np.where(odd, cs, sn)[1:], np.where(odd, -ky * sn, ky * cs)[1:]
    parts = [(range(0, K0), Eu, dEu), (range(K0, 2 * K0 - 1), Ev, dEv), (range(2 * K0 - 1, 3 * K0 - 1), Eu, dEu)]
    acc = [0] * (3 * K0 - 1)
    for iy in range(8):
        def at(A, part, E):
            return sum(A[f] * E[j, iy] for j, f in enumerate(part))
        U, V, W = (at(F, r, E) for r, E, _ in parts)
        for r, E, dE in parts:
            N = U * at(Fx, r, E) + V * at(F, r, dE) + W * at(Fz, r, E)
            for j, f in enumerate(r):
                acc[f] = acc[f] + N * E[j, iy] / 4
    out = []
    for f in range(3 * K0 - 1):
        a = acc[f] / (REAL(X) * Z) * (REAL(0.5) if f in (0, 2 * K0 - 1) else 1)
        out.append(sf.fft(sf.rfft(a, axis=0)[:NN], axis=1)[:, m % X])
    uu, vv, ww = out[:K0], [0 * out[0]] + out[K0:2 * K0 - 1], out[2 * K0 - 1:]
    ps = [i * (n1 * uu[q] - m1 * ww[q]) for q in range(K0)]
    ph = [i * kap[q] * (m1 * uu[q] + n1 * ww[q]) - h * vv[q] for q in range(K0)]
    for q in range(K0):
        ps[q][0, 0], ph[q][0, 0] = -uu[q][0, 0], -ww[q][0, 0]
    ps[0][0, 0] = 0
    return np.stack(ps + ph[1:], -1)


def state(p, kind):
    c = mwf.ic.gaussian_ic(p, seed=1)
    if kind == "gauss":
        return c
    rng = np.random.default_rng(2)
    w = rng.standard_normal(p.shape) + 1j * rng.standard_normal(p.shape)
    if kind == "falling":                     # in k = (m, n) as 1 / (1 + k^2 / 20), in the wall-normal mode by 10 a mode
        m = np.minimum(np.arange(p.M), p.M - np.arange(p.M))
        w /= (1 + 0.05 * (np.arange(p.NN)[:, None] ** 2 + m[None, :] ** 2))[:, :, None]
        w *= 0.1 ** np.concatenate([np.arange(p.K0), np.arange(1, p.K0)])
    w[0] = 0.0
    return w + c * (np.arange(p.NN) == 0)[:, None, None] * (0.1 ** np.concatenate([np.arange(p.K0), np.arange(1, p.K0)]) if kind == "falling" else 1.0)


def norm(a):
    return float(np.sqrt((np.abs(a) ** 2).sum()))


@pytest.mark.skipif(np.finfo(REAL).eps > 2e-19, reason="long double is not wider than double")
@pytest.mark.parametrize("kind", ["gauss", "white", "falling"])
@pytest.mark.parametrize("K0,MM,NN", [(4, 32, 48), (6, 24, 32), (6, 8, 512), (4, 4, 768)])
def test_no_further_off_than_fp64_arithmetic(built_lib, K0, MM, NN, kind):
    """One Euler step leaves the nonlinear term as the history.  Both paths round thousands of values a
    coefficient, so that the norms of their errors are sharp to a few per cent: the whole term may be no further off than
    with FP64 arithmetic (1.05 of it), and with wall-normal modes of like size no mode more than 4 times.  (The coupling
    holds its operands to 2^-59 of the largest value of a component, FP64 to 2^-54 of themselves: of modes that fall
    by 10 from one to the next the last has the coarser operands, and no bound of that kind.)"""
    p = mwf.RunParams(K0=K0, MM=MM, NN=NN, alpha=3.0 / MM, gamma=3.0 / NN, dt=0.01, theta=0.3)
    c0 = state(p, kind)
    want = nonlinear_term(p, c0)
    err = []
    for q in (p, p.with_(x_radix=12)):
        with mwf.Ensemble([q]) as ens:
            ens.set_state(0, c0)
            ens.step(1)
            err.append(ens.get_history(0)[0].astype(CPLX) - want)
    here, fp64 = err
    assert norm(here) <= 1.05 * norm(fp64), norm(here) / norm(fp64)
    if kind != "falling":
        modes = [norm(here[..., k]) / norm(fp64[..., k]) for k in range(p.K)]
        assert max(modes) <= 4.0, modes
