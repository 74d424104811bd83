"""The tuner's choice with the timings replaced by models of them (host only)."""
import pytest

import mwf_gb300 as mwf
from mwf_gb300 import autotune


def tuned_with(monkeypatch, passes, precision="fp64"):
    monkeypatch.setattr(autotune, "_time", lambda p, *a: passes(p))
    p = mwf.RunParams(K0=4, MM=48, NN=48, alpha=0.2, gamma=0.2, precision=precision)
    knobs = autotune.tune(p)
    return {n: knobs[n] for n in autotune.KNOBS}, sum(passes(p)), sum(passes(p.with_(**{n: knobs[n] for n in autotune.KNOBS})))


@pytest.mark.parametrize("best", ["xf_cols", "xi_cols", "z_lines", "x_radix"])
def test_a_knob_that_costs_the_other_passes_is_not_taken(monkeypatch, best):
    """Any knob moves all three passes to slower kernels, of which one pass happens to be faster at one setting."""
    def passes(p):
        if not any(getattr(p, n) for n in autotune.KNOBS):
            return [1.0, 1.0, 1.0]
        t = [2.0, 2.0, 2.0]
        if getattr(p, best) == 8:
            t[{"xf_cols": 0, "xi_cols": 2, "z_lines": 1, "x_radix": 0}[best]] = 0.5
        return t

    knobs, default, chosen = tuned_with(monkeypatch, passes)
    assert chosen <= default
    assert not any(knobs.values())


def test_knobs_that_help_are_taken(monkeypatch):
    def passes(p):
        return [0.9 if p.xf_cols == 2 else 1.0, 0.8 if p.z_lines == 1 else 1.0, 0.7 if p.xi_cols == 4 else 1.0]

    knobs, default, chosen = tuned_with(monkeypatch, passes)
    assert (knobs["xf_cols"], knobs["xi_cols"], knobs["z_lines"]) == (2, 4, 1) and chosen < default
