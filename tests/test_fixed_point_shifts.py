"""The rounding shift of the fixed-point passes (fx_down, mwf_fx.cuh) over all shifts, on the host."""
import os
import subprocess

import pytest

from mwf_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def half_even(x, r):
    """x / 2^r to the nearest integer, ties to even, in Python's integers."""
    q, rest = divmod(x, 1 << r)
    half = 1 << (r - 1)
    return q + (rest > half or (rest == half and q % 2 == 1))


@pytest.fixture(scope="module")
def fx_down(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fx") / "fx_shifts")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, os.path.join(ROOT, "tests", "cpp", "fx_shifts.cu"),
                    "-o", exe], check=True)

    def call(pairs):
        text = "".join(f"{x} {r}\n" for x, r in pairs)
        return [int(v) for v in subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()]
    return call


def test_rounds_to_nearest_even_for_every_shift(fx_down):
    """Any shift, as a direction of the coupling that is zero has an exponent of 2^20: zero stays zero and what lies
    below half a unit becomes zero, from above and from below."""
    values = [0, 1, -1, 2, -2, 3, -3, 5, -5, 6, -6, 2 ** 32 + 1, -2 ** 32 - 1, 2 ** 61, -2 ** 61, 2 ** 61 + 1, 2 ** 62 - 1, 1 - 2 ** 62,
              2 ** 62, -2 ** 62, 0x2aaaaaaaaaaaaaaa, -0x2aaaaaaaaaaaaaaa]
    shifts = list(range(1, 70)) + [100, 127, 128, 129, 1000, 1 << 20, 1 << 22]
    pairs = [(x, r) for r in shifts for x in values]
    want = [half_even(x, min(r, 200)) for x, r in pairs]
    assert fx_down(pairs) == want
