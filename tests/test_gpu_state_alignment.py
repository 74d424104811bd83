"""State arrays in pinned memory that are not 8-byte aligned (a packed record of a host program): copied, as
ordinary memory is, where aligned ones are accessed in place."""
import numpy as np
import pytest

import mwf_gb300 as mwf

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [4, 1, 8])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_unaligned_pinned_arrays(built_lib, prec, offset):
    p = mwf.RunParams(K0=4, MM=9, NN=16, alpha=0.3, gamma=0.2, dt=0.01, precision=prec)
    n = p.dof
    rng = np.random.default_rng(1)
    want = rng.standard_normal((2, n))
    raw = torch.zeros(2 * 8 * n + 16, dtype=torch.uint8, pin_memory=True).numpy()
    block = np.ndarray((2, n), np.float64, buffer=raw, offset=offset)
    block[:] = want
    kept = want if prec == "fp64" else want.astype(np.float32)
    with mwf.Ensemble([p]) as ens:
        ens.set_state_ref(0, block[0], block[1])
        assert np.array_equal(ens.get_state(0).ravel(), kept[0] + 1j * kept[1])
        block[:] = -1.0
        ens.get_state_ref(0, block[0], block[1])
        assert np.array_equal(block, kept)
        ens.set_history(0, (want[1] + 1j * want[0]).reshape(p.shape), False)
        h, euler = ens.get_history(0)
        assert not euler and np.array_equal(h.ravel(), kept[1] + 1j * kept[0])
