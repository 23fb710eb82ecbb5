"""The gather of the ladder's contracted vertex (tensor-core paths) against the oracle at the sizes where its launch
changes: ranges of 256 nodes and their remainders, columns left over from groups of four, split-K partials, and the
grids fine enough for their modes that a block stages two columns or one. The bounds are the ones that the paths
state: 1e-4 (BF16x3) and 1e-3 (TF32) relative."""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid, synthetic

pytestmark = pytest.mark.gpu

W_AC = 1e-3


@pytest.mark.parametrize("nw,unit,modes", [(2, 0.05, 3), (64, 0.01, 15), (255, 0.01, 4), (256, 0.01, 3), (257, 0.005, 15),
                                           (513, 0.002, 4), (1537, 0.0002, 3), (2049, 0.0001, 3)])
def test_apply_matches_oracle(oracle, nw, unit, modes):
    from epspectral_gb300 import api
    ws = FrequencyGrid(-unit * (nw // 2), unit, np.arange(nw))
    s = synthetic.cubic_t2g_setup(N=3, nmodes=modes, ws=ws, g2_dtype=np.float64, seed=5)
    ni = s["eps_i"].size
    sig = np.asfortranarray(np.full((nw, ni), complex(0.001, -0.02)))
    J = R.pseudorandom_complex(nw, 4, 3, 2, ni, seed=1.3)
    J[0] = 0
    J[-1] = 0
    T = 300 * synthetic.KELVIN
    ref = oracle.apply_ladder_kernel(s, J, sig, 0.0, T, 0.05, omega_acoustic=W_AC)
    for path, tol, bk in (("gemm_bf16", 1e-4, 64), ("gemm_tf32", 1e-3, 32)):
        plan = api.LadderPlan(s, path=path, omega_acoustic=W_AC)
        for splits in (1, 2):
            plan.set_gemm_config(128, splits, bk)
            got = plan.apply(J, sig, 0.0, T, 0.05)
            assert np.all(np.isfinite(got))
            assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref), (path, splits)
        plan.close()
