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


def test_solutions_of_more_vectors_than_one_pass_combines():
    # Four solves of 6 to 14 Krylov vectors (a pass sums eight): batched, each pair's vertex is formed from its own
    # count of vectors and must equal the sequential solve's (warm-started: its sum adds to a vertex) to 1e-4, as both
    # residuals are 1e-6.
    from epspectral_gb300 import api, graded_frequency_grid
    ws = graded_frequency_grid([(-0.3, 0.3, 0.01), (-0.9, 0.9, 0.1)])
    s = synthetic.cubic_t2g_setup(N=4, ws=ws, g2_dtype=np.float64, seed=3)
    s["g2"] = 0.1 * s["g2"]
    sig = np.empty((len(ws), s["eps_i"].size, 2), dtype=complex, order="F")
    sig[:, :, 0], sig[:, :, 1] = 0.001 - 0.02j, -0.002 - 0.05j
    plan = api.LadderPlan(s, path="gemm_bf16", omega_acoustic=W_AC)
    args = (sig, [0.0, 0.01], [0.02, 0.05], [0.0, 0.1])
    kw = dict(rtol=1e-6, maxiter=40, store_vertex=True)
    seq, bat = plan.run(*args, **kw), plan.run(*args, batch_rhs=4, **kw)
    assert seq["converged"].all() and bat["converged"].all()
    assert bat["niter"].max() > 8 > bat["niter"].min() and seq["niter"].max() > 8
    for iT in range(2):
        for iO in range(2):
            a, b = bat["J"][..., iO, iT], seq["J"][..., iO, iT]
            assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), (iO, iT)
    plan.close()
