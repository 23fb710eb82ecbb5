"""The term-by-term FP32 Fan-Migdal sum of the tensor-core plans (dispersive modes) against the oracle at the sizes and
temperatures where its kernels change: node tiles of 256, (ν, f) tiles of 256 and their splits, graded
grids, sides of μ, and temperatures where exp(ωq/T) leaves the factored kernel's range. The bound is the
one the path states, 1e-5 relative (FP32 terms; measured near 1e-6)."""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid
from test_oracle_scgd0 import per_pair_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,ni,nm,nf,T,mu", [
    (2, 1, 1, 1, 0.03, 0.07), (255, 2, 1, 255, 0.03, -2.0), (256, 3, 2, 128, 0.03, 2.0), (257, 5, 3, 86, 0.008, 0.07),
    (65, 3, 4, 1201, 7e-3, 0.0), (65, 3, 4, 1201, 6e-3, 0.0), (40, 3, 2, 9, 0.0, 0.07), (97, 33, 5, 101, 0.5, 0.3)])
@pytest.mark.parametrize("graded", [False, True])
def test_sum_matches_oracle(oracle, nw, ni, nm, nf, T, mu, graded):
    from epspectral_gb300 import api
    off = np.arange(nw) if not graded else np.cumsum(1 + 4 * (np.abs(np.arange(nw) - nw // 2) > nw // 4))
    g = FrequencyGrid(-1.0, 2.0 / (off[-1] - off[0]), off - off[0])
    wq = 0.05 + 0.2 * np.abs(R.pseudorandom(nm, ni, nf, seed=10))
    g2 = np.abs(R.pseudorandom(nm, ni, nf, seed=9))
    if ni > 2:
        wq[0, 1, :], g2[0, 1, :] = 0.0, np.inf  # below the acoustic cutoff: never read
    s = per_pair_setup(g, g2, wq, 0.8 * R.pseudorandom(nf, seed=11),
                       np.array([(5 * (f + 1)) % ni for f in range(nf)], dtype=np.int32), np.full(nf, 1.0 / nf))
    S = 0.1 * R.pseudorandom(nw, ni, seed=7) + 1j * (-0.05 - 0.05 * np.abs(R.pseudorandom(nw, ni, seed=8)))
    ref = oracle.imsigma(s, S, mu, T, np.zeros((nw, ni)), omega_acoustic=1e-3)
    plan = api.Scgd0Plan(s, path="gemm_bf16", omega_acoustic=1e-3)
    got = plan.imsigma(S, mu, T, np.zeros((nw, ni)))
    assert np.all(np.isfinite(got))
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
    assert np.array_equal(plan.imsigma(S, mu, T, np.zeros((nw, ni))), got)
    plan.close()


@pytest.mark.parametrize("off,unit,nm", [
    (np.arange(513), 0.004, 3),                                        # two nodes a thread, one over
    (np.cumsum(1 + 4 * (np.arange(700) % 3 == 0)) - 5, 0.002, 2),      # uneven cells
    (np.append(50 * np.arange(520), 50 * 519 + 1), 8e-5, 2),           # a table too long for shared memory
    (np.append(0, 40000 + 3 * np.arange(96)), 5e-5, 2),                # a cell too wide for it: the general sum
    (np.arange(60), 5e-6, 2), (np.arange(90) * 7, 3e-3, 3)])           # ωq of more units than it holds; a common divisor
def test_sum_on_uneven_grids(oracle, off, unit, nm):
    from epspectral_gb300 import api
    ni, nf, T, mu, nw = 3, 130, 0.03, 0.01, len(off)
    off = off - off[0]
    g = FrequencyGrid(-0.5 * unit * off[-1], unit, off)
    wq = 0.05 + 0.1 * np.abs(R.pseudorandom(nm, ni, nf, seed=10))
    wq[0, 0, 0], wq[1, 2, 5] = unit * 3, unit * 250  # whole numbers of units
    s = per_pair_setup(g, np.abs(R.pseudorandom(nm, ni, nf, seed=9)), wq, 0.4 * R.pseudorandom(nf, seed=11),
                       np.array([(5 * (f + 1)) % ni for f in range(nf)], dtype=np.int32), np.full(nf, 1.0 / nf))
    S = 0.1 * R.pseudorandom(nw, ni, seed=7) + 1j * (-0.05 - 0.05 * np.abs(R.pseudorandom(nw, ni, seed=8)))
    ref = oracle.imsigma(s, S, mu, T, np.zeros((nw, ni)), omega_acoustic=1e-5)
    plan = api.Scgd0Plan(s, path="gemm_bf16", omega_acoustic=1e-5)
    got = plan.imsigma(S, mu, T, np.zeros((nw, ni)))
    assert np.all(np.isfinite(got))
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
    plan.close()
