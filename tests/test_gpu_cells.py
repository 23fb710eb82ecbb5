"""The kernel tensor of the tensor-core path (csrc/scgd0_tc.cu) where Σ(ω ± ω_ν) lies far inside wide cells of the grid and
a pole lies within its width of the point: Re z = (x - ε) - Re Σ(x) has to keep the distance to the pole.

Tolerance: Re z comes from float pairs but for the step along the cell times Σ's slope, rounded to 2^-25 of 0.25 x 0.01 eV:
7e-11 eV, which against the width of 2e-4 eV moves an element by 4e-7 at most; half a dozen FP32 roundings an element and the
three-part products add 6e-7. (The step itself rounded to FP32, 2^-27 x 0.25 eV, moves elements by up to 4e-5.)
"""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nf,wq", [(31, 31, 0.13), (32, 64, 0.2371), (5, 96, 0.0613)])
def test_sharp_poles_in_wide_cells_match_oracle(oracle, ni, nf, wq):
    from epspectral_gb300 import api
    from test_gpu_fp64_products import _setup
    nw, eta = 33, 2e-4
    g = FrequencyGrid(-4.0, 0.25, np.arange(nw))
    w = g.nodes()
    s = dict(_setup(nw, ni, 1, nf), omegas=g, omegas_spectral=g, omega_ph=np.full((1, 2), wq, order="F"))
    s["g2"] = np.asfortranarray(1.0 + np.abs(R.pseudorandom(1, ni, nf, seed=9)))
    S = np.empty((nw, ni), dtype=np.complex128, order="F")
    S.real = 0.1 * R.pseudorandom(ni, seed=7)[None, :] + 0.01 * w[:, None]
    S.imag = -eta
    # inner state f's pole: within its width of ω_j + ω_ν (j = f mod nω), where it takes Σ of its representative
    j, rep = np.arange(nf) % nw, s["f_to_i"]
    s["eps_f"] = w[j] + wq - (S.real[j, rep] + 0.01 * wq) + 2 * eta * R.pseudorandom(nf, seed=11)
    ref = oracle.imsigma(s, S, 0.07, 0.03, np.zeros((nw, ni)), omega_acoustic=1e-3)
    plan = api.Scgd0Plan(s, path="gemm_bf16", omega_acoustic=1e-3)
    got = plan.imsigma(S, 0.07, 0.03, np.zeros((nw, ni)))
    plan.close()
    assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)
