"""The Fan-Migdal sums of the tensor-core path (csrc/scgd0_tc.cu: the kernel tensor, and term by term for dispersive modes)
where Σ(ω ± ω_ν) lies far inside wide cells of the grid and a pole lies within its width of the point: Re z =
(x - ε) - Re Σ(x) has to keep the distance to the pole.

Tolerance: Re z comes from float pairs but for the step along the cell times Σ's slope, rounded to 2^-25 of 0.25 x 0.01 eV:
7e-11 eV, which against the width of 2e-4 eV moves an element by 4e-7 at most; half a dozen FP32 roundings an element and the
three-part products add 6e-7. (The step itself rounded to FP32, 2^-27 x 0.25 eV, moves elements by up to 4e-5.)
"""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid

pytestmark = pytest.mark.gpu


def _setup_with_poles(ni, nf, wq, off, unit, dispersive):
    """Inner state f's pole lies within its width of ω_j + ω_ν (j = f mod nω), where it takes Σ of its representative."""
    from test_gpu_fp64_products import _setup
    eta, g = 2e-4, FrequencyGrid(-4.0, unit, off)
    w, nw = g.nodes(), len(off)
    wph = np.full((1, 2), wq, order="F")
    if dispersive:
        wph[0, 1] = 0.9 * wq  # (every pair reads the first)
    s = dict(_setup(nw, ni, 1, nf), omegas=g, omegas_spectral=g, omega_ph=wph)
    s["g2"] = np.asfortranarray(1.0 + np.abs(R.pseudorandom(1, ni, nf, seed=9)))
    S = np.empty((nw, ni), dtype=np.complex128, order="F")
    S.real = 0.1 * R.pseudorandom(ni, seed=7)[None, :] + 0.01 * w[:, None]
    S.imag = -eta
    j, rep = np.arange(nf) % nw, s["f_to_i"]
    s["eps_f"] = w[j] + wq - (S.real[j, rep] + 0.01 * wq) + 2 * eta * R.pseudorandom(nf, seed=11)
    return s, S


UNIFORM = (np.arange(33), 0.25)
GRADED = (np.concatenate([np.arange(0, 65, 5), np.arange(65, 95), np.arange(95, 161, 5)]), 0.05)


@pytest.mark.parametrize("dispersive", [False, True])
@pytest.mark.parametrize("off,unit", [UNIFORM, GRADED])
@pytest.mark.parametrize("ni,nf,wq", [(31, 31, 0.13), (32, 64, 0.2371), (5, 96, 0.0613)])
def test_sharp_poles_in_wide_cells_match_oracle(oracle, ni, nf, wq, off, unit, dispersive):
    from epspectral_gb300 import api
    s, S = _setup_with_poles(ni, nf, wq, off, unit, dispersive)
    zero = np.zeros(S.shape)
    ref = oracle.imsigma(s, S, 0.07, 0.03, zero, omega_acoustic=1e-3)
    plan = api.Scgd0Plan(s, path="gemm_bf16", omega_acoustic=1e-3)
    got = plan.imsigma(S, 0.07, 0.03, zero)
    plan.close()
    assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("dispersive", [False, True])
@pytest.mark.parametrize("unit,steps", [(0.1, 3), (0.07, 2), (0.013, 7)])
def test_points_that_round_onto_nodes_take_the_nodes_values(oracle, unit, steps, dispersive):
    # ω_ν a multiple of the step: ω ± ω_ν are nodes but for their rounding, to either side. Σ is 0.1 eV wide at the even
    # nodes and 1e-5 at the odd ones, where the poles are: an element there is the node's value to 2^-24 (2^-24 of 0.1 eV
    # would be 6e-4 of it), the sums as above.
    from epspectral_gb300 import api
    from test_gpu_fp64_products import _setup
    nw, ni, nf = 41, 7, 40
    g = FrequencyGrid(-20 * unit, unit, np.arange(nw))
    w, wq = g.nodes(), steps * unit
    x = np.concatenate([w + wq, w - wq])
    j = np.rint((x - w[0]) / unit).astype(int)
    on = (j > 0) & (j < nw - 1)
    assert np.any(x[on] < w[j[on]]) and np.any(x[on] > w[j[on]])  # both roundings are there
    wph = np.full((1, 2), wq, order="F")
    if dispersive:
        wph[0, 1] = 0.9 * wq  # (every pair reads the first)
    s = dict(_setup(nw, ni, 1, nf), omegas=g, omegas_spectral=g, omega_ph=wph)
    s["g2"] = np.asfortranarray(1.0 + np.abs(R.pseudorandom(1, ni, nf, seed=9)))
    S = np.empty((nw, ni), dtype=np.complex128, order="F")
    S.real = 0.1 * R.pseudorandom(nw, ni, seed=7)
    S.imag = np.where(np.arange(nw) % 2 == 0, -0.1, -1e-5)[:, None]
    at = 2 * (np.arange(nf) % (nw // 2)) + 1
    s["eps_f"] = w[at] - S.real[at, s["f_to_i"]] + 2e-5 * R.pseudorandom(nf, seed=11)
    zero = np.zeros(S.shape)
    ref = oracle.imsigma(s, S, 0.07, 0.3, zero, omega_acoustic=1e-4)
    plan = api.Scgd0Plan(s, path="gemm_bf16", omega_acoustic=1e-4)
    got = plan.imsigma(S, 0.07, 0.3, zero)
    plan.close()
    assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)
