"""The FP64 products (csrc/oz_gemm.cu) element by element where rows and columns are widely scaled: resonances 1e-6 wide in the
kernel tensor (elements from 1e6 down to 1e-7 in a row) against couplings over 16 decades, so that an element of the product may
be far below its row's and its column's largest terms.

Tolerance: the products' own bound, K 2^-60 times the largest of the row and of the column (the operands' 62-bit fixed point
and the orders left out); and, of the element, 4e-12 for its terms and the oracle's K roundings (as in test_gpu_fp64_products)
and for a resonance's distance, |x| <= 1.3 rounded to 2^-53 against a width of 1e-6: 2e-10.
"""
import numpy as np
import pytest

import refimpl as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,ni,nm,nf", [(129, 65, 2, 48), (40, 193, 3, 40)])
def test_small_elements_of_widely_scaled_products(oracle, nw, ni, nm, nf):
    from epspectral_gb300 import api
    from test_gpu_fp64_products import _setup
    s = _setup(nw, ni, nm, nf)
    s["g2"] = np.asfortranarray(10.0 ** (8 * R.pseudorandom(nm, ni, nf, seed=9)))
    S = np.asfortranarray(0.1 * R.pseudorandom(nw, ni, seed=7) - 1e-6j)
    T, mu, w, wq = 0.03, 0.07, s["omegas"].nodes(), s["omega_ph"][:, 0]
    zero = np.zeros((nw, ni))
    ref = oracle.imsigma(s, S, mu, T, zero, omega_acoustic=1e-3)
    plan = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3)
    got = plan.imsigma(S, mu, T, zero)
    plan.close()
    # the largest of each row of the kernel tensor and of each column of the couplings
    row, col = np.zeros(nw), np.abs(s["g2"]).max(axis=(0, 2)) * s["w_f"].max()
    for nu in range(nm):
        for f in range(nf):
            Sf, k = S[:, s["f_to_i"][f]], 0.0
            for sg in (1, -1):
                x = w + sg * wq[nu]
                z = x - s["eps_f"][f] - np.interp(x, w, Sf.real) + 1e-6j
                n = 1 / np.expm1(wq[nu] / T) + (1 / (np.exp((x - mu) / T) + 1) if sg > 0 else 1 / (np.exp((mu - x) / T) + 1))
                k = k - (1 / z).imag * n
            row = np.maximum(row, np.abs(k))
    K = nm * nf
    bound = K * 2.0 ** -60 * row[:, None] * col[None, :] + 2e-10 * np.abs(ref)
    assert np.abs(ref).min() < 1e-6 * (row[:, None] * col[None, :]).max()
    assert np.all(np.abs(got - ref) <= bound)
