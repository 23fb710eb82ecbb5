"""A launch that CUDA refuses on the host (a grid dimension beyond its limit, before anything runs) is reported by the call
that made it and by no later one."""
import numpy as np
import pytest

import refimpl as R

pytestmark = pytest.mark.gpu


def test_a_refused_launch_is_reported_once():
    from epspectral_gb300 import api
    from test_gpu_fp64_products import _setup, _sigma
    small, S = _setup(9, 3, 2, 5), _sigma(9, 3)
    zero = np.zeros((9, 3))
    good = api.Scgd0Plan(small, path="gemm_fp64", omega_acoustic=1e-3)
    want = good.imsigma(S, 0.07, 0.03, zero)
    # modes x inner states = 66000 blocks on the y dimension of the kernel tensor's grid
    big = api.Scgd0Plan(_setup(3, 1, 1000, 66), path="gemm_fp64", omega_acoustic=1e-3)
    with pytest.raises(api.EpspError, match="ECUDA"):
        big.imsigma(_sigma(3, 1), 0.07, 0.03, np.zeros((3, 1)))
    assert np.array_equal(good.imsigma(S, 0.07, 0.03, zero), want)
    api.Scgd0Plan(small, path="gemm_fp64", omega_acoustic=1e-3).close()
    big.close()
    good.close()
