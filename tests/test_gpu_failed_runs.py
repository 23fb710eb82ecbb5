"""What a plan holds after a run that ends in an error: no Σ of it, on any path, and nothing that the next run sees."""
import ctypes as C

import numpy as np
import pytest

from epspectral_gb300 import FrequencyGrid, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["gemm_bf16", "gemm_fp64", "direct_fp64"])
def test_a_failed_run_leaves_no_sigma_behind(path):
    from epspectral_gb300 import api
    s = synthetic.holstein_1d_setup(16, 1.0, 0.2, 0.2, FrequencyGrid.from_nodes(np.arange(-100, 101) * 0.04))
    plan = api.Scgd0Plan(s, path=path, omega_acoustic=1e-6)
    occ = dict(Tlist=[0.1, 0.2], nlist=[0.0, 0.0], nelec=1.0, spin_degeneracy=2.0, type="metal")
    kw = dict(eta_init=0.05, tol=1e-6, maxiter=6, mu_start=[0.0, 0.0])
    ptr, nT = C.c_void_p(), C.c_int64()

    def sigma_device():
        return api.lib().epsp_scgd0_sigma_device(plan.handle, C.byref(ptr), C.byref(nT))

    assert sigma_device() != 0  # no run yet
    want = plan.run(occ, **kw)
    assert sigma_device() == 0 and nT.value == 2
    # a refused call leaves the last run's Σ where it is
    with pytest.raises(api.ArgumentError):
        plan.run(dict(occ, Tlist=[-0.1, 0.2]), **kw)
    assert sigma_device() == 0 and nT.value == 2
    # one that fails in its first iteration, the next one launched behind it, does not
    with pytest.raises(api.ArgumentError, match="no chemical potential"):
        plan.run(dict(occ, nlist=[0.0, 5.0]), **kw)
    assert sigma_device() != 0
    got = plan.run(occ, **kw)
    assert sigma_device() == 0
    assert np.array_equal(got["sigma"], want["sigma"]) and np.array_equal(got["mu"], want["mu"])
    plan.close()
