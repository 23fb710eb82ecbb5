"""The bounded waits of the FP64 products (csrc/oz_gemm.cu): a K block that never arrives ends the call with EPSP_EDEVICE_TIMEOUT,
from every entry point that forms such a product, and the next call is sound. The block is left out by a host-selected hook,
with a short limit on the waits: nothing faults or hangs.
"""
import time

import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid, abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from epspectral_gb300 import api as A
    A.lib()
    return A


def _times_out(api, ctx, kblock, call):
    ctx.stall_gemm(kblock, 4096)
    try:
        t0 = time.perf_counter()
        with pytest.raises(api.EpspError) as err:
            call()
        assert err.value.status == abi.EPSP_EDEVICE_TIMEOUT
        assert time.perf_counter() - t0 < 60
    finally:
        ctx.stall_gemm()


# K blocks of 64: the first, one in the middle of a chunk of four, and the last of K = 300 (5 blocks) or 155 (3)
@pytest.mark.parametrize("ni", [5, 65, 129, 257])  # tiles of 64, 128, 192 and 256 columns
@pytest.mark.parametrize("kblock", [0, 2, 4])
def test_scgd0_products_time_out_and_recover(api, ni, kblock):
    from test_gpu_fp64_products import _setup, _sigma
    s, S = _setup(300, ni, 5, 31), _sigma(300, ni)
    occ = dict(Tlist=[0.03], nlist=[0.0], nelec=1.0, spin_degeneracy=2.0, type="metal")
    kw = dict(eta_init=0.05, tol=0.0, maxiter=2, mu_start=[0.07], fix_mu=True, sigma_init=S[:, :, None])
    for path in ("gemm_fp64", "direct_fp64"):
        ctx = api.Context(0)
        plan = api.Scgd0Plan(s, path=path, omega_acoustic=1e-3, ctx=ctx)
        im, run = plan.imsigma(S, 0.07, 0.03, np.zeros(S.shape)), plan.run(occ, **kw)["sigma"]
        if path == "gemm_fp64" and kblock < 3:
            _times_out(api, ctx, kblock, lambda: plan.imsigma(S, 0.07, 0.03, np.zeros(S.shape)))
        _times_out(api, ctx, kblock, lambda: plan.run(occ, **kw))
        assert np.array_equal(plan.imsigma(S, 0.07, 0.03, np.zeros(S.shape)), im)
        assert np.array_equal(plan.run(occ, **kw)["sigma"], run)
        plan.close()


@pytest.mark.parametrize("path", ["direct_fp64", "gemm_fp64"])
def test_ladder_products_time_out_and_recover(api, path):
    s = synthetic.holstein_1d_setup(16, 1.0, 0.2, 0.2, FrequencyGrid.from_nodes(np.arange(-60, 61) * 0.05))
    nw, ni = 121, len(s["eps_i"])
    S = 0.1 * R.pseudorandom(nw, ni, seed=7) - 0.1j
    J = R.pseudorandom_complex(nw, 4, 3, 2, ni, seed=0.41)
    J[0] = J[-1] = 0
    ctx = api.Context(0)
    plan = api.LadderPlan(s, path=path, omega_acoustic=1e-3, ctx=ctx)
    args = (J, S, 0.05, 0.1, 0.07)
    run = lambda: plan.run(S[:, :, None], [0.05], [0.1], [0.07], rtol=1e-3, maxiter=10)  # noqa: E731
    L, sigma = plan.apply(*args), run()["sigma_ladder"]
    _times_out(api, ctx, 1, lambda: plan.apply(*args))
    _times_out(api, ctx, 1, run)
    assert np.array_equal(plan.apply(*args), L)
    assert np.array_equal(run()["sigma_ladder"], sigma)
    plan.close()
