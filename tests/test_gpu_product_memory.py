"""The FP64 products (csrc/oz_gemm.cu) where the device has little room: in panels of rows and columns, without kept
planes of the operands that do not change, and with those given back to another plan's allocation. Each element is its own
exact sum, so everything but the last resort (plain FP64 sums) is bitwise the same.
"""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid, synthetic

pytestmark = pytest.mark.gpu

OCC = dict(Tlist=[0.03], nlist=[0.0], nelec=1.0, spin_degeneracy=2.0, type="metal")
RUN = dict(eta_init=0.05, tol=0.0, maxiter=2, mu_start=[0.07], fix_mu=True)


@pytest.fixture(scope="module")
def api():
    from epspectral_gb300 import api as A
    A.lib()
    return A


@pytest.fixture(scope="module")
def model():
    from test_gpu_fp64_products import _setup, _sigma
    return _setup(300, 257, 5, 31), _sigma(300, 257)


def _outputs(plan, S):
    """The Fan-Migdal product (a kept B, a split A, added to 0.5) and the Kramers-Kronig one (a kept A, a split B)."""
    return plan.imsigma(S, 0.07, 0.03, np.full(S.shape, 0.5)), plan.run(OCC, sigma_init=S[:, :, None], **RUN)["sigma"]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def _planes_bytes(s):
    return 16 * len(s["eps_i"]) * (-(-s["g2"].shape[0] * s["g2"].shape[2] // 64) * 64)


def test_panels_do_not_change_an_element(api, model):
    s, S = model
    ctx = api.Context(0)
    plan = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3, ctx=ctx)
    want = _outputs(plan, S)
    ctx.product_panels(1 << 20)  # panels of 128 rows (300 = 2 x 128 + 44), of 192 columns (257 = 192 + 65)
    assert _same(_outputs(plan, S), want)
    ctx.product_panels(1)  # plain sums: K = 155 and 300 terms, of one sign and of either
    for x, y in zip(_outputs(plan, S), want):
        assert np.linalg.norm(x - y) <= 1e-13 * np.linalg.norm(y)
    ctx.product_panels()
    assert _same(_outputs(plan, S), want)
    plan.close()


def test_a_plan_fits_where_its_planes_do_not(api, model):
    s, S = model
    ctx = api.Context(0)
    kept = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3, ctx=ctx)
    want = _outputs(kept, S)
    kept.close()
    ctx.fail_next_alloc(_planes_bytes(s))  # the largest allocation of the set-up: those planes
    plan = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3, ctx=ctx)
    assert _same(_outputs(plan, S), want)
    ctx.product_panels(1 << 20)  # B in panels of columns for each panel of rows
    assert _same(_outputs(plan, S), want)
    plan.close()


def test_planes_and_work_buffers_make_room_for_another_plan(api, model):
    s, S = model
    ctx = api.Context(0)
    first = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3, ctx=ctx)
    want = _outputs(first, S)
    ctx.fail_next_alloc(1)
    second = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3, ctx=ctx)
    assert _same(_outputs(second, S), want)
    assert _same(_outputs(first, S), want)  # without its planes
    ctx.fail_next_alloc(4 * 9 * 128 * 257)  # its work buffers come back
    second.close()
    assert _same(_outputs(first, S), want)
    first.close()


@pytest.mark.parametrize("path", ["direct_fp64", "gemm_fp64"])
def test_ladder_in_panels_and_without_planes(api, path):
    s = synthetic.holstein_1d_setup(48, 1.0, 0.2, 0.2, FrequencyGrid.from_nodes(np.arange(-60, 61) * 0.05))
    nw, ni = 121, len(s["eps_i"])
    J = R.pseudorandom_complex(nw, 4, 3, 2, ni, seed=0.41)
    J[0] = J[-1] = 0
    args = (J, 0.1 * R.pseudorandom(nw, ni, seed=7) - 0.1j, 0.05, 0.1, 0.07)
    ctx = api.Context(0)
    plan = api.LadderPlan(s, path=path, omega_acoustic=1e-3, ctx=ctx)
    want = plan.apply(*args)
    ctx.product_panels(1 << 20)
    assert np.array_equal(plan.apply(*args), want)
    ctx.product_panels()
    ctx.fail_next_alloc(1)
    api.LadderPlan(s, path=path, omega_acoustic=1e-3, ctx=ctx).close()  # takes this one's planes
    assert np.array_equal(plan.apply(*args), want)
    plan.close()
