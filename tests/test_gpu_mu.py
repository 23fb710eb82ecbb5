"""The chemical potential of semiconductors on the GPU against the oracle: hole counts over a spectral window that reaches
far beyond exp's and FP32's ranges above μ, started at, near and far from the root.

Tolerance: on the FP64 paths the loop agrees to 1e-10 (its gate), on the tensor-core path Σ to 1e-5 eV; an error of that
size in the count moves its root by dμ/dn, which the oracle gives (the larger of it and 1).
"""
import numpy as np
import pytest

from epspectral_gb300 import FrequencyGrid, synthetic

pytestmark = pytest.mark.gpu

W_AC = 1e-6
GATE = {"direct_fp64": 1e-10, "gemm_fp64": 1e-10, "gemm_bf16": 1e-5}


@pytest.fixture(scope="module")
def api():
    from epspectral_gb300 import api as A
    A.lib()
    return A


def occ(nlist, T, nelec):
    return dict(Tlist=[T], nlist=[nlist], nelec=nelec, spin_degeneracy=2.0, type="semiconductor")


# ---- holes: nodes up to (4 - μ)/T above μ, 89 T (where 1 + exp leaves the FP32 range) and 709 T (exp's own) among them
@pytest.fixture(scope="module")
def chain():
    return synthetic.holstein_1d_setup(24, 0.4, 0.1, 0.2, FrequencyGrid.from_nodes(np.arange(-200, 201) * 0.02))


@pytest.mark.parametrize("kelvin,nlist", [(40, -0.3), (100, -1e-3), (100, -0.3), (300, -0.3), (900, -0.05)])
def test_hole_counts_match_oracle(api, oracle, chain, kelvin, nlist):
    T = kelvin * synthetic.KELVIN
    kw = dict(eta_init=0.1, tol=0.0, maxiter=1, omega_acoustic=W_AC)

    def mu(start, n=nlist):
        return oracle.loop_scgd0(chain, occ(n, T, 2.0), mu_start=[start], **kw)["mu"][0]

    root = mu(0.5)
    for start in (root, root - 3 * T, root + 3 * T, root - 40 * T, root + 40 * T, -3.0, 3.0):
        ref = mu(start)
        slope = max(1.0, abs(mu(start, nlist - 1e-6) - ref) / 1e-6)
        for path, gate in GATE.items():
            got = api.loop_scgd0(chain, occ(nlist, T, 2.0), path=path, mu_start=[start], **kw)["mu"][0]
            assert abs(got - ref) <= gate * slope, (path, start)


# ---- electrons: counts that only nodes far above μ hold, in a density of states with an edge (Σ without width outside it)
@pytest.mark.parametrize("count", [1e-6, 1e-12, 1e-18, 1e-24, 1e-30])
def test_small_electron_counts_match_oracle(api, oracle, chain, count):
    # the sum is all in nodes 14 to 69 T above μ; the first nodes above the edge hold most of it, so an error of it is one
    # of their Σ (1e-10 of its size; 1e-5 eV of width and energy) and moves the root by T times its relative size
    T = 100 * synthetic.KELVIN
    w, ni = chain["omegas"].nodes(), len(chain["eps_i"])
    S = np.zeros((len(w), ni, 1), dtype=np.complex128, order="F")
    S[np.abs(w) <= 1.2] = -0.1j
    kw = dict(eta_init=0.1, tol=0.0, maxiter=1, omega_acoustic=W_AC, sigma_init=S)
    root = oracle.loop_scgd0(chain, occ(count, T, 0.0), mu_start=[-2.0], **kw)["mu"][0]
    for start in (root, root - 3 * T, root + 3 * T, root - 40 * T, root + 40 * T, -3.9, 0.0):
        ref = oracle.loop_scgd0(chain, occ(count, T, 0.0), mu_start=[start], **kw)["mu"][0]
        for path, gate in GATE.items():
            got = api.loop_scgd0(chain, occ(count, T, 0.0), path=path, mu_start=[start], **kw)["mu"][0]
            assert abs(got - ref) <= gate, (path, start)
