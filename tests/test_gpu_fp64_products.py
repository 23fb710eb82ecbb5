"""The FP64 products on the tensor cores (csrc/oz_gemm.cu) at the sizes where they can go wrong, through
GEMM_FP64 plans against the oracle: tile edges in M = nω (128) and N = ni (64, 128, 192, 256), K = nm nf
around one chunk of 256 terms, above one 32-bit segment of 16128, and odd.

Tolerance: the Fan-Migdal sum has K terms of one sign, each formed by the same FP64 expressions on either
side. The oracle's own sum rounds K times (K 2^-53 relative at most, 2e-12 at K = 17000); a term's
difference (x - ε) - Re Σ(x) loses no more than the ratio of |x| <= 1.3 to |Im Σ| >= 0.05 (about 2^5 of its
2^-53 per rounding, a few roundings). 4e-12 covers both. The Kramers-Kronig map then sums nω terms of
either sign, |H| <= 3 against |Σ| ~ 0.1: 1e-11 of the norm.
"""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from epspectral_gb300 import api as A
    A.lib()
    return A


def _setup(nw, ni, nm, nf):
    g = FrequencyGrid(-1.0, 2.0 / (nw - 1), np.arange(nw))
    # (a chain of nf q points: iq_kk only has to be valid for dispersionless modes)
    return dict(g2=np.asfortranarray(np.abs(R.pseudorandom(nm, ni, nf, seed=9)) ** 4 * 10.0 ** (-4 * R.pseudorandom(nm, ni, nf, seed=3))),
                omega_ph=np.asfortranarray(np.repeat(0.05 + 0.2 * np.abs(R.pseudorandom(nm, seed=4))[:, None], 2, axis=1)),
                iq_kk=np.zeros((1, 1), dtype=np.int32, order="F"), iks_i=np.zeros(ni, np.int32), iks_f=np.zeros(nf, np.int32),
                eps_i=0.8 * R.pseudorandom(ni, seed=12), w_i=np.full(ni, 1.0 / ni), eps_f=0.8 * R.pseudorandom(nf, seed=11),
                w_f=np.full(nf, 1.0 / nf), f_to_i=np.array([(5 * (f + 1)) % ni for f in range(nf)], dtype=np.int32),
                W=1.0, nstates_base=0.0, multiplets=[], omegas=g, omegas_spectral=g)


def _sigma(nw, ni):
    return 0.1 * R.pseudorandom(nw, ni, seed=7) + 1j * (-0.05 - 0.05 * np.abs(R.pseudorandom(nw, ni, seed=8)))


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


SIZES = [(2, 1, 1, 1), (127, 33, 5, 51), (128, 64, 4, 64), (129, 65, 1, 257), (300, 128, 3, 7), (40, 193, 2, 40),
         (131, 256, 1, 11), (40, 257, 5, 13), (40, 3, 16, 1063)]


@pytest.mark.parametrize("nw,ni,nm,nf", SIZES)
def test_products_match_oracle(api, oracle, nw, ni, nm, nf):
    s, S = _setup(nw, ni, nm, nf), _sigma(nw, ni)
    ref = oracle.imsigma(s, S, 0.07, 0.03, np.full((nw, ni), 0.5), omega_acoustic=1e-3)
    plan = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3)
    got = plan.imsigma(S, 0.07, 0.03, np.full((nw, ni), 0.5))
    assert rel(got - 0.5, ref - 0.5) <= 4e-12
    assert np.array_equal(plan.imsigma(S, 0.07, 0.03, np.full((nw, ni), 0.5)), got)
    plan.close()
    # the Kramers-Kronig product, from the same Σ
    if nw > 2:
        occ = dict(Tlist=[0.03], nlist=[0.0], nelec=1.0, spin_degeneracy=2.0, type="metal")
        kw = dict(eta_init=0.05, tol=0.0, maxiter=1, mu_start=[0.07], fix_mu=True, sigma_init=S[:, :, None], omega_acoustic=1e-3)
        want = oracle.loop_scgd0(s, occ, **kw)
        have = api.loop_scgd0(s, occ, path="gemm_fp64", **kw)
        assert rel(have["sigma"], want["sigma"]) <= 1e-11


def test_not_finite_values_go_where_the_sums_take_them(api, oracle):
    # a NaN in one column's Σ reaches the nodes that read it, for every outer state, and nothing else
    nw, ni, nm, nf = 130, 5, 2, 9
    s, S = _setup(nw, ni, nm, nf), _sigma(nw, ni)
    S[17, 0] = np.nan  # (every inner state of this size has representative 0)
    ref = oracle.imsigma(s, S, 0.07, 0.03, np.zeros((nw, ni)), omega_acoustic=1e-3)
    plan = api.Scgd0Plan(s, path="gemm_fp64", omega_acoustic=1e-3)
    got = plan.imsigma(S, 0.07, 0.03, np.zeros((nw, ni)))
    plan.close()
    assert np.isnan(ref).any() and not np.isnan(ref).all()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    fin = ~np.isnan(ref)
    assert rel(got[fin], ref[fin]) <= 4e-12


# ---- the term-by-term FP64 sum (DIRECT_FP64) ----
# The same terms as the oracle's, to a few roundings each (2^-53 of |x| <= 1.3 against |z| >= 0.05: 3e-15), all of one
# sign: the sum's own gate of 1e-13 (the Fan-Migdal test of the reference's kernel) holds at every size.
@pytest.mark.parametrize("nw,ni,nm,nf,T,mu", [
    (2, 1, 1, 1, 0.03, 0.07), (33, 2, 1, 31, 0.03, -2.0), (127, 3, 2, 16, 0.03, 2.0), (129, 5, 3, 11, 0.003, 0.07),
    (65, 7, 4, 75, 8.4e-4, 0.0), (65, 7, 4, 75, 5e-4, 0.0), (40, 3, 2, 9, 0.0, 0.07), (97, 33, 5, 101, 0.5, 0.3)])
@pytest.mark.parametrize("graded", [False, True])
def test_direct_sum_matches_oracle(api, oracle, nw, ni, nm, nf, T, mu, graded):
    from test_oracle_scgd0 import per_pair_setup
    off = np.arange(nw) if not graded else np.cumsum(1 + 4 * (np.abs(np.arange(nw) - nw // 2) > nw // 4))
    g = FrequencyGrid(-1.0, 2.0 / (off[-1] - off[0]), off - off[0])
    wq = 0.05 + 0.2 * np.abs(R.pseudorandom(nm, ni, nf, seed=10))
    g2 = np.abs(R.pseudorandom(nm, ni, nf, seed=9))
    if ni > 2:
        wq[0, 1, :], g2[0, 1, :] = 0.0, np.inf  # below the acoustic cutoff: never read
    s = per_pair_setup(g, g2, wq, 0.8 * R.pseudorandom(nf, seed=11),
                       np.array([(5 * (f + 1)) % ni for f in range(nf)], dtype=np.int32), np.full(nf, 1.0 / nf))
    S = _sigma(nw, ni)
    ref = oracle.imsigma(s, S, mu, T, np.zeros((nw, ni)), omega_acoustic=1e-3)
    for tile in (None, 7):
        plan = api.Scgd0Plan(s, path="direct_fp64", omega_acoustic=1e-3, gpu_tile=tile)
        got = plan.imsigma(S, mu, T, np.zeros((nw, ni)))
        assert np.all(np.isfinite(got)) and rel(got, ref) <= 1e-13
        assert np.array_equal(plan.imsigma(S, mu, T, np.zeros((nw, ni))), got)
        plan.close()


# ---- the spectral functions (FP64 paths) ----
# The smallest ∫A over the states, where |z|² is ordinary and, for one state, at the ends of the range (0 to rounding):
# a few roundings a node, the sums' terms of one sign, so 1e-13 relative holds.
@pytest.mark.parametrize("shift", [0.0, 3.0, 1e30, 1e100, 1e140, 1e154, 1e170])
def test_spectral_weight_matches_oracle(api, oracle, shift):
    nw, ni, nm, nf = 65, 3, 2, 9
    s, S = _setup(nw, ni, nm, nf), _sigma(nw, ni)
    s["eps_i"] = np.array(s["eps_i"], dtype=np.float64)
    s["eps_i"][1] += shift
    occ = dict(Tlist=[0.03], nlist=[0.0], nelec=1.0, spin_degeneracy=2.0, type="metal")
    kw = dict(eta_init=0.05, tol=0.0, maxiter=1, mu_start=[0.07], fix_mu=True, sigma_init=S[:, :, None], omega_acoustic=1e-3)
    want = oracle.loop_scgd0(s, occ, **kw)["history"]["min_spectral_weight"]
    have = api.loop_scgd0(s, occ, path="gemm_fp64", **kw)["history"]["min_spectral_weight"]
    assert np.all(np.isfinite(have)) and np.allclose(have, want, rtol=1e-13, atol=1e-300)
