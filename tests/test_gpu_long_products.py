"""FP64 ladder applications beyond 65535 of something that a kernel might put on a grid's y or z dimension. Tolerance of the
FP64 paths: 1e-10."""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid, synthetic

pytestmark = pytest.mark.gpu


def test_ladder_over_more_shifts_than_a_grid_dimension_holds_tiles(oracle):
    # the default path on a grid of two nodes, a gap of 2e6 of its units apart: K = 3 x 1.4e6 shifts in tiles of 64 terms
    from epspectral_gb300 import api
    g = FrequencyGrid(-1.0, 1e-6, np.array([0, 2_000_000]))
    s = synthetic.holstein_1d_setup(1, 1.0, 1.4, 0.2, g, omegas_spectral=FrequencyGrid(-1.0, 0.1, np.arange(21)))
    J = R.pseudorandom_complex(2, 4, 3, 2, 1, seed=0.41)
    args = (J, 0.1 * R.pseudorandom(2, 1, seed=7) - 0.1j, 0.05, 0.1, 0.07)
    ref = oracle.apply_ladder_kernel(s, *args, omega_acoustic=1e-3)
    got = api.apply_ladder_kernel(s, *args, omega_acoustic=1e-3, path="direct_fp64")
    assert np.abs(ref).max() > 0 and np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)


def test_ladder_over_more_modes_than_a_grid_dimension_holds(oracle):
    # the regrouped path with 2 x 32800 (mode, component) pairs
    from epspectral_gb300 import api
    g = FrequencyGrid(-1.0, 0.25, np.arange(9))
    s = synthetic.holstein_1d_setup(1, 1.0, 0.2, 0.2, g)
    nm = 32800
    s["omega_ph"] = np.asfortranarray(np.repeat(0.05 + 0.4 * np.abs(R.pseudorandom(nm, seed=4))[:, None], 1, axis=1))
    s["g2"] = np.asfortranarray(np.abs(R.pseudorandom(nm, 1, 1, seed=9)) / nm)
    J = R.pseudorandom_complex(9, 4, 3, 2, 1, seed=0.41)
    J[0] = J[-1] = 0
    args = (J, 0.1 * R.pseudorandom(9, 1, seed=7) - 0.1j, 0.05, 0.1, 0.07)
    ref = oracle.apply_ladder_kernel(s, *args, omega_acoustic=1e-3)
    got = api.apply_ladder_kernel(s, *args, omega_acoustic=1e-3, path="gemm_fp64")
    assert np.abs(ref).max() > 0 and np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)
