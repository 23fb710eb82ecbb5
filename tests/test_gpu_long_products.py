"""A product longer than a grid's y dimension of 64-term tiles (K = 3 x 1.4e6 shifts): one ladder application through the
default path on a grid of two nodes, a gap of 2e6 of its units apart. Tolerance of the FP64 paths: 1e-10."""
import numpy as np
import pytest

import refimpl as R
from epspectral_gb300 import FrequencyGrid, synthetic

pytestmark = pytest.mark.gpu


def test_ladder_over_more_shifts_than_a_grid_dimension_holds_tiles(oracle):
    from epspectral_gb300 import api
    g = FrequencyGrid(-1.0, 1e-6, np.array([0, 2_000_000]))
    s = synthetic.holstein_1d_setup(1, 1.0, 1.4, 0.2, g, omegas_spectral=FrequencyGrid(-1.0, 0.1, np.arange(21)))
    J = R.pseudorandom_complex(2, 4, 3, 2, 1, seed=0.41)
    args = (J, 0.1 * R.pseudorandom(2, 1, seed=7) - 0.1j, 0.05, 0.1, 0.07)
    ref = oracle.apply_ladder_kernel(s, *args, omega_acoustic=1e-3)
    got = api.apply_ladder_kernel(s, *args, omega_acoustic=1e-3, path="direct_fp64")
    assert np.abs(ref).max() > 0 and np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)
