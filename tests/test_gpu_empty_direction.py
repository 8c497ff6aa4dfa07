"""The passes of 2-D runs (periodic o8 in x and y, empty z): partial plane tiles, the shortest periodic
lines, several independent planes, forcing and every RK stage, against the oracle to 1e-12 relative L2 per
variable (the RHS tolerance of the parity tests)."""
import numpy as np
import pytest

from oracle import cruna_oracle as O
from public_b200 import cases
from public_b200.cruna import Cruna, Settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(32, 4 * 2, 1), (33, 13, 1), (8, 8, 3), (65, 31, 2)])
def test_empty_z_passes(n):
    s = dict(n=n, diff=("o8_e_c_p", "o8_e_c_p", "empty"), x1=(1.0, 1.1, 1.0), R=1.0, W=1.0, mu0=0.01, T0=1.0, dt=1e-3)
    q = cases.smooth_random_state(n, seed=9)
    f = np.asfortranarray(0.1 * np.random.default_rng(2).standard_normal(q.shape))
    S = O.Solver(O.Config(**s), force=f)
    with Cruna(Settings(**s), force=f) as c:
        assert c.rhs_path == "fused"
        pairs = [(c.rhs_direct(q), S.rhs_direct(q)), (c.time_stepper_direct(q), S.time_stepper_direct(q))]
    for got, ref in pairs:
        for v in range(5):
            assert np.linalg.norm(got[..., v] - ref[..., v]) <= 1e-12 * np.linalg.norm(ref[..., v]), v
