"""Which kernels the generic path runs, by the names of the built-in profile: the sequence of single derivatives
where it is the faster one, and that sequence against the oracle on lines that no other path takes."""
import numpy as np
import pytest

from public_b200 import cases
from public_b200.cruna import Cruna, Settings

pytestmark = pytest.mark.gpu

BASE = dict(x1=(1.0, 1.2, 0.9), R=1.0, W=1.0, mu0=0.01, T0=1.0, dt=1e-3)


def kernels(c, call):
    """Names of the kernel families that call() launches."""
    c.profile(True)
    call()
    names = set(c.profile_report())
    c.profile(False)
    return names


@pytest.mark.parametrize("diff", [("o6_i_c_p",) * 3, ("o6_i_c_o", "o8_e_c_p", "o6_i_c_p"), ("o4_e_c_o",) * 3, ("o8_e_c_p",) * 3])
def test_generic_adjoint_is_a_sequence_of_derivatives(diff):
    n = (24, 20, 18)
    q = cases.smooth_random_state(n, seed=1)
    with Cruna(Settings(n=n, diff=diff, **BASE)) as c:
        c.force_generic(True)
        names = kernels(c, lambda: c.time_stepper_adjoint(0.1 * q, q))
    for d, scheme in zip("xyz", diff):
        assert ("compact_diff_" if "_i_" in scheme else "line_diff_") + d in names
    assert not any(k.startswith("dir_") for k in names)
