"""Work buffers kept with the context between gradient and objective calls: whatever was called before, with
other snapshot counts, host snapshots or another context in between, a call gives the bits that a fresh context gives."""
import numpy as np
import pytest

from public_b200 import cases
from public_b200.cruna import Cruna, Settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_calls_on_one_context_match_fresh_contexts(mode):
    s, q = cases.mixing_layer(n=(20, 40, 17))
    goal = Cruna.objective("plane_p2", normal=2, index=12, p_inf=1.0)
    energy = Cruna.objective("kinetic_energy")

    def context():
        c = Cruna(Settings.from_dict(s), qref=q)
        c.set_adjoint_mode(mode)
        return c

    def gradient(c, objective, nsnap, host):
        c.set_snapshot_memory(host)
        return c.gradient(q, 5, nsnap, objective)

    calls = [lambda c: gradient(c, goal, 2, False), lambda c: c.objective_value(q, 4, goal), lambda c: gradient(c, energy, 4, False),
             lambda c: gradient(c, goal, 3, True), lambda c: c.objective_value(q, 2, energy), lambda c: gradient(c, goal, 3, True),
             lambda c: gradient(c, energy, 1, False), lambda c: gradient(c, goal, 2, False)]
    with context() as c, context() as other:
        for call in calls:
            got = call(c)
            call(other)
            with context() as fresh:
                ref = call(fresh)
            for a, b in zip(np.atleast_1d(got) if np.isscalar(got) else got, np.atleast_1d(ref) if np.isscalar(ref) else ref):
                assert np.array_equal(np.asarray(a), np.asarray(b))
