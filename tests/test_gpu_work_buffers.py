"""Work buffers of a context: whatever gradient or objective call ran before, with other snapshot counts, host
snapshots or another context in between, a call gives the bits that a fresh context gives; and a step allocates no more
than its path needs."""
import numpy as np
import pytest
import torch

from public_b200 import cases
from public_b200.cruna import Cruna, Settings
from public_b200.slabs import HALO_FN

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


def test_a_marching_run_with_a_sponge_allocates_no_rhs_buffer():
    # 49 workspace fields and 15 intermediates; the 5 of an RHS buffer (31 MB here) would not fit the 16 MB of slack
    n = (128, 96, 64)
    used = []
    for size in ((20, 40, 17), n):              # the first run loads the kernels
        s, q = cases.mixing_layer(n=size)
        with Cruna(Settings.from_dict(s), qref=q) as c:
            qd, qs = torch.from_numpy(np.ascontiguousarray(q.T)).cuda(), torch.zeros(q.size, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            c.step_direct_dev(qd.data_ptr(), qd.data_ptr())
            c.step_adjoint_dev(qs.data_ptr(), qd.data_ptr(), None, qs.data_ptr())
            c.sync()
            used.append(before - torch.cuda.mem_get_info()[0])
    assert used[-1] <= 64 * 8 * n[0] * n[1] * n[2] + (16 << 20), used


def test_adjoint_stages_keep_the_frozen_state_across_a_halo_callback():
    # between the stages the callback evaluates a direct RHS and closure features on the same context and workspace
    s, q = cases.mixing_layer(n=(24, 33, 18))
    s = dict(s, bc=None)
    rng = np.random.default_rng(2)
    q = q * (1.0 + 1e-2 * rng.standard_normal(q.shape))
    dev = [torch.from_numpy(np.ascontiguousarray(a.T)).cuda() for a in (q, 1e-3 * rng.standard_normal(q.shape), 1.1 * q)]
    qd, qs, other = dev
    rhs, out, plain = (torch.empty_like(qd) for _ in range(3))
    x = torch.empty(q[..., 0].size, 12, dtype=torch.float32, device="cuda")
    with Cruna(Settings.from_dict(s)) as c:
        c.step_adjoint_dev(qs.data_ptr(), qd.data_ptr(), None, plain.data_ptr())
        @HALO_FN
        def halo(user, fields, nfields, stream):
            c.rhs_direct_dev(other.data_ptr(), rhs.data_ptr())
            c.closure_features_dev(other.data_ptr(), 0.1, x.data_ptr())
            return 0

        c.set_halo_exchange(halo)
        c.step_adjoint_dev(qs.data_ptr(), qd.data_ptr(), None, out.data_ptr())
        c.set_halo_exchange(None)
        c.sync()
    assert torch.equal(out, plain)
