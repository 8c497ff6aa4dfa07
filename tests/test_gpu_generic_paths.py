"""Which kernels the generic path runs, by the names of the built-in profile, and the sequence of single
derivatives against the oracle on lines that no other path takes."""
import numpy as np
import pytest

from oracle import cruna_oracle as O
from oracle import discrete_adjoint as DA
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


@pytest.mark.parametrize("diff, n, passes", [
    (("o6_i_c_p",) * 3, (24, 20, 18), True), (("o6_i_c_o", "o8_e_c_p", "o6_i_c_p"), (24, 20, 18), True),
    (("o8_e_c_p",) * 3, (128, 128, 64), True), (("o8_e_c_p",) * 3, (24, 20, 18), False),
    (("o8_e_c_p",) * 3, (512, 64, 32), False), (("o4_e_c_o",) * 3, (24, 20, 18), False),
    (("o4_e_c_p", "o6_i_c_o", "o4_e_c_p"), (24, 20, 18), False)])
def test_generic_direct_passes_only_where_they_are_faster(diff, n, passes):
    q = cases.smooth_random_state(n, seed=1)
    with Cruna(Settings(n=n, diff=diff, **BASE)) as c:
        c.force_generic(True)
        names = kernels(c, lambda: c.time_stepper_direct(q))
    assert ("dir_flux_x" in names) == passes
    assert any(k.startswith(("line_diff_", "compact_diff_")) for k in names) != passes


LONG = [(2049, 8, 9), (8, 2049, 8), (9, 8, 2049)]    # one line past the line engine: single derivatives throughout
MIXED = [(33, 9, 18), (17, 16, 15)]                  # o8 along x or y beside compact directions: passes


@pytest.mark.parametrize("n, diff", [(n, d) for n in LONG for d in (("o4_e_c_o", "o8_e_c_p", "o4_e_c_p"),
                                                                    ("o6_i_c_p", "o6_i_c_o", "o4_i_c_p_pade"))]
                         + [(n, d) for n in MIXED for d in (("o8_e_c_p", "o6_i_c_o", "o6_i_c_p"),
                                                            ("o6_i_c_p", "o8_e_c_p", "o6_i_c_o"))]
                         + [(n, ("o8_e_c_p", "o6_i_c_o", "o8_e_c_p")) for n in ((2051, 9, 8), (8, 9, 2051))])
def test_rhs_and_steps_against_the_oracle(n, diff):
    # RHS to 1e-12 relative L2 per variable plus 1e-13 max|q| / dx (one-sided closure rows), a step to dt times the latter
    q = cases.smooth_random_state(n, seed=5)
    rng = np.random.default_rng(7)
    qs, g, f = (np.asfortranarray(0.1 * rng.standard_normal(q.shape)) for _ in range(3))
    s = dict(BASE, n=n, diff=diff, dt=1e-6)  # dt within the viscous limit of 2049 points
    S = O.Solver(O.Config(**s), force=f)
    with Cruna(Settings(**s), force=f) as c:
        c.force_generic(True)
        floor = 1e-13 * np.max(np.abs(q)) / min(c.dx)
        got = [(c.rhs_direct(q), S.rhs_direct(q), floor), (c.rhs_adjoint(qs, q, g), S.rhs_adjoint(qs, q, g), floor),
               (c.time_stepper_direct(q), S.time_stepper_direct(q), s["dt"] * floor),
               (c.time_stepper_adjoint(qs, q, g), S.time_stepper_adjoint(qs, q, g), s["dt"] * floor)]
    for a, b, f0 in got:
        for v in range(5):
            assert np.linalg.norm(a[..., v] - b[..., v]) <= 1e-12 * np.linalg.norm(b[..., v]) + f0 * np.sqrt(b[..., v].size), v


@pytest.mark.parametrize("length", [24, 64, 1023, 1024, 1025])
@pytest.mark.parametrize("scheme", ["o6_i_c_p", "o10_i_c_o"])
def test_filters_beyond_diagonal_dominance_run_one_kernel_along_y_and_z(scheme, length):
    # alpha > 0.5: no row table.  Both sides eliminate with row interchanges: 50 eps cond(B) of the field maximum
    alpha = 0.55
    B = np.eye(length) + alpha * (np.eye(length, k=1) + np.eye(length, k=-1))
    if scheme.endswith("p"):
        B[0, -1] = B[-1, 0] = alpha
    else:
        B[0, 1] = B[-1, -2] = 0.0
    tol = 50 * np.finfo(float).eps * np.linalg.cond(B)
    for d in (1, 2):
        n = [3, 2, 2]
        n[d] = length
        n = tuple(n)
        f = np.asfortranarray(np.random.default_rng(length).standard_normal(n))
        filt = ["empty"] * 3
        filt[d] = scheme
        kw = dict(n=n, diff=("empty",) * 3, filt=tuple(filt), alpha=alpha)
        out = []
        with Cruna(Settings(**kw)) as c:
            names = kernels(c, lambda: out.append(getattr(c, f"filter_i{d + 1}")(f)))
        axis = "xyz"[d]
        assert names == ({"compact_filter_" + axis} if length <= 1024 else {"line_filter_" + axis, "line_solve_" + axis})
        ref = O.filter_dir(O.Config(**kw), d, f[..., None])[..., 0]
        assert np.max(np.abs(np.squeeze(out[0]) - np.squeeze(ref))) <= tol * np.max(np.abs(ref)), d


@pytest.mark.parametrize("n, d, diff, filt", [
    ((256, 209, 103), 1, "o6_i_c_o", "o10_i_c_o"), ((128, 390, 205), 1, "o6_i_c_p", "o6_i_c_p"),
    ((64, 400, 103), 1, "o6_i_c_o", "o10_i_c_o"), ((64, 32, 800), 2, "o6_i_c_o", "o6_i_c_o"),
    ((64, 800, 52), 1, "o6_i_c_p", "o6_i_c_p"), ((64, 1024, 52), 1, "o4_i_c_o_pade", "o2_i_c_o"),
    ((64, 32, 900), 2, "o4_i_c_p_pade", "o8_i_c_o"), ((64, 800, 32), 1, "o4_i_c_o_pade", "o4_i_c_o"),
    ((1800, 50, 50), 0, "o6_i_c_o", "o10_i_c_o")])
def test_long_lines_leave_the_line_engine_on_many_lines(n, d, diff, filt):
    # five fields at the sizes where the rule changes: to 1e-12 of the field maximum, as the operator parity tests
    f = np.asfortranarray(np.random.default_rng(n[d]).standard_normal((*n, 5)))
    dd, ff, x1 = ["empty"] * 3, ["empty"] * 3, [1.0] * 3
    dd[d], ff[d] = diff, filt
    kw = dict(n=n, diff=tuple(dd), filt=tuple(ff), x1=tuple(x1), alpha=0.45)
    got = {}
    with Cruna(Settings(**kw)) as c:
        names = kernels(c, lambda: got.update(dx=getattr(c, f"Dx{d + 1}")(f, h=c.dx[d]), filt=getattr(c, f"filter_i{d + 1}")(f)))
        h = c.dx[d]
    assert ("line_solve_x" in names) == (d == 0)
    cfg = O.Config(**kw)
    for v in range(5):
        ref = O.Dx(cfg, d, np.asfortranarray(f[..., v]), h)
        assert np.max(np.abs(got["dx"][..., v] - ref)) < 1e-12 * np.max(np.abs(ref)), v
    ref = O.filter_dir(cfg, d, f)
    assert np.max(np.abs(got["filt"] - ref)) < 1e-12 * np.max(np.abs(ref))


def test_type_201_rows_join_in_runs_and_keep_table_order():
    # overlapping faces (joined, more than one launch holds), a box of more than 2^19 points and a row by itself,
    # none of which commute: to 1e-12 relative L2 per variable; launches: 8 + 1, the box, the last row
    n = (96, 80, 72)
    full = [1, n[0], 1, n[1], 1, n[2]]
    faces = []
    for d in range(3):
        for end in (1, n[d]):
            box, k = list(full), [0.0, 0.0, 0.0]
            box[2 * d] = box[2 * d + 1] = end
            k[d] = -1.0 if end == 1 else 1.0
            faces.append([201, *box, *k])
    bc = np.array(faces + faces[:3] + [[201, *full, 0, 1, 0], faces[2]], dtype=float)
    q = cases.smooth_random_state(n, seed=3)
    rng = np.random.default_rng(4)
    ref = np.asfortranarray(q * (1.0 + 1e-2 * rng.standard_normal(q.shape)))
    qs = np.asfortranarray(0.1 * rng.standard_normal(q.shape))
    s = dict(BASE, n=n, diff=("o4_e_c_o",) * 3, bc=bc)
    S = O.Solver(O.Config(**s), qref=ref)
    with Cruna(Settings(**s), qref=ref) as c:
        before = c.launches
        got = c.set_boundary_condition_q(q)
        assert c.launches - before == 4
        got_s = c.set_boundary_condition_qs(qs, q)
        assert c.launches - before == 8
    for a, b in ((got, S.set_boundary_condition_q(q)), (got_s, S.set_boundary_condition_qs(qs, q))):
        for v in range(5):
            assert np.linalg.norm(a[..., v] - b[..., v]) <= 1e-12 * np.linalg.norm(b[..., v]), v


def test_step_vjp_with_filters_beyond_diagonal_dominance():
    # transposed solves with row interchanges along y and z; 1e-10 relative L2 as the discrete adjoint's other tests
    # (the matrices' condition numbers are below 1e3 at these sizes)
    n = (14, 15, 16)
    s = dict(BASE, n=n, diff=("o6_i_c_p", "o6_i_c_o", "o8_e_c_p"), filt=("o6_i_c_p", "o10_i_c_o", "o6_i_c_o"), alpha=0.55,
             di_freq=(1, 1, 1))
    for size, scheme in zip(n, s["filt"]):
        B = np.eye(size) + 0.55 * (np.eye(size, k=1) + np.eye(size, k=-1))
        if scheme.endswith("p"):
            B[0, -1] = B[-1, 0] = 0.55
        else:
            B[0, 1] = B[-1, -2] = 0.0
        assert np.linalg.cond(B) < 1e3
    q = cases.smooth_random_state(n, seed=7)
    lam = np.asfortranarray(np.random.default_rng(9).standard_normal(q.shape))
    ref, _ = DA.step_vjp(O.Solver(O.Config(**s)), q, lam, 1)
    with Cruna(Settings(**s)) as c:
        out = []
        names = kernels(c, lambda: out.append(c.step_direct_vjp(q, lam, 1)))
    assert {"line_solve_x", "line_solve_y", "line_solve_z"} <= names
    for v in range(5):
        scale = max(np.linalg.norm(ref[..., v]), 1e-3 * np.linalg.norm(ref))
        assert np.linalg.norm(out[0][..., v] - ref[..., v]) <= 1e-10 * scale, v
