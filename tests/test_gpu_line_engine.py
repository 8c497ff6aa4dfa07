"""The line engine and the passes built on it, at the sizes where they can go wrong: lines one point short
of, at and past a multiple of the 16 points a thread holds, lines shorter than one chunk, lines long enough
for fewer lines per block, partial plane tiles, and mixes of compact, explicit, open and empty directions.
Against the oracle: compact operators to 1e-12 of the field maximum (as the operator parity tests), RHS and
RK4 steps to 1e-12 relative L2 per variable (plus 1e-13 max|q| / dx for the one-sided closure rows)."""
import numpy as np
import pytest

from oracle import cruna_oracle as O
from public_b200 import cases
from public_b200.cruna import Cruna, Settings

pytestmark = pytest.mark.gpu


def close(a, b, floor=0.0):
    for v in range(5):
        d = np.linalg.norm(a[..., v] - b[..., v])
        assert d <= 1e-12 * np.linalg.norm(b[..., v]) + floor * np.sqrt(b[..., v].size), (v, d)


@pytest.mark.parametrize("length", [11, 15, 16, 17, 33, 97, 193, 400, 1000, 2048, 2049])
def test_compact_operators_at_chunk_edges(length):
    rng = np.random.default_rng(length)
    for d in range(3):
        n = [3, 2, 3]
        n[d] = length
        n = tuple(n)
        for scheme in ("o6_i_c_p", "o6_i_c_o", "o4_i_c_p_pade", "o4_i_c_o_pade"):
            diff, x1 = ["empty"] * 3, [1.0] * 3
            diff[d] = scheme
            f = np.asfortranarray(rng.standard_normal(n))
            with Cruna(Settings(n=n, diff=tuple(diff), x1=tuple(x1))) as c:
                got = getattr(c, f"Dx{d + 1}")(f, h=c.dx[d])
                ref = O.Dx(O.Config(n=n, diff=tuple(diff), x1=tuple(x1)), d, f, c.dx[d])
            assert np.max(np.abs(np.squeeze(got) - np.squeeze(ref))) < 1e-12 * np.max(np.abs(ref)), (scheme, d)
        for scheme in ("o6_i_c_p", "o10_i_c_o", "o2_i_c_o"):
            filt = ["empty"] * 3
            filt[d] = scheme
            f = np.asfortranarray(rng.standard_normal(n))
            kw = dict(n=n, diff=("empty",) * 3, filt=tuple(filt), alpha=0.45)
            with Cruna(Settings(**kw)) as c:
                got = getattr(c, f"filter_i{d + 1}")(f)
            ref = O.filter_dir(O.Config(**kw), d, f[..., None])[..., 0]
            assert np.max(np.abs(np.squeeze(got) - np.squeeze(ref))) < 1e-12 * np.max(np.abs(ref)), (scheme, d)


@pytest.mark.parametrize("scheme", ["o6_i_c_p", "o10_i_c_o"])
def test_filters_beyond_diagonal_dominance_keep_the_pivoted_solve(scheme):
    # alpha > 0.5: elimination without row interchanges meets pivots of 0.02, so these take the general path
    n = (40, 37, 33)
    f = np.asfortranarray(np.random.default_rng(4).standard_normal(n))
    kw = dict(n=n, diff=("empty",) * 3, filt=(scheme,) * 3, alpha=0.55)
    with Cruna(Settings(**kw)) as c:
        for d in range(3):
            got = getattr(c, f"filter_i{d + 1}")(f)
            ref = O.filter_dir(O.Config(**kw), d, f[..., None])[..., 0]
            assert np.max(np.abs(np.squeeze(got) - ref)) < 1e-12 * np.max(np.abs(ref)), d


MIXES = [("o6_i_c_p", "o6_i_c_p", "o6_i_c_p"), ("o6_i_c_o", "o4_i_c_p_pade", "o8_e_c_p"),
         ("o8_e_c_p", "o6_i_c_o", "o8_e_c_p"), ("o8_e_c_p", "o4_i_c_p_pade", "o8_e_c_p"),
         ("o4_e_c_o", "o4_i_c_o_pade", "empty"), ("o2_e_c_o", "o8_e_c_p", "o6_i_c_o"), ("empty", "empty", "o6_i_c_p")]


@pytest.mark.parametrize("n", [(17, 16, 15), (33, 9, 18), (12, 50, 11)])
@pytest.mark.parametrize("diff", MIXES)
def test_rhs_and_steps_of_scheme_mixes(n, diff):
    n = tuple(1 if s == "empty" and d == 2 else m for d, (m, s) in enumerate(zip(n, diff)))
    s = dict(n=n, diff=diff, x1=(1.0, 1.2, 0.9), R=1.0, W=1.0, mu0=0.01, T0=1.0, dt=1e-3)
    q = cases.smooth_random_state(n, seed=5)
    rng = np.random.default_rng(7)
    qs, g, f = (np.asfortranarray(0.1 * rng.standard_normal(q.shape)) for _ in range(3))
    S = O.Solver(O.Config(**s), force=f)
    with Cruna(Settings(**s), force=f) as c:
        floor = 1e-13 * np.max(np.abs(q)) / min(h for h in c.dx if np.isfinite(h))
        close(c.rhs_direct(q), S.rhs_direct(q), floor)
        close(c.rhs_adjoint(qs, q, g), S.rhs_adjoint(qs, q, g), floor)
        close(c.time_stepper_direct(q), S.time_stepper_direct(q), s["dt"] * floor)
        close(c.time_stepper_adjoint(qs, q, g), S.time_stepper_adjoint(qs, q, g), s["dt"] * floor)


@pytest.mark.parametrize("rows", ["sponge", "sponge and wall", "two sponges"])
def test_sponge_in_the_last_pass_or_after_it(rows):
    s, q = cases.mixing_layer(n=(20, 40, 17))
    bc = s["bc"]
    if rows == "sponge and wall":
        bc = np.vstack([bc, [100, 1, 20, 1, 1, 1, 17, 3, 0, 0]])
    elif rows == "two sponges":
        bc = np.vstack([bc, bc[-1]])
    s = dict(s, bc=bc)
    cfg = O.Config(**{k: v for k, v in s.items() if k in {f.name for f in O.dataclasses.fields(O.Config)}})
    qp = np.asfortranarray(q * (1.0 + 1e-2 * np.random.default_rng(3).standard_normal(q.shape)))
    S = O.Solver(cfg, qref=q.copy())
    with Cruna(Settings.from_dict(s), qref=q) as c:
        close(c.rhs_direct(qp), S.rhs_direct(qp))
        close(c.calc_direct(qp, 2), S.calc_direct(qp, 2))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [0, 47, 149])
def test_a_non_finite_value_reaches_its_whole_line_and_no_other(at, bad):
    # a sequential solve carries it to both ends; the lines beside it keep their values to rounding (1e-14 of the maximum)
    rng = np.random.default_rng(3)
    for d in range(3):
        for diff, filt in (("o6_i_c_o", "o10_i_c_o"), ("o6_i_c_p", "o6_i_c_p")):
            n = [6, 5, 7]
            n[d] = 150
            dd, ff, x1 = ["empty"] * 3, ["empty"] * 3, [1.0] * 3
            dd[d], ff[d] = diff, filt
            f = np.asfortranarray(rng.standard_normal(n))
            g = f.copy(order="F")
            where = [2, 3, 4]
            where[d] = at
            g[tuple(where)] = bad
            with Cruna(Settings(n=tuple(n), diff=tuple(dd), filt=tuple(ff), x1=tuple(x1), alpha=0.45)) as c:
                ops = [getattr(c, f"Dx{d + 1}"), getattr(c, f"filter_i{d + 1}")]
                out = [(np.asarray(op(f)).reshape(n, order="F"), np.asarray(op(g)).reshape(n, order="F")) for op in ops]
            line = tuple(slice(None) if k == d else where[k] for k in range(3))
            for clean, got in out:
                assert not np.any(np.isfinite(got[line])), (d, diff)
                rest = np.ones(n, dtype=bool)
                rest[line] = False
                assert np.max(np.abs(got[rest] - clean[rest])) <= 1e-14 * np.max(np.abs(clean)), (d, diff)
