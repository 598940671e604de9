"""A block of an on-chip red-black run that gives up a wait: the call that hands
out the half-swept fields, or a number made of them, returns MDX_ERR_TIMEOUT,
and the context works again afterwards.  The wait is made to run out by a limit
of no reads at all; every block still ends by itself."""
import numpy as np
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import channel_case, random_fields, to_device

pytestmark = pytest.mark.gpu

SHAPE = (64, 32, 32)   # dozens of blocks

READOUTS = {
    "get": lambda s, tmp: s.get("un"),
    "update_host": lambda s, tmp: s.update_host(np.empty(s.padded)),
    "write_field_h5": lambda s, tmp: s.write_field_h5(str(tmp / "f.h5")),
    "get_cfl": lambda s, tmp: s.get_cfl(),
    "center_vel": lambda s, tmp: s.center_vel(),
    "divergence_norms": lambda s, tmp: s.divergence_norms(),
    "step_adaptive": lambda s, tmp: s.step_adaptive(1, 0.5, 1e-3),
    "channel_ic": lambda s, tmp: s.channel_ic(1),
    "increment": lambda s, tmp: s.get_increment(0),
}


@pytest.mark.parametrize("readout", list(READOUTS))
def test_fixed_count_reports_at_the_next_readout(readout, tmp_path):
    g, bc = channel_case(*SHAPE)
    f = random_fields(g, 7, scale=0.1)
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=200, sor=1.7, sor_variant=6))
        s.set_pressure_guess(M.GUESS_ZERO, record=True)
        s.set_wait_limit(0)
        if readout not in ("step_adaptive", "channel_ic"):   # these make their own runs
            s.pressure_projection(1e-3)
        with pytest.raises(M.MdxError) as e:
            READOUTS[readout](s, tmp_path)
        assert e.value.code == M.MDX_ERR_TIMEOUT
        assert not (tmp_path / "f.h5").exists()
        # reported once; fresh fields and the usual limit give the oracle's bits
        s.set_wait_limit(-1)
        s.set_pressure_guess(M.GUESS_ZERO, record=False)
        for n in ("us", "vs", "ws", "pn"):
            s.set(n, getattr(f, n))
        s.pressure_projection(1e-3)
        O.pressure_projection_redblack(g, bc, f, 1e-3, niter=200, sor=1.7, tol=0.0)
        for n in ("un", "vn", "wn", "pn"):
            assert np.array_equal(s.get(n), getattr(f, n)), n


@pytest.mark.parametrize("precision,form", [(M.PREC_FP64, 0), (M.PREC_MIXED, 0), (M.PREC_MIXED, 1)])
def test_tolerance_solve_reports_itself(precision, form):
    g, bc = channel_case(*SHAPE)
    f = random_fields(g, 8, scale=0.1)
    f.vs[:, 1, :] = f.vs[:, g.ny + 1, :] = 0.0   # walls: no net flux, so that the residual has no floor
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=1e-6, check_every=50,
                                                  precision=precision, inner_form=form))
        s.set_wait_limit(0)
        with pytest.raises(M.MdxError) as e:
            s.pressure_projection(1e-3)
        assert e.value.code == M.MDX_ERR_TIMEOUT
        s.set_wait_limit(-1)
        for n in ("us", "vs", "ws", "pn"):
            s.set(n, getattr(f, n))
        assert s.pressure_projection(1e-3).residual <= 1.0000001e-6


@pytest.mark.parametrize("form", [0, 1])
def test_mixed_solve_after_a_timeout_equals_a_fresh_one(form):
    """Nothing of the abandoned FP32 corrections reaches the next solve: the
    same bits as in a context that never gave up.  Runs of one iteration, so
    that some blocks finish and write while others give up; limits from no
    reads up to where whole runs succeed before one does not."""
    g, bc = channel_case(*SHAPE)
    f = random_fields(g, 9, scale=0.1)
    f.vs[:, 1, :] = f.vs[:, g.ny + 1, :] = 0.0
    opts = M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=1e-6, check_every=1, precision=M.PREC_MIXED,
                              inner_form=form, adaptive_checks=False)

    def solve(s):
        for n in ("us", "vs", "ws", "pn"):
            s.set(n, getattr(f, n))
        st = s.pressure_projection(1e-3, check=False)
        return st.rc, st.iterations

    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(opts)
        fresh = solve(s)
        assert fresh[0] == M.MDX_OK
        want = {n: s.get(n) for n in ("un", "vn", "wn", "pn")}
    gave_up = 0
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(opts)
        for polls in (0, 1, 2, 3, 4, 6, 8, 12, 16, 32):
            s.set_wait_limit(polls)
            rc, _ = solve(s)
            assert rc in (M.MDX_OK, M.MDX_ERR_TIMEOUT)
            gave_up += rc == M.MDX_ERR_TIMEOUT
            s.set_wait_limit(-1)
            assert solve(s) == fresh, polls
            for n, a in want.items():
                assert np.array_equal(s.get(n), a), (polls, n)
    assert gave_up > 0
