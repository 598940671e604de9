"""The on-chip red-black runs (k_sor_resident.cu): the same bits as the
one-launch-per-colour sweeps and, in FP64, as the oracle, on grids with one
block, one row or plane per box, boxes of uneven size, a warp's remainder,
walls and periodic y, IBM factors or none."""
import numpy as np
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import random_fields, to_device

SHAPES = [(4, 2, 2), (8, 6, 2), (20, 8, 6), (42, 34, 18), (64, 10, 40), (116, 70, 62), (256, 24, 40)]


def _case(shape, periodic_y, ibm):
    g = O.Grid(*shape, lx=1.1, ly=0.8, lz=1.7, re=800.0)
    bc = O.BC((True, True, True)) if periodic_y else O.channel_bc()
    return g, bc, random_fields(g, 13, ibm)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("periodic_y,ibm", [(False, "zinv"), (False, "none"), (True, "zinv"), (True, "none")])
def test_fp64_run_equals_oracle(shape, periodic_y, ibm):
    g, bc, f = _case(shape, periodic_y, ibm)
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=7, sor=1.7, sor_variant=6))
        for _ in range(2):   # a second run: later sequence numbers in the same inboxes
            O.pressure_projection_redblack(g, bc, f, 0.5e-3, niter=7, sor=1.7, tol=0.0)
            assert s.pressure_projection(0.5e-3).variant == 6
        for n in ("un", "vn", "wn", "pn"):
            assert np.array_equal(s.get(n), getattr(f, n)), n


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("periodic_y", [False, True])
@pytest.mark.parametrize("form", [0, 1])
def test_fp32_runs_equal_colour_sweeps(shape, periodic_y, form):
    """Potential form (nx a multiple of 4) and face form: 12 fixed iterations
    per inner pass, two projections."""
    g, bc, f = _case(shape, periodic_y, "zinv")
    out = []
    for variant in (1, 0):
        with to_device(M, g, bc, f) as s:
            s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=1e-30, check_every=6, max_iter=12,
                                                      precision=M.PREC_MIXED, sor_variant=variant, inner_form=form,
                                                      adaptive_checks=False))
            its = [s.pressure_projection(0.5e-3, check=False).iterations for _ in range(2)]
            out.append((its, {n: s.get(n) for n in ("un", "vn", "wn", "pn")}, s.launch_count()))
    assert out[0][0] == out[1][0] and out[1][2] < out[0][2]   # same iterations in fewer launches
    for n, a in out[0][1].items():
        assert np.array_equal(a, out[1][1][n]), (n, float(np.max(np.abs(a - out[1][1][n]))))
