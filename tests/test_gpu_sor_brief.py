"""Which kernels a fixed count of red-black iterations takes on grids that fit
the SMs: the sweeps for one or two (three on larger grids), the on-chip run
from there on and wherever it is asked for.  The same bits as the oracle."""
import numpy as np
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import channel_case, random_fields, to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n_iter,variant,record,runs", [
    ((32, 24, 32), 1, 0, False, 1), ((32, 24, 32), 2, 0, False, 1), ((32, 24, 32), 3, 0, False, 6),
    ((128, 76, 62), 3, 0, False, 1), ((128, 76, 62), 4, 0, False, 6), ((32, 24, 32), 1, 6, False, 6),
    ((32, 24, 32), 1, 0, True, 6), ((32, 24, 32), 0, 0, False, 1)])
def test_kernels_of_a_fixed_count(shape, n_iter, variant, record, runs):
    g, bc = channel_case(*shape)
    f = random_fields(g, 19, "zinv")
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=n_iter, sor=1.7, sor_variant=variant))
        if record:
            s.set_pressure_guess(M.GUESS_ZERO, record=True)
        assert s.pressure_projection(0.5e-3).variant == runs
        O.pressure_projection_redblack(g, bc, f, 0.5e-3, niter=n_iter, sor=1.7, tol=0.0)
        for n in ("un", "vn", "wn", "pn"):
            assert np.array_equal(s.get(n), getattr(f, n)), n
