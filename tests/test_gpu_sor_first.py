"""A fixed number of red-black sweeps starts from u* without copying it: the
first sweep reads u*, v*, w* and the ghost layers and wall rows are set beside
it.  The same bits as the oracle, everywhere in the arrays, on tiles' edges and
remainders, odd ny, one iteration and more."""
import numpy as np
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import random_fields, to_device


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 2, 2), (8, 5, 6), (66, 9, 4), (130, 34, 10)])
@pytest.mark.parametrize("periodic_y,ibm", [(False, "zinv"), (False, "none"), (True, "zinv"), (True, "none")])
@pytest.mark.parametrize("n_iter", [1, 3])
def test_first_sweep_from_ustar(shape, periodic_y, ibm, n_iter):
    if periodic_y and shape[1] % 2:
        pytest.skip("periodic y takes even ny")
    g = O.Grid(*shape, lx=1.1, ly=0.8, lz=1.7, re=800.0)
    bc = O.BC((True, True, True)) if periodic_y else O.channel_bc()
    f = random_fields(g, 29, ibm)
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=n_iter, sor=1.7, sor_variant=1))
        for _ in range(2):   # the second starts from u, v, w that differ from u*, v*, w*
            O.pressure_projection_redblack(g, bc, f, 0.5e-3, niter=n_iter, sor=1.7, tol=0.0)
            s.pressure_projection(0.5e-3)
        for n in ("un", "vn", "wn", "pn"):
            assert np.array_equal(s.get(n), getattr(f, n)), n
