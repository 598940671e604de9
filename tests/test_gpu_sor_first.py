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


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 2, 2), (60, 18, 4), (62, 34, 8), (122, 28, 14), (186, 12, 6)])
@pytest.mark.parametrize("periodic_y,ibm", [(False, "zinv"), (False, "none"), (True, "zinv"), (True, "none")])
@pytest.mark.parametrize("variant,kz", [(2, 0), (3, 0), (3, 1), (3, 3)])
def test_passes_from_ustar(shape, periodic_y, ibm, variant, kz):
    """Red+black passes on tiles' edges, chunks of one plane and more, an even
    and an odd number of them (they end in u, v, w either way)."""
    g = O.Grid(*shape, lx=1.1, ly=0.8, lz=1.7, re=800.0)
    bc = O.BC((True, True, True)) if periodic_y else O.channel_bc()
    f = random_fields(g, 31, ibm)
    with to_device(M, g, bc, f) as s:
        for n_iter in (1, 2, 3):
            s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=n_iter, sor=1.7, sor_variant=variant,
                                                      sor_kz=kz))
            O.pressure_projection_redblack(g, bc, f, 0.5e-3, niter=n_iter, sor=1.7, tol=0.0)
            assert s.pressure_projection(0.5e-3).variant == variant
            for n in ("un", "vn", "wn", "pn"):
                assert np.array_equal(s.get(n), getattr(f, n)), (n, n_iter)


@pytest.mark.gpu
def test_auto_takes_the_pass_on_large_grids():
    """240x102x96 walls: beyond the SMs' shared memory, where the pass is the
    faster one; the same bits as the sweeps."""
    out = []
    for variant in (0, 1):
        g = M.make_grid(240, 102, 96, 6.0, 2.0, 3.0, 3000.0, 1e-3, (2 / 3000.0, 0, 0))
        s = M.Solver(g, M.channel_bc())
        s.enter_field_data()
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=3, sor=1.5, sor_variant=variant))
        s.channel_ic(3)
        s.step(2)
        took = s.pressure_projection(0.5e-3).variant
        out.append((took, {n: s.get(n) for n in ("un", "vn", "wn", "pn")}))
        s.close()
    assert [o[0] for o in out] == [3, 1]
    for n, a in out[0][1].items():
        assert np.array_equal(a, out[1][1][n]), n
