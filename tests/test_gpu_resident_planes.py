"""The on-chip red-black runs whose threads hold 8 and 16 planes
(test_gpu_resident.py's grids take the 4-plane kernels, but for one): boxes of
even, odd and unequal numbers of planes, and one row of blocks in y, whose
neighbours in a periodic y are themselves.  Same bits as the oracle (FP64) and
as the colour sweeps (FP32)."""
import numpy as np
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import random_fields, to_device

pytestmark = pytest.mark.gpu

# on 148 SMs, planes per box: 8-plane kernel 5-6, 8; 16-plane kernel 10-11, 9-10, 13-14, 8-9
FP64 = [(128, 64, 64), (4, 148, 1184), (66, 74, 134), (34, 148, 118), (128, 96, 80), (8, 4, 1200)]
# potential form (nx a multiple of 4): 8-plane 5, 4-5, 4-5 (one row of blocks); 16-plane 8-9, 14-15, 8-9
POT = [(128, 96, 80), (100, 90, 110), (8, 148, 600), (248, 40, 150), (256, 128, 128), (8, 4, 1200)]
# FP32 faces: 8-plane 5-6, 6-7, 8; 16-plane 8-9, 10, 8-9
FACE = [(128, 64, 64), (66, 74, 134), (160, 80, 80), (34, 148, 118), (100, 90, 110), (8, 4, 1200)]


def _case(shape, periodic_y, ibm):
    g = O.Grid(*shape, lx=1.1, ly=0.8, lz=1.7, re=800.0)
    return g, O.BC((True, True, True)) if periodic_y else O.channel_bc(), random_fields(g, 13, ibm)


@pytest.mark.parametrize("shape", FP64)
@pytest.mark.parametrize("periodic_y,ibm", [(False, "zinv"), (False, "none"), (True, "zinv"), (True, "none")])
def test_fp64_planes_equal_oracle(shape, periodic_y, ibm):
    g, bc, f = _case(shape, periodic_y, ibm)
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=3, sor=1.7, sor_variant=6))
        O.pressure_projection_redblack(g, bc, f, 0.5e-3, niter=3, sor=1.7, tol=0.0)
        assert s.pressure_projection(0.5e-3).variant == 6
        for n in ("un", "vn", "wn", "pn"):
            assert np.array_equal(s.get(n), getattr(f, n)), n


@pytest.mark.parametrize("form,shape", [(0, s) for s in POT] + [(1, s) for s in FACE])
@pytest.mark.parametrize("periodic_y", [False, True])
def test_fp32_planes_equal_colour_sweeps(form, shape, periodic_y):
    g, bc, f = _case(shape, periodic_y, "zinv")
    out = []
    for variant in (1, 0):
        with to_device(M, g, bc, f) as s:
            s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=1e-30, check_every=3, max_iter=6,
                                                      precision=M.PREC_MIXED, sor_variant=variant, inner_form=form,
                                                      adaptive_checks=False))
            it = s.pressure_projection(0.5e-3, check=False).iterations
            out.append((it, {n: s.get(n) for n in ("un", "vn", "wn", "pn")}, s.launch_count()))
    assert out[0][0] == out[1][0] and out[1][2] < out[0][2]   # same iterations in fewer launches
    for n, a in out[0][1].items():
        assert np.array_equal(a, out[1][1][n]), n
