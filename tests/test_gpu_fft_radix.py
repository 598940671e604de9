"""The Stockham transforms on lengths that use every radix (2, 3, 4, 5, 7, 8)
alone, repeated and mixed, one line per block up to many, against the oracle."""
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import channel_case, random_fields, rel_l2, to_device


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 3, 2), (4, 5, 3), (28, 10, 14), (14, 6, 49), (98, 5, 35), (126, 7, 30),
                                   (16, 9, 64), (256, 6, 128), (90, 40, 75), (2048, 2, 16), (20, 4, 1024)])
def test_projection_on_every_radix(shape):
    g, bc = channel_case(*shape)
    f = random_fields(g, 21, scale=0.5)
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_FFT, fft_kernel=1))
        O.apply_bc(g, f)
        s.apply_bc()
        O.pressure_projection_fft(g, f, 0.4e-3)
        s.pressure_projection(0.4e-3)
        for n in ("un", "vn", "wn", "pn"):
            assert rel_l2(s.get(n), getattr(f, n)) <= 1e-12, n
