"""The FFT path's kernels behind planes too large for the one-kernel middle of
the solve (z transforms and tridiagonal solves of a (z, y) plane in shared
memory), which takes every smaller FP64 plane: FP64 warp z transforms of every
length, Stockham z transforms and the three-kernel route with walls.  The
largest planes of the one-kernel route beside them.  The route is seen by the
number of launches.  Against the oracle; 1e-12 as elsewhere on the FFT path."""
import numpy as np
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import channel_case, random_fields, rel_l2, to_device

pytestmark = pytest.mark.gpu

# (nx, ny, nz), launches of a projection: 6 with three kernels in the middle, 4 with one
CHANNELS = [((64, 194, 32), 6), ((128, 98, 64), 6), ((256, 50, 128), 6), ((512, 25, 256), 6), ((1024, 13, 512), 6),
            ((96, 50, 128), 6), ((64, 156, 40), 6), ((42, 155, 40), 6), ((42, 154, 40), 4), ((64, 192, 32), 4), ((32, 12, 512), 4)]


@pytest.mark.parametrize("shape,launches", CHANNELS)
def test_channel_projection(shape, launches):
    g, bc = channel_case(*shape)
    f = random_fields(g, 31, scale=0.5)
    out = []
    for fft_kernel in (0, 1):
        with to_device(M, g, bc, f) as s:
            s.init_pressure_solver(M.make_solver_opts(M.SOLVER_FFT, fft_kernel=fft_kernel))
            s.apply_bc()
            n0 = s.launch_count()
            s.pressure_projection(0.4e-3)
            assert s.launch_count() - n0 == (6 if fft_kernel else launches)
            out.append({n: s.get(n) for n in ("phi", "un", "vn", "wn", "pn")})
    O.apply_bc(g, f)
    phi = O.pressure_projection_fft(g, f, 0.4e-3)
    assert rel_l2(out[0]["phi"], phi) < 1e-12
    for n in ("un", "vn", "wn", "pn"):
        assert rel_l2(out[0][n], getattr(f, n)) < 1e-12, n
        assert rel_l2(out[0][n], out[1][n]) < 1e-12, n


@pytest.mark.parametrize("x_wall,z_wall,shape,launches", [
    (True, False, (14, 98, 64), 6), (False, True, (16, 50, 64), 6), (True, True, (10, 80, 48), 6),
    (True, False, (14, 96, 64), 4), (False, True, (16, 48, 64), 4)])
@pytest.mark.parametrize("fft_kernel", [0, 1])
def test_walls_projection(x_wall, z_wall, shape, launches, fft_kernel):
    """phi against the oracle's periodic solve of the mirrored right-hand side
    on the grid of twice the length, which is what the walls' problem is."""
    nx, ny, nz = shape
    g = O.Grid(nx, ny, nz, lx=1.3, ly=0.8, lz=1.1, re=400.0)
    bc = O.BC((not x_wall, False, not z_wall))
    for d, wall in ((1, x_wall), (2, True), (3, z_wall)):
        if wall:
            bc.set(d, 0, 0, typ=1, value=0.0).set(d, 1, 0, typ=1, value=0.0)
    dg = 0.3e-3
    with to_device(M, g, bc, random_fields(g, 17, scale=0.5)) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_FFT, fft_kernel=fft_kernel))
        s.apply_bc()
        u, v, w = (s.get(n) for n in ("us", "vs", "ws"))
        n0 = s.launch_count()
        s.pressure_projection(dg)
        assert s.launch_count() - n0 == (6 if fft_kernel else launches)
        phi = s.get("phi")
        s.apply_bc()
        linf = s.divergence_norms()[1]
    c = (slice(1, -1),) * 3
    rhs = ((u[1:-1, 1:-1, 2:] - u[c]) / g.dx + (v[1:-1, 2:, 1:-1] - v[c]) / g.dy + (w[2:, 1:-1, 1:-1] - w[c]) / g.dz) / dg
    rhs = np.ascontiguousarray(rhs.transpose(1, 0, 2))   # [j, k, i]
    if x_wall:
        rhs = np.concatenate([rhs, rhs[:, :, ::-1]], axis=2)
    if z_wall:
        rhs = np.concatenate([rhs, rhs[:, ::-1, :]], axis=1)
    e = O.Grid(nx * (1 + x_wall), ny, nz * (1 + z_wall), lx=1.3 * (1 + x_wall), ly=0.8, lz=1.1 * (1 + z_wall), re=400.0)
    want = O.solve_pressure_fft(e, np.ascontiguousarray(rhs))[:, :nz, :nx]
    assert rel_l2(phi, want) < 1e-12
    assert linf <= 1e-12 * float(np.max(np.abs(rhs))) * dg * 100, linf   # of ||div u*||, 100 roundings
