"""The allocation-free solve on grids that take its other routes: planes beyond
a block's shared memory (tables in the scratch, five kernels), rows longer than
the chained route takes, blocks that ask for more than the default shared
memory; and a call captured into a graph, behind a copy and alone.  Against
the oracle, 1e-12 as for the regular entry point."""
import ctypes as C

import numpy as np
import pytest

import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


def _solve(g, rhs, phi, stream):
    fn = M.lib().mdx_solve_pressure_fft_noalloc
    rc = fn(C.c_void_p(rhs.data_ptr()), C.c_void_p(phi.data_ptr()), C.c_int(g.nx), C.c_int(g.ny), C.c_int(g.nz),
            C.c_double(g.dx), C.c_double(g.dy), C.c_double(g.dz), C.c_void_p(stream))
    assert rc == M.MDX_OK, M.lib().mdx_last_error(None).decode()


def _case(shape, seed):
    g = O.Grid(*shape, lx=2.0, ly=1.0, lz=1.5)
    rhs = np.random.default_rng(seed).standard_normal((g.ny, g.nz, g.nx))
    return g, rhs, O.solve_pressure_fft(g, rhs)


# five kernels; chained, more than 48 KB in the middle kernel; in the row kernels; the longest chained rows
@pytest.mark.parametrize("shape", [(16, 98, 64), (30, 50, 128), (2058, 3, 4), (24, 40, 40), (2000, 4, 6), (2048, 3, 5)])
def test_routes_match_oracle(shape):
    import torch

    g, rhs, want = _case(shape, 51)
    d = torch.from_numpy(rhs).to("cuda")
    out = torch.full_like(d, float("nan"))
    for _ in range(2):
        _solve(g, d, out, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), want) <= 1e-12


@pytest.mark.parametrize("shape", [(32, 24, 32), (16, 98, 64)])
@pytest.mark.parametrize("copy_first", [False, True])
def test_captured_call(shape, copy_first):
    import torch

    g, rhs, want = _case(shape, 52)
    src = torch.from_numpy(rhs).to("cuda")
    d, out = torch.zeros_like(src), torch.zeros_like(src)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        _solve(g, src, out, st.cuda_stream)   # the first call on a device comes before any capture
        if not copy_first:
            d.copy_(src)
        st.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            if copy_first:
                d.copy_(src)
            _solve(g, d, out, st.cuda_stream)
            _solve(g, out, d, st.cuda_stream)   # and one that reads what the first wrote
        for _ in range(2):
            if not copy_first:
                d.copy_(src)
            out.zero_()
            graph.replay()
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), want) <= 1e-12
    assert rel_l2(d.cpu().numpy(), O.solve_pressure_fft(g, np.ascontiguousarray(out.cpu().numpy()))) <= 1e-12
