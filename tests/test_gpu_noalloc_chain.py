"""Calls of the allocation-free solve queued one behind another on a stream,
each reading what the one before wrote: its kernels are placed while those of
the call before still run, so what they read must come from L2 after their
wait.  The same bits as the same calls with a synchronisation between them."""
import ctypes as C

import pytest

import mobydiff_b200 as M


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 2, 2), (32, 24, 32), (64, 48, 60)])
@pytest.mark.parametrize("in_place", [False, True])
def test_queued_calls_equal_synchronised_calls(shape, in_place):
    import torch

    nx, ny, nz = shape
    fn = M.lib().mdx_solve_pressure_fft_noalloc
    g = torch.Generator(device="cuda")
    g.manual_seed(17)
    first = torch.randn((ny, nz, nx), device="cuda", dtype=torch.float64, generator=g)
    out = []
    for sync in (True, False):
        a = [first.clone(), torch.zeros_like(first)]
        st = torch.cuda.current_stream()
        torch.cuda.synchronize()
        for n in range(12):
            src, dst = (a[0], a[0]) if in_place else (a[n % 2], a[1 - n % 2])
            rc = fn(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), C.c_int(nx), C.c_int(ny), C.c_int(nz),
                    C.c_double(0.2), C.c_double(0.1), C.c_double(0.15), C.c_void_p(st.cuda_stream))
            assert rc == M.MDX_OK, M.lib().mdx_last_error(None).decode()
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        out.append(a[0])
    assert bool(torch.isfinite(out[0]).all()) and float(out[0].abs().max()) > 0.0
    assert torch.equal(out[0], out[1])
