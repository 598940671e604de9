"""A device that refuses cooperative launches (cudaErrorCooperativeLaunchTooLarge,
as a stream with part of the SMs gets it), or has no memory left for the on-chip
runs' inboxes: the red-black solves run with their other kernels and give the
same bits.  The refusal is made on the host, by a cudaLaunchCooperativeKernel or
a cudaMalloc of the test's own that a child process loads first."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import numpy as np
import mobydiff_b200 as M
from tests.helpers import channel_case, random_fields, to_device

g, bc = channel_case(64, 32, 32)
f = random_fields(g, 11, "zinv", scale=0.1)
f.vs[:, 1, :] = f.vs[:, g.ny + 1, :] = 0.0
out = {}
for name, kw in (("fixed", dict(n_iter=5)), ("tol", dict(tol=1e-3)), ("pot", dict(tol=1e-3, precision=M.PREC_MIXED)),
                 ("face", dict(tol=1e-3, precision=M.PREC_MIXED, inner_form=1))):
    with to_device(M, g, bc, f) as s:
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, adaptive_checks=False, **kw))
        for p in range(2):
            st = s.pressure_projection(1e-3)
            out["%s%d" % (name, p)] = np.array([st.iterations, st.variant])
        for n in ("un", "vn", "wn", "pn"):
            out[name + n] = s.get(n)
np.savez(sys.argv[1], **out)
"""


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_refused_cooperative_launch_falls_back(tmp_path):
    src, shim = tmp_path / "refuse.c", tmp_path / "refuse.so"
    src.write_text("int cudaLaunchCooperativeKernel(void) { return 720; }\n")   # cudaErrorCooperativeLaunchTooLarge
    subprocess.check_call(["gcc", "-shared", "-fPIC", str(src), "-o", str(shim)])
    out = []
    for preload in ("", str(shim)):
        env = dict(os.environ, PYTHONPATH=ROOT)
        if preload:
            env["LD_PRELOAD"] = preload
        f = tmp_path / ("b.npz" if preload else "a.npz")
        subprocess.run([sys.executable, "-c", CHILD, str(f)], cwd=ROOT, env=env, check=True, timeout=300)
        out.append(dict(np.load(f)))
    a, b = out
    assert a["fixed0"][1] == 6 and b["fixed0"][1] == 1   # the shim is what ran
    for k in a:
        if k[-1] in "01":
            assert a[k][0] == b[k][0], k
        else:
            assert np.array_equal(a[k], b[k]), k


NO_ROOM = """
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int refuse = 0, refused = 0;
int cudaMalloc(void** p, size_t n) {
    static int (*real)(void**, size_t);
    if (refuse) { ++refused; return 2; }   /* cudaErrorMemoryAllocation */
    /* the library is not in the global scope: by name, already loaded */
    if (!real) real = (int (*)(void**, size_t))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaMalloc");
    return real(p, n);
}
"""

CHILD_NO_ROOM = """
import ctypes as C
import sys
import numpy as np
import mobydiff_b200 as M
from oracle import oracle as O
from tests.helpers import channel_case, random_fields, to_device

shim = C.CDLL(sys.argv[1])
refuse, refused = C.c_int.in_dll(shim, "refuse"), C.c_int.in_dll(shim, "refused")
g, bc = channel_case(64, 32, 32)
f = random_fields(g, 11, scale=0.1)
with to_device(M, g, bc, f) as s:
    s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, n_iter=5))
    refuse.value = 1
    st = s.pressure_projection(1e-3)
    refuse.value = 0
    assert refused.value > 0 and st.variant == 1, (refused.value, st.variant)
    O.pressure_projection_redblack(g, bc, f, 1e-3, niter=5, sor=1.7, tol=0.0)
    for n in ("un", "vn", "wn", "pn"):
        assert np.array_equal(s.get(n), getattr(f, n)), n
"""


CHILD_NO_ROOM_ENSEMBLE = """
import ctypes as C
import sys
import numpy as np
import mobydiff_b200 as M

shim = C.CDLL(sys.argv[1])
refuse, refused = C.c_int.in_dll(shim, "refuse"), C.c_int.in_dll(shim, "refused")
opts = M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=1e-4, check_every=25, precision=M.PREC_MIXED)
out = []
for no_room in (0, 1):
    with M.Ensemble([M.make_member(64, 32, 32, seed=5), M.make_member(32, 32, 48, seed=6)], opts) as E:
        E.config(256, 1)
        E.ic()
        E.step(1)
        E.config(512, 1)     # larger inboxes
        refuse.value = no_room
        E.step(1)
        refuse.value = 0
        E.step(1)            # and room again
        out.append([E.get(k, n) for k in range(2) for n in ("un", "vn", "wn", "pn")])
assert refused.value > 0
assert all(np.array_equal(a, b) for a, b in zip(*out))
"""


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
@pytest.mark.parametrize("child", [CHILD_NO_ROOM, CHILD_NO_ROOM_ENSEMBLE], ids=["channel", "ensemble"])
def test_no_room_for_the_inboxes_falls_back(tmp_path, child):
    src, shim = tmp_path / "full.c", tmp_path / "full.so"
    src.write_text(NO_ROOM)
    subprocess.check_call(["gcc", "-shared", "-fPIC", str(src), "-o", str(shim), "-ldl"])
    env = dict(os.environ, PYTHONPATH=ROOT, LD_PRELOAD=str(shim))
    r = subprocess.run([sys.executable, "-c", child, str(shim)], cwd=ROOT, env=env, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
