"""Performance cases of the library's public entry points: what a program that
runs channel flows with it calls, over the sizes it calls it with.

A case is a dict of plain values.  ``listed()`` are the standing ones,
``draw(rng)`` makes another of the same ranges, ``prepare(case, seed)`` is what
a program holds before the call, ``run(state)`` one pass, ``work(case)`` what a
pass cannot do without and ``exact(case, seed)`` the pass in plain 64-bit torch.

Kinds
  poisson   the allocation-free FFT pressure solve on the caller's device arrays
  fft       RK3 steps on the FFT path between two outputs of u, v, w, p
  sor       RK3 steps with a fixed number of FP64 red-black sweeps, then output
  solve     one coupled RK3 step with red-black to a tolerance (FP64, or FP32
            sweeps in FP64 defect correction): fields in from the host program,
            step, fields out to it
  ensemble  one RK3 step of several uneven channels, fields in and out
  unet      forward and backward pass of the warm-start network
"""
import ctypes as C
import math

import numpy as np
import torch
import torch.nn.functional as F

import mobydiff_b200 as M

LX, LZ = 2 * math.pi, math.pi
RE, DT = 3000.0, 1e-3
RK = M.rk_coeffs()
SLOPE = 0.1


def listed():
    return [
        # one pressure plane set of a small coupled program: launches and latency
        {"name": "poisson_32x24x32", "kind": "poisson", "nx": 32, "ny": 24, "nz": 32},
        # the small laminar channel of the tests and the benchmark, ten steps per output
        {"name": "fft_64x32x32", "kind": "fft", "nx": 64, "ny": 32, "nz": 32, "steps": 10, "duct": False, "adaptive": False},
        # a duct (walls in z too) with the CFL-controlled time step
        {"name": "fft_duct_96x64x48", "kind": "fft", "nx": 96, "ny": 64, "nz": 48, "steps": 10, "duct": True, "adaptive": True},
        # the reference's default grid: lengths that are no powers of two
        {"name": "fft_200x200x200", "kind": "fft", "nx": 200, "ny": 200, "nz": 200, "steps": 10, "duct": False, "adaptive": False},
        # the benchmark's large turbulent channel
        {"name": "fft_512x256x256", "kind": "fft", "nx": 512, "ny": 256, "nz": 256, "steps": 10, "duct": False, "adaptive": False},
        # the reference's red-black defaults (3 sweeps, omega 1.5) on an uneven grid
        {"name": "sor_180x150x140", "kind": "sor", "nx": 180, "ny": 150, "nz": 140, "steps": 10, "n_iter": 3},
        # plain FP64 red-black of a wavy channel to a tolerance
        {"name": "solve_fp64_128x64x64", "kind": "solve", "nx": 128, "ny": 64, "nz": 64, "mixed": False, "guess": False, "tol": 1e-6},
        # mixed precision, ragged grid, from phi = 0
        {"name": "solve_mixed_116x70x62", "kind": "solve", "nx": 116, "ny": 70, "nz": 62, "mixed": True, "guess": False, "tol": 1e-8},
        # the benchmark's wavy channel: mixed precision from the extrapolated increment
        {"name": "solve_mixed_256x128x128", "kind": "solve", "nx": 256, "ny": 128, "nz": 128, "mixed": True, "guess": True, "tol": 1e-8},
        # a batch of uneven channels
        {"name": "ensemble_6", "kind": "ensemble", "sizes": "64x48x64,32x32x48,96x64x32,48x40x48,64x32x32,80x48x64", "tol": 1e-6},
        # the warm-start network, one training gradient
        {"name": "unet_128x64x64", "kind": "unet", "nx": 128, "ny": 64, "nz": 64},
    ]


# ---- drawn cases -------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(rng, lo, hi, even=False):
    """A length that factors into 2, 3, 5, 7 (its half does when `even`)."""
    while True:
        n = _log(rng, lo, hi)
        n += n & 1 if even else 0
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def _even(rng, lo, hi, q=2):
    return q * max(1, _log(rng, lo, hi) // q)


def draw(rng):
    kind = rng.choice(["poisson", "fft", "fft", "sor", "solve", "solve", "solve", "ensemble", "unet"])
    c = {"kind": kind}
    if kind == "poisson":
        return dict(c, nx=_smooth(rng, 16, 64, True), ny=_log(rng, 8, 64), nz=_smooth(rng, 8, 64))
    if kind == "fft":
        duct = rng.random() < 0.25
        top = 96 if duct else 256
        return dict(c, nx=_smooth(rng, 32, 128 if duct else 400, True), ny=_log(rng, 20, top), nz=_smooth(rng, 20, top),
                    steps=rng.choice([5, 10]), duct=duct, adaptive=rng.random() < 0.3)
    if kind == "sor":
        return dict(c, nx=_even(rng, 32, 200), ny=_log(rng, 20, 150), nz=_even(rng, 20, 140), steps=rng.choice([5, 10]),
                    n_iter=rng.choice([3, 6]))
    if kind == "solve":
        if rng.random() < 0.34:
            return dict(c, nx=_even(rng, 32, 128), ny=_log(rng, 20, 64), nz=_even(rng, 20, 64), mixed=False, guess=False,
                        tol=1e-6)
        guess = rng.random() < 0.5
        return dict(c, nx=_even(rng, 32, 256 if guess else 160), ny=_log(rng, 24, 128 if guess else 80),
                    nz=_even(rng, 24, 128 if guess else 80), mixed=True, guess=guess, tol=1e-8)
    if kind == "ensemble":
        n = rng.randint(2, 6)
        return dict(c, sizes=",".join("%dx%dx%d" % (_even(rng, 32, 96), _even(rng, 24, 64), _even(rng, 24, 64))
                                      for _ in range(n)), tol=1e-6)
    return dict(c, nx=8 * rng.randint(4, 16), ny=8 * rng.randint(2, 8), nz=8 * rng.randint(2, 8))


# ---- inputs --------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _fields(c, seed, ly=2.0):
    """u, v, w, p of a perturbed channel between y = (ly - 2)/2 and that + 2, padded [k, j, i], on the GPU."""
    g, shape = _gen(seed), (c["nz"] + 2, c["ny"] + 2, c["nx"] + 2)
    y = (torch.arange(c["ny"] + 2, device="cuda", dtype=torch.float64) - 0.5) * (ly / c["ny"]) - ly / 2
    out = [torch.empty(shape, device="cuda", dtype=torch.float64).uniform_(-a, a, generator=g) for a in (0.1, 0.01, 0.01)]
    out[0] += (1.0 - y * y).clamp_min(0.0)[None, :, None]
    return out + [torch.zeros(shape, device="cuda", dtype=torch.float64)]


def _pinned(like):
    """Host arrays a coupled program keeps for transfers (page-locked)."""
    return [torch.empty(t.shape, dtype=torch.float64, pin_memory=True) for t in like]


def _grid(c, ly):
    return M.make_grid(c["nx"], c["ny"], c["nz"], LX, ly, LZ, RE, DT, (2.0 / RE, 0.0, 0.0))


def _duct_bc():
    t = {(d, s, 0): 1 for d in (2, 3) for s in (0, 1)}   # Neumann pressure, no-slip walls in y and z
    return M.make_bc((True, False, False), types=t)


def _sizes(c):
    return [tuple(int(v) for v in s.split("x")) for s in c["sizes"].split(",")]


def prepare(case, seed):
    c = case
    st = {"case": c}
    if c["kind"] == "poisson":
        st["rhs"] = torch.randn((c["ny"], c["nz"], c["nx"]), device="cuda", dtype=torch.float64, generator=_gen(seed))
        st["phi"] = torch.empty_like(st["rhs"])
        st["h"] = (LX / c["nx"], 2.0 / c["ny"], LZ / c["nz"])
        return st
    if c["kind"] == "unet":
        n = c["nx"] * c["ny"] * c["nz"]
        s = st["s"] = M.Solver(_grid(c, 2.0), M.channel_bc())
        s.enter_field_data()
        s.unet_create(capacity=0, slope=SLOPE)
        st["in"], st["target"], p = _unet_inputs(n, s.unet_param_count(), seed)
        s.unet_set_params(p)
        return st
    if c["kind"] == "ensemble":
        mem = [M.make_member(*q, re=2500.0 + 300.0 * k, amp=0.02 * (k % 4), seed=seed + k) for k, q in enumerate(_sizes(c))]
        e = st["e"] = M.Ensemble(mem, M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=c["tol"], check_every=25,
                                                         precision=M.PREC_MIXED))
        e.ic()
        st["start"] = [[e.get(k, f) for f in ("un", "vn", "wn", "pn")] for k in range(len(mem))]
        return st
    ly = 2.25 if c["kind"] == "solve" else 2.0
    dev = _fields(c, seed, ly)
    host = _pinned(dev)
    for h, d in zip(host, dev):
        h.copy_(d)
    del dev
    f = [h.numpy() for h in host]
    s = st["s"] = M.Solver(_grid(c, ly), _duct_bc() if c.get("duct") else M.channel_bc())
    s.enter_field_data(un=f[0], vn=f[1], wn=f[2], pn=f[3])
    if c["kind"] == "fft":
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_FFT))
        s.apply_bc()
    elif c["kind"] == "sor":
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, n_iter=c["n_iter"], sor=1.5))
        s.apply_bc_redblack()
    else:
        y0 = (ly - 2.0) / 2.0
        s.enter_ibm_geometry(M.ibm_wavy(0.05, LX / 2.0, y0))
        s.init_pressure_solver(M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=c["tol"], check_every=50,
                                                  precision=M.PREC_MIXED if c["mixed"] else M.PREC_FP64))
        if c["guess"]:
            s.set_pressure_guess(M.GUESS_EXTRAPOLATED, record=True)
        s.channel_ic(seed, 0.1, 0.01, y0, 0.05, LX / 2.0)
        s.step(3 if c["guess"] else 1)
        if c["guess"]:
            s.warm_checkpoint()
        st["start"] = f
        s.update_host(*f)
        host = _pinned(host)
    st["host"] = host
    st["out"] = [h.numpy() for h in host]
    return st


def run(state):
    c = state["case"]
    if c["kind"] == "poisson":
        rhs, phi, h = state["rhs"], state["phi"], state["h"]
        rc = M.lib().mdx_solve_pressure_fft_noalloc(C.c_void_p(rhs.data_ptr()), C.c_void_p(phi.data_ptr()), C.c_int(c["nx"]),
                                                    C.c_int(c["ny"]), C.c_int(c["nz"]), C.c_double(h[0]), C.c_double(h[1]),
                                                    C.c_double(h[2]), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != M.MDX_OK:
            raise M.MdxError(rc, M.lib().mdx_last_error(None).decode())
        return phi
    if c["kind"] == "unet":
        loss, grad, out = state["s"].unet_loss_grad(state["in"], state["target"])
        return {"loss": loss, "grad": grad, "out": out}
    if c["kind"] == "ensemble":
        e = state["e"]
        for k, fields in enumerate(state["start"]):
            for name, a in zip(("un", "vn", "wn", "pn"), fields):
                e.set(k, name, a)
        e.step(1)
        return [[e.get(k, f) for f in ("un", "vn", "wn", "pn")] for k in range(len(state["start"]))]
    s = state["s"]
    if c["kind"] == "solve":
        s.update_device(*state["start"])
        if c["guess"]:
            s.warm_checkpoint(restore=True)
        s.step(1)
    elif c.get("adaptive"):
        s.step_adaptive(c["steps"], 0.5, 2e-3)
    else:
        s.step(c["steps"])
    s.update_host(*state["out"])
    return state["host"]


# ---- what a pass cannot do without -----------------------------------------------
def work(case):
    c = case
    if c["kind"] == "ensemble":
        n = sum(a * b * d for a, b, d in _sizes(c))
    else:
        n = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "poisson":
        return {"bytes": 16.0 * n, "flops": n * (5.0 * math.log2(c["nx"] * c["nz"]) + 8.0)}
    if c["kind"] == "unet":
        # 3x3x3 convolutions (channels 16 at full resolution, 32 below), forward, data and weight gradients
        macs = 27.0 * (16 * 16 * 3 + (16 * 32 + 32 * 32 + 32 * 16) / 8 + 32 * 32 * 3 / 64 + 32 * 32 * 2 / 512)
        return {"bytes": 28.0 * n, "flops": 6.0 * macs * n}
    # a substage reads and writes u, v, w, p and the three stored right-hand sides
    sub = 3 * c.get("steps", 1)
    b, f = 112.0 * n * sub, 220.0 * n * sub
    if c["kind"] == "fft":
        f += sub * n * (5.0 * math.log2(c["nx"] * c["nz"]) + 8.0)
    elif c["kind"] == "sor":   # an iteration reads and writes u, v, w, p
        b, f = b + sub * c["n_iter"] * 64.0 * n, f + sub * c["n_iter"] * 30.0 * n
    else:   # the iterations depend on the flow: a thousand per substage stand for them, from on-chip memory
        f += sub * 1000 * 16.0 * n
    return {"bytes": b, "flops": f}


# ---- the pass in 64 bits, without the library --------------------------------------
def exact(case, seed):
    c = case
    if c["kind"] == "poisson":
        rhs = torch.randn((c["ny"], c["nz"], c["nx"]), device="cuda", dtype=torch.float64, generator=_gen(seed))
        return _poisson(rhs, LX / c["nx"], 2.0 / c["ny"], LZ / c["nz"])
    if c["kind"] == "unet":
        return _unet_exact(c, seed)
    if c["kind"] in ("fft", "sor") and not c.get("duct"):
        return _steps(c, seed)
    return None


def _poisson(rhs, dx, dy, dz):
    """rhs [j, k, i] -> phi, periodic in i and k, Neumann in j with the mean mode's first row pinned to 0."""
    ny, nz, nx = rhs.shape
    kx = (4 / dx ** 2) * torch.sin(math.pi * torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64) / nx) ** 2
    kz = (4 / dz ** 2) * torch.sin(math.pi * torch.arange(nz, device="cuda", dtype=torch.float64) / nz) ** 2
    k = kz[:, None] + kx[None, :]
    h, a = torch.fft.rfft2(rhs), 1.0 / (dy * dy)
    cp, dp = torch.empty(h.shape, device="cuda", dtype=torch.float64), torch.empty_like(h)
    for j in range(ny):
        b = -k - (a if j in (0, ny - 1) else 2 * a)
        den = b if j == 0 else b - a * cp[j - 1]
        cp[j] = a / den
        dp[j] = (h[j] if j == 0 else h[j] - a * dp[j - 1]) / den
        if j == 0:
            cp[0, 0, 0], dp[0, 0, 0] = 0.0, 0.0
    for j in range(ny - 2, -1, -1):
        dp[j] -= cp[j] * dp[j + 1]
    return torch.fft.irfft2(dp, s=(nz, nx))


def _steps(c, seed):
    u, v, w, p = f = _fields(c, seed)
    us, vs, ws = g = [torch.zeros_like(t) for t in (u, v, w)]
    old = [torch.zeros((c["nz"], c["ny"], c["nx"]), device="cuda", dtype=torch.float64) for _ in range(3)]
    dx, dy, dz, dt = LX / c["nx"], 2.0 / c["ny"], LZ / c["nz"], DT
    I, H, L, A = slice(1, -1), slice(2, None), slice(0, -2), slice(None)
    fft = c["kind"] == "fft"

    def at(t, x=I, y=I, z=I):
        return t[z, y, x]

    def bc_fft():
        for a, b, n in ((u, v, w), (us, vs, ws)):
            for t in (a, n):
                t[:, -1], t[:, 0] = -t[:, -2], -t[:, 1]
            b[:, -1], b[:, 1] = 0.0, 0.0
        for t, y in ((u, A), (w, A), (us, A), (ws, A), (v, slice(1, None)), (vs, slice(1, None)), (p, I)):
            t[:, y, 0], t[:, y, -1] = t[:, y, -2].clone(), t[:, y, 1].clone()
        for t, y in ((u, A), (w, A), (us, A), (ws, A), (v, slice(1, None)), (vs, slice(1, None)), (p, I)):
            t[0, y], t[-1, y] = t[-2, y].clone(), t[1, y].clone()

    def bc_sor():
        for t in (u, w):
            t[I, 0, I], t[I, -1, I] = -t[I, 1, I], -t[I, -2, I]
        v[I, 1, I], v[I, -1, I] = 0.0, 0.0
        for t in f:
            t[I, I, 0], t[I, I, -1] = t[I, I, -2].clone(), t[I, I, 1].clone()
        for t in f:
            t[0, I, I], t[-1, I, I] = t[-2, I, I].clone(), t[1, I, I].clone()

    def lap(t):
        m = 2.0 * at(t)
        return (((at(t, x=L) - m + at(t, x=H)) / dx ** 2 + (at(t, y=L) - m + at(t, y=H)) / dy ** 2)
                + (at(t, z=L) - m + at(t, z=H)) / dz ** 2) / RE

    def momentum(a, b, gam):
        q = 0.25
        ru = (-q * ((at(u, x=H) + at(u)) ** 2 - (at(u) + at(u, x=L)) ** 2) / dx
              - q * ((at(u, y=H) + at(u)) * (at(v, y=H) + at(v, y=H, x=L)) - (at(u) + at(u, y=L)) * (at(v) + at(v, x=L))) / dy
              - q * ((at(u, z=H) + at(u)) * (at(w, z=H) + at(w, z=H, x=L)) - (at(u) + at(u, z=L)) * (at(w) + at(w, x=L))) / dz
              + 2.0 / RE + lap(u))
        rv = (-q * ((at(v, x=H) + at(v)) * (at(u, x=H) + at(u, x=H, y=L)) - (at(v) + at(v, x=L)) * (at(u) + at(u, y=L))) / dx
              - q * ((at(v, y=H) + at(v)) ** 2 - (at(v) + at(v, y=L)) ** 2) / dy
              - q * ((at(v, z=H) + at(v)) * (at(w, z=H) + at(w, z=H, y=L)) - (at(v) + at(v, z=L)) * (at(w) + at(w, y=L))) / dz
              + lap(v))
        rw = (-q * ((at(w, x=H) + at(w)) * (at(u, x=H) + at(u, x=H, z=L)) - (at(w) + at(w, x=L)) * (at(u) + at(u, z=L))) / dx
              - q * ((at(w, y=H) + at(w)) * (at(v, y=H) + at(v, y=H, z=L)) - (at(w) + at(w, y=L)) * (at(v) + at(v, z=L))) / dy
              - q * ((at(w, z=H) + at(w)) ** 2 - (at(w) + at(w, z=L)) ** 2) / dz
              + lap(w))
        grad = ((at(p) - at(p, x=L)) / dx, (at(p) - at(p, y=L)) / dy, (at(p) - at(p, z=L)) / dz)
        for n, (t, s, r) in enumerate(zip((u, v, w), g, (ru, rv, rw))):
            new = at(t) + a * r + b * old[n] - gam * grad[n]
            y = slice(1, None) if n == 1 else A   # v on the wall face is not advanced
            s[I, I, I][:, y] = new[:, y]
            old[n][:, y] = r[:, y]

    def project_fft(gam):
        div = (at(us, x=H) - at(us)) / dx + (at(vs, y=H) - at(vs)) / dy + (at(ws, z=H) - at(ws)) / dz
        phi = _poisson(div.transpose(0, 1).contiguous() / gam, dx, dy, dz).transpose(0, 1)
        u[I, I, I] = at(us) - gam * (phi - phi.roll(1, 2)) / dx
        w[I, I, I] = at(ws) - gam * (phi - phi.roll(1, 0)) / dz
        v[I, 2:-1, I] = vs[I, 2:-1, I] - gam * (phi[:, 1:] - phi[:, :-1]) / dy
        p[I, I, I] += phi

    k, j, i = torch.meshgrid(*[torch.arange(1, c[n] + 1, device="cuda") for n in ("nz", "ny", "nx")], indexing="ij")
    odd = ((i + j + k) & 1).double()

    def project_sor(gam):
        for t, s in zip((u, v, w), g):
            t.copy_(s)
        v[I, 1, I], v[I, -1, I] = 0.0, 0.0
        fac = -1.5 / (2.0 / dx ** 2 + 2.0 / dy ** 2 + 2.0 / dz ** 2)
        for _ in range(c["n_iter"]):
            for mask in (odd, 1.0 - odd):
                ui, wi = at(u), at(w)
                phi = ((ui.roll(-1, 2) - ui) / dx + (at(v, y=H) - at(v)) / dy + (wi.roll(-1, 0) - wi) / dz) * fac * mask
                p[I, I, I] += phi / gam
                ui += (phi.roll(1, 2) - phi) / dx
                wi += (phi.roll(1, 0) - phi) / dz
                v[I, 2:-1, I] += (phi[:, :-1] - phi[:, 1:]) / dy

    bc_fft() if fft else bc_sor()
    for _ in range(c["steps"]):
        for a, b, gam in zip(*RK):
            momentum(dt * a, dt * b, dt * gam)
            if fft:
                bc_fft()
                project_fft(dt * gam)
                bc_fft()
            else:
                project_sor(dt * gam)
                bc_sor()
        if c.get("adaptive"):
            dt = min(0.5 / max(float((t / h).abs().max()) for t, h in ((u, dx), (v, dy), (w, dz))), 2e-3)
    return f


def _unet_inputs(n, nparam, seed):
    r = np.random.default_rng(seed)
    x = r.standard_normal((M.UNET_INPUTS, n), dtype=np.float32)
    p, o = np.zeros(nparam, np.float32), 0
    for cin, cout in _UNET:
        p[o:o + 27 * cin * cout] = r.uniform(-1, 1, 27 * cin * cout) * math.sqrt(6.0 / (27 * cin * (1 + SLOPE ** 2)))
        o += 27 * cin * cout
        p[o:o + cout] = r.uniform(-0.1, 0.1, cout)
        o += cout
    p[o:] = r.uniform(-0.4, 0.4, nparam - o)
    return x, r.standard_normal(n, dtype=np.float32), p


_UNET = [(16, 16), (16, 16), (16, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 16), (16, 16)]


def _unet_exact(c, seed):
    shape = (c["nz"], c["ny"], c["nx"])
    nparam = sum(27 * a * b + b for a, b in _UNET) + 17
    x, target, p = _unet_inputs(int(np.prod(shape)), nparam, seed)
    p = torch.tensor(p, device="cuda", dtype=torch.float64, requires_grad=True)
    x = torch.tensor(x, device="cuda", dtype=torch.float64).reshape(1, M.UNET_INPUTS, *shape)
    x = torch.cat([x, x.new_zeros(1, 16 - M.UNET_INPUTS, *shape)], 1)
    layer, offset = iter(_UNET), [0]

    def conv(t):
        cin, cout = next(layer)
        o = offset[0]
        wt = p[o:o + 27 * cin * cout].reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
        b = p[o + 27 * cin * cout:o + 27 * cin * cout + cout]
        offset[0] = o + 27 * cin * cout + cout
        t = F.pad(F.pad(t, (1, 1, 0, 0, 1, 1), mode="circular"), (0, 0, 1, 1, 0, 0))
        return F.leaky_relu(F.conv3d(t, wt, b), SLOPE)

    skips = []
    for level in range(4):
        x = conv(conv(F.avg_pool3d(x, 2) if level else x))
        skips.append(x)
    for level in (2, 1, 0):
        x = conv(F.interpolate(x, scale_factor=2, mode="nearest") + skips[level])
    out = (x * p[-17:-1].reshape(1, 16, 1, 1, 1)).sum(1).reshape(-1) + p[-1]
    loss = ((out - torch.tensor(target, device="cuda", dtype=torch.float64)) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "grad": p.grad, "out": out.detach()}
