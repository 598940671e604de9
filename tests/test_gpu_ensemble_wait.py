"""On-chip sweeps of the ensemble that give up a wait: MDX_ERR_TIMEOUT from the
call, also when the projections after it end well, and the ensemble works again
afterwards with the bits of one that never gave up."""
import numpy as np
import pytest

import mobydiff_b200 as M

pytestmark = pytest.mark.gpu

SIZES = [(64, 32, 32), (32, 32, 48)]


def _opts(**kw):
    return M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, check_every=25, precision=M.PREC_MIXED, **kw)


def _members(**kw):
    return [M.make_member(*q, seed=5 + k, **kw) for k, q in enumerate(SIZES)]


def _fields(E):
    return [E.get(k, n) for k in range(len(SIZES)) for n in ("un", "vn", "wn", "pn")]


@pytest.mark.parametrize("graph", [False, True])
def test_step_reports_and_recovers(graph):
    out = []
    for give_up in (False, True):
        with M.Ensemble(_members(amp=0.04), _opts(tol=1e-6)) as E:
            E.use_graph(graph)
            if give_up:
                E.fail_waits(True)
                with pytest.raises(M.MdxError) as e:   # the t=0 projection
                    E.ic()
                assert e.value.code == M.MDX_ERR_TIMEOUT
                E.fail_waits(False)
                E.ic()
                E.fail_waits(True)
                with pytest.raises(M.MdxError) as e:
                    E.step(2)
                assert e.value.code == M.MDX_ERR_TIMEOUT
                with pytest.raises(M.MdxError) as e:
                    E.tune()
                assert e.value.code == M.MDX_ERR_TIMEOUT
                E.fail_waits(False)
            E.ic()
            its = E.step(2)
            out.append((its, _fields(E)))
    assert out[0][0] == out[1][0]
    assert all(np.array_equal(a, b) for a, b in zip(out[0][1], out[1][1]))


def test_timeout_of_an_early_step_is_not_lost():
    """Strong viscosity: the divergence of a disturbed field falls from step to
    step even though the projections give up.  With the absolute target between
    the first step's and the second's, only the first step sweeps."""
    rng = np.random.default_rng(3)
    noise = []
    for nx, ny, nz in SIZES:
        a = [rng.uniform(-1e-3, 1e-3, (nz + 2, ny + 2, nx + 2)) for _ in range(3)]
        a[1][:, 1, :] = a[1][:, ny + 1, :] = 0.0
        noise.append(a)

    def ready(atol):
        E = M.Ensemble(_members(re=1.0, amp=0.0), _opts(tol=1e-12, atol=atol))
        E.ic()
        for k, a in enumerate(noise):
            for n, x in zip(("un", "vn", "wn"), a):
                E.set(k, n, x)
        E.fail_waits(True)
        return E

    last = []   # per member, ||div u*|| of each step's last projection
    with ready(1e-6) as E:
        for _ in range(2):
            with pytest.raises(M.MdxError):
                E.step(1)
            last.append([E.member_stats(k)[0].residual0 for k in range(len(SIZES))])
    lo, hi = max(last[1]), min(last[0])
    assert 0.0 < lo < 0.9 * hi, last
    with ready((lo * hi) ** 0.5) as E:
        with pytest.raises(M.MdxError) as e:
            E.step(2)
        assert e.value.code == M.MDX_ERR_TIMEOUT
        assert all(E.member_stats(k)[0].status == M.MDX_OK for k in range(len(SIZES)))   # the last projections'
        assert E.step(0) == 0   # reported once
