"""The ensemble's on-chip rounds against its rounds of grid-wide barriers (the
64-register variant never goes on chip): the same bits and iterations, members
converging at different rounds, rows and planes that do not divide evenly, and
a batch that fits the blocks only once its smaller members are done.  Which
batches go on chip is seen by rounds made to fail, which only they have."""
import numpy as np
import pytest

import mobydiff_b200 as M

pytestmark = pytest.mark.gpu

BATCHES = {
    "uneven": [(64, 48, 64), (34, 17, 22), (32, 32, 48), (90, 24, 20)],
    "one": [(48, 20, 18)],
    "fits_later": [(128, 64, 128), (64, 48, 64), (32, 24, 32)],
}


def _members(name):
    return [M.make_member(*q, re=2500.0 + 300.0 * k, amp=0.03 * (k % 3), seed=5 + k) for k, q in enumerate(BATCHES[name])]


def _opts(form, check_every, precision=M.PREC_MIXED):
    return M.make_solver_opts(M.SOLVER_REDBLACK, sor=1.7, tol=1e-4, check_every=check_every, precision=precision,
                              inner_form=form)


def _run(name, opts, threads, low_regs):
    with M.Ensemble(_members(name), opts) as E:
        E.config(threads, 0, low_regs=low_regs)
        E.set_guess(M.GUESS_EXTRAPOLATED)
        E.ic()
        its = E.step(2)
        n = len(BATCHES[name])
        return its, [E.member_stats(k)[1] for k in range(n)], [E.get(k, f) for k in range(n) for f in ("un", "vn", "wn", "pn")]


@pytest.mark.parametrize("name", list(BATCHES))
@pytest.mark.parametrize("form,check_every", [(1, 25), (1, 7), (1, 4), (1, 3), (2, 25)])
@pytest.mark.parametrize("threads", [256, 512])
def test_on_chip_rounds_equal_grid_barriers(name, form, check_every, threads):
    a = _run(name, _opts(form, check_every), threads, False)
    b = _run(name, _opts(form, check_every), threads, True)
    assert a[:2] == b[:2]
    assert all(np.array_equal(x, y) for x, y in zip(a[2], b[2]))


@pytest.mark.parametrize("form,precision,low_regs,check_every,on_chip", [
    (0, M.PREC_MIXED, False, 25, True), (1, M.PREC_MIXED, False, 25, True), (0, M.PREC_MIXED, True, 25, False),
    (2, M.PREC_MIXED, False, 25, False), (0, M.PREC_FP64, False, 25, False), (0, M.PREC_MIXED, False, 4, True),
    (0, M.PREC_MIXED, False, 3, False)])
def test_which_batches_go_on_chip(form, precision, low_regs, check_every, on_chip):
    with M.Ensemble(_members("uneven"), _opts(form, check_every, precision)) as E:
        E.config(512, 0, low_regs=low_regs)
        E.ic()
        E.fail_waits(True)
        if on_chip:
            with pytest.raises(M.MdxError) as e:
                E.step(1)
            assert e.value.code == M.MDX_ERR_TIMEOUT
        else:
            E.step(1)


def test_tuned_shapes_are_kept_per_kind_of_sweep(tmp_path):
    """The same members in FP64, mixed face form, mixed with short rounds and
    mixed potential form run different kernels: one cache entry each, and a
    second ensemble of a kind takes its own."""
    import json
    cache = str(tmp_path / "tune.json")
    kinds = [_opts(0, 25, M.PREC_FP64), _opts(0, 25), _opts(0, 3), _opts(2, 25)]
    chosen = []
    for n, opts in enumerate(kinds):
        with M.Ensemble(_members("one"), opts) as E:
            E.ic()
            chosen.append(E.tune(cache))
            assert chosen[-1][3] > 0.0           # timed, not another kind's entry
            assert E.info()["grid"] % chosen[-1][1] == 0
        assert len(json.load(open(cache))) == n + 1
    for opts, c in zip(kinds, chosen):
        with M.Ensemble(_members("one"), opts) as E:
            E.ic()
            assert E.tune(cache) == c[:3] + (-1.0,)
