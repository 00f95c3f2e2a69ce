"""Forms of a stage that a grid's size, order or dimension selects, against the oracle bit for bit: the 1D
stage in one kernel at the edges of its blocks, the 2nd-order fused sweep on odd extents, the sub-cycle loop
of the captured dissipative step, the ensemble's fused sweeps."""
import numpy as np
import pytest

from oracle import refcase as R
from qasmhd_b200 import lib as L
from qasmhd_b200 import problems as P
from tests.cases import assert_bitwise, run_gpu

pytestmark = pytest.mark.gpu
TC = 56  # cells a block of the 1D stage kernel updates


def _wave1d(n, flag, **kw):
    p = P.smooth_wave(1, n, amp=0.1, **{k: v for k, v in kw.items() if k != "char_mode"})
    p.dnx = (flag,) * P.NM
    p.char_mode = kw.get("char_mode", 0)
    return p


@pytest.mark.parametrize("n", [4, 8, TC - 1, TC, TC + 1, 3 * TC + 2])
@pytest.mark.parametrize("flag", [0, 1, 2])
def test_1d_stage_block_edges(restatement, n, flag):
    p = _wave1d(n, flag)
    a = restatement.run(p, 5, mode=R.MODE_RUN)
    for graph in (True, False):
        assert_bitwise(run_gpu(p, R.MODE_RUN, 5, use_graph=graph)["state"], a["state"], f"{n} {flag} graph={graph}")


@pytest.mark.parametrize("rmn", [0, 1, 2, 3])
@pytest.mark.parametrize("kw", [dict(odr=2), dict(odr=4), dict(odr=4, rk=2), dict(odr=2, rk=1), dict(odr=3),
                                dict(odr=4, char_mode=1)], ids=str)
def test_1d_stage_schemes(restatement, rmn, kw):
    p = _wave1d(61, 1, rmn=rmn, **kw)
    a = restatement.run(p, 4, mode=R.MODE_RUN)
    assert_bitwise(run_gpu(p, R.MODE_RUN, 4)["state"], a["state"], f"rmn {rmn} {kw}")


def test_1d_resumed_and_finished_run(restatement):
    """Two calls equal one; a call with no step left changes nothing, the ghosts neither."""
    p = P.brio_wu(130)
    a = restatement.run(p, 7, mode=R.MODE_RUN)
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        ctx.run(max_steps=3, flg=p.flg, cfl=p.cfl)
        info = ctx.run(max_steps=4, flg=p.flg, cfl=p.cfl)
        assert info.n == 7 and info.steps == 4
        assert_bitwise(ctx.download(p.state.shape), a["state"], "resumed")
    q = P.brio_wu(130)
    b = restatement.run(q, 0, mode=R.MODE_EXEC)
    with L.Context.from_problem(q) as ctx:
        ctx.upload(q.state)
        n = ctx.run(flg=q.flg, stop_rule=2, cfl=q.cfl, dtrec=q.dtrec, nout=q.nout).steps
        assert_bitwise(ctx.download(q.state.shape), b["state"], "to its stop")
        other = q.state + 1.0  # its ghosts are not what a fill would give
        ctx.upload(other)
        assert n > 0 and ctx.run(flg=q.flg, stop_rule=2, cfl=q.cfl, dtrec=q.dtrec, nout=q.nout).steps == 0
        assert_bitwise(ctx.download(q.state.shape), other, "no step left")


@pytest.mark.parametrize("rmn", [0, 1, 2, 3])
@pytest.mark.parametrize("make", [lambda r: P.orszag_tang(31, nym=70, rmn=r, odr=2),
                                  lambda r: P.kelvin_helmholtz(3, 9, nym=35, nzm=13, mach=0.3, rmn=r, odr=2)],
                         ids=["2d", "3d"])
def test_second_order_sweep(restatement, rmn, make):
    p = make(rmn)
    a = restatement.run(p, 3, mode=R.MODE_RUN)
    for fused in (None, 0, 1):
        with L.Context.from_problem(p) as ctx:
            if fused is not None:
                ctx.set_option(L.QAS_OPT_FUSED_SWEEP, fused)
            ctx.upload(p.state)
            ctx.run(max_steps=3, flg=p.flg, cfl=p.cfl)
            assert_bitwise(ctx.download(p.state.shape), a["state"], f"rmn {rmn} fused {fused}")
