"""Forms of a stage that a grid's size, order or dimension selects, against the oracle bit for bit: the 1D
stage in one kernel at the edges of its blocks, the 2nd-order fused sweep on odd extents, the sub-cycle loop
of the captured dissipative step, the ensemble's fused sweeps."""
import ctypes

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


@pytest.mark.parametrize("dim,eta,sub", [(2, 1e-3, 1), (2, 0.15, 3), (3, 0.12, 2)])
@pytest.mark.parametrize("nu", [0.0, 0.01])
def test_subcycle_loop(restatement, dim, eta, sub, nu):
    """The captured step's loop over the dissipative sub-cycles against the eager guarded ones and the
    oracle, with and without viscosity."""
    p = P.kelvin_helmholtz(dim, 22, nym=17, nzm=9, mach=0.3, rmn=1)
    p.eta0, p.nu0 = eta, nu
    a = restatement.run(p, 4, mode=R.MODE_DRUN)
    n = 1 + int(2 * (max(2 * nu, eta) * a["dt"]) / min(p.dx, p.dy, p.dz if dim == 3 else p.dx) ** 2)
    assert abs(n - sub) <= 1, n
    for graph in (True, False):
        assert_bitwise(run_gpu(p, R.MODE_DRUN, 4, use_graph=graph)["state"], a["state"], f"{eta} {nu} graph={graph}")


def test_too_many_subcycles_are_refused():
    p = P.kelvin_helmholtz(2, 22, nym=17, mach=0.3, rmn=1)
    with L.Context.from_problem(p) as ctx:
        for graph in (True, False):
            ctx.run_reset()
            ctx.upload(p.state)
            with pytest.raises(L.QasError) as e:
                ctx.run(max_steps=4, flg=1, cfl=p.cfl, eta0=2.0, use_graph=graph)
            assert e.value.status == L.QAS_ERR_UNSUPPORTED


def _flags(*dn):
    return tuple((f,) * P.NM for f in dn)


WALLS = ((2, -2, 2, 2, 2, 2, 2, 2), (1, 1, -1, 1, 1, -1, 1, 1), (2, 1, 2, -1, 1, 2, -1, 2))  # field by field


@pytest.mark.parametrize("rmn,odr", [(1, 4), (3, 4), (2, 2), (0, 3), (2, 1)])
@pytest.mark.parametrize("dn", [_flags(0, 0, 0), _flags(1, 2, 0), WALLS, _flags(0, 1, 2)],
                         ids=["periodic", "neumann_open", "walls", "mixed_axes"])
@pytest.mark.parametrize("dim", [2, 3])
def test_small_grids_and_boundary_kinds(restatement, dim, rmn, odr, dn):
    """The overlapped launches of small steps: every boundary kind, grids down to the narrowest, runs in one
    call and in two, a single step."""
    for n in (4, 5, 11, 33):
        p = P.smooth_wave(dim, n, rmn=rmn, odr=odr, amp=0.05, dn=dn)
        a = restatement.run(p, 5, mode=R.MODE_RUN)
        with L.Context.from_problem(p) as ctx:
            ctx.upload(p.state)
            ctx.run(max_steps=2, flg=p.flg, cfl=p.cfl)
            ctx.run(max_steps=3, flg=p.flg, cfl=p.cfl)
            assert_bitwise(ctx.download(p.state.shape), a["state"], f"{dim}d {n}")
        b = restatement.run(p, 1, mode=R.MODE_STEP, dt=1e-3)
        assert_bitwise(run_gpu(p, R.MODE_STEP, dt=1e-3)["state"], b["state"], f"{dim}d {n} one step")
        if dim == 3 and n > 10:
            break


def test_step_keeps_the_callers_ghosts(restatement):
    """ideal(dt) does not fill the ghosts first: its first stage sees the caller's."""
    p = P.orszag_tang(20, nym=15)
    rng = np.random.default_rng(3)
    ghost = np.ones(p.state.shape[1:], dtype=bool)
    ghost[:, 4:-4, 4:-4] = False
    p.state[:, ghost] *= 1.0 + 0.01 * rng.standard_normal(int(ghost.sum()))
    g = restatement.grid(p)
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        ctx.step(1e-3)
        out = ctx.download(p.state.shape)
    want = np.ascontiguousarray(p.state.copy())
    assert restatement.lib.qo_step(ctypes.byref(g), restatement._ptr(want), 1e-3) == 0
    assert_bitwise(out, want, "step without bound")


@pytest.mark.parametrize("n", [(24, 21), (150, 300), (12, 10, 14), (44, 46, 45)])
def test_host_step_windows_by_size(restatement, n):
    """The host round trip with the windows its grid selects: one, two and several."""
    d = dict(zip(("nym", "nzm"), n[1:]))
    p = P.orszag_tang(n[0], **d) if len(n) == 2 else P.kelvin_helmholtz(3, n[0], mach=0.2, rmn=3, **d)
    a = restatement.run(p, 3, mode=R.MODE_RUN)
    with L.Context.from_problem(p) as ctx:
        x = np.ascontiguousarray(p.state.copy())
        for _ in range(3):
            ctx.step_host(x, x, flg=p.flg, cfl=p.cfl)
        assert_bitwise(x, a["state"], f"{n}")
