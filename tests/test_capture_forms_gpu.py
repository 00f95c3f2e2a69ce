"""The captured steps of a run in both of their forms, one launch after the other and with the face sweeps as branches,
as the number of steps and of calls selects them: the state against the oracle."""
import pytest

from oracle import refcase as R
from qasmhd_b200 import lib as L
from qasmhd_b200 import problems as P
from tests.cases import assert_bitwise

pytestmark = pytest.mark.gpu

CASES = {"ot2d_hlld": (lambda: P.orszag_tang(31, nym=22), 0.0),
         "kh2d_mlau": (lambda: P.kelvin_helmholtz(2, 24, nym=19, mach=0.3), 0.0),
         "kh3d_mlau": (lambda: P.kelvin_helmholtz(3, 11, nym=9, nzm=10, mach=0.3), 0.0),
         "rt2d_lhlld": (lambda: P.rayleigh_taylor(2, 16, 40, rmn=2), 0.0),
         "kh2d_roe_eta": (lambda: P.kelvin_helmholtz(2, 24, nym=19, mach=0.3, rmn=0), 0.02),
         "kh3d_hlld_eta": (lambda: P.kelvin_helmholtz(3, 11, nym=9, nzm=10, mach=0.3, rmn=1), 0.02),
         "ot2d_lhlld_odr2": (lambda: P.orszag_tang(31, nym=22, rmn=2, odr=2), 0.0)}


@pytest.mark.parametrize("calls", [(4, 4, 5), (35,)], ids=str)
@pytest.mark.parametrize("case", list(CASES))
def test_calls_of_a_context(restatement, case, calls):
    make, eta = CASES[case]
    p = make()
    p.eta0 = eta
    want = restatement.run(p, sum(calls), mode=R.MODE_DRUN if eta else R.MODE_RUN)["state"]
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        for n in calls:
            ctx.run(max_steps=n, flg=p.flg, cfl=p.cfl, eta0=eta)
        assert_bitwise(ctx.download(p.state.shape), want, f"{case} {calls}")


@pytest.mark.parametrize("calls", [(4, 30, 5), (35,)], ids=str)
@pytest.mark.parametrize("odr", [2, 4])
def test_calls_of_an_ensemble(restatement, calls, odr):
    probs = P.ensemble(5, lo=12, hi=36, seed=4, odr=odr)
    with L.Batch(probs) as b:
        for q, p in enumerate(probs):
            b.upload(q, p.state)
        for n in calls:
            b.run(max_steps=n, flg=1, cfl=0.4)
        for q, p in enumerate(probs):
            want = restatement.run(p, sum(calls), mode=R.MODE_RUN)["state"]
            assert_bitwise(b.download(q, p.state.shape), want, f"{p.name} {calls}")


@pytest.mark.parametrize("n", [(1 << 18) - 8, (1 << 18) - 7])
@pytest.mark.parametrize("rmn,odr", [(1, 4), (0, 2), (3, 2)])
def test_1d_stage_form_by_size(restatement, n, rmn, odr):
    """The padded sizes on either side of the line between one kernel a stage and separate ones."""
    p = P.smooth_wave(1, n, amp=0.1, rmn=rmn, odr=odr)
    want = restatement.run(p, 3, mode=R.MODE_RUN)["state"]
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        ctx.run(max_steps=3, flg=p.flg, cfl=p.cfl)
        assert_bitwise(ctx.download(p.state.shape), want, f"{n} {rmn} {odr}")


@pytest.mark.parametrize("case", ["kh2d_roe_eta", "kh3d_hlld_eta"])
def test_captured_subcycles_without_a_loop_node(restatement, case):
    """Where the loop node cannot be made the captured step holds the guarded sub-cycles."""
    make, eta = CASES[case]
    p = make()
    p.eta0 = eta
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        n = 0
        for steps, no_loop in ((4, 1), (4, None), (3, 0)):  # the second call's capture has branches
            if no_loop is not None:
                ctx.set_option(L.QAS_OPT_TEST_NO_LOOP, no_loop)
            ctx.run(max_steps=steps, flg=p.flg, cfl=p.cfl, eta0=eta)
            n += steps
            want = restatement.run(p, n, mode=R.MODE_DRUN)["state"]
            assert_bitwise(ctx.download(p.state.shape), want, f"{case} {n} steps")
