"""qas_profile_run times the kernels of a run: their names and numbers in the forms that a grid selects, and the state
that it leaves, ghosts included."""
import pytest

from oracle import refcase as R
from qasmhd_b200 import lib as L
from qasmhd_b200 import problems as P
from tests.cases import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,want", [
    (lambda: P.smooth_wave(1, 61, amp=0.1), {"k_stage1": 3}),
    (lambda: P.orszag_tang(32), {"k_sweep": 6, "k_update": 3}),
    (lambda: P.orszag_tang(32, rmn=2, odr=2), {"k_sweep": 3, "k_dv": 3}),
    (lambda: P.kelvin_helmholtz(3, 12, mach=0.3), {"k_sweep": 9, "k_emf": 3})], ids=["1d", "2d", "2d_odr2", "3d"])
@pytest.mark.parametrize("steps", [2, 3])
def test_profiled_kernels(restatement, make, want, steps):
    p = make()
    with L.Context.from_problem(p) as ctx:
        ctx.set_option(L.QAS_OPT_PROFILE_AS_RUN, 1)
        ctx.upload(p.state)
        prof = ctx.profile(steps, flg=p.flg, cfl=p.cfl)
        out = ctx.download(p.state.shape)
    assert {k: prof[k][0] for k in want} == {k: n * steps for k, n in want.items()}
    assert "k_lr" not in prof and "k_flux" not in prof
    # a fresh context runs one step before the timed ones
    assert_bitwise(out, restatement.run(p, steps + 1, mode=R.MODE_RUN)["state"], p.name)
