"""Options set between two runs of a context: the state, ghosts included, against the oracle."""
import pytest

from oracle import refcase as R
from qasmhd_b200 import lib as L
from qasmhd_b200 import problems as P
from tests.cases import assert_bitwise

pytestmark = pytest.mark.gpu


def _periodic(dim):
    return P.smooth_wave(dim, 61 if dim == 1 else 13, amp=0.1)


@pytest.mark.parametrize("option", [L.QAS_OPT_FUSED_SWEEP, L.QAS_OPT_LR_STAGING])
@pytest.mark.parametrize("value", [0, 1])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_option_between_runs(restatement, dim, value, option):
    """The stages' form changes with the option, the captured steps of the run before do not outlive it: an odd
    number of steps (the last one issued by itself), then an even one."""
    if option == L.QAS_OPT_LR_STAGING and dim == 1:
        pytest.skip("the staged reconstruction is for 2D and 3D")
    p = _periodic(dim)
    if option == L.QAS_OPT_LR_STAGING:
        p = P.smooth_wave(dim, 16, amp=0.1)  # an even padded extent
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        ctx.run(max_steps=4, flg=p.flg, cfl=p.cfl)
        n = 4
        for value_, steps in ((value, 3), (value, 2), (1 - value, 3)):
            ctx.set_option(option, value_)
            ctx.run(max_steps=steps, flg=p.flg, cfl=p.cfl)
            n += steps
            want = restatement.run(p, n, mode=R.MODE_RUN)["state"]
            assert_bitwise(ctx.download(p.state.shape), want, f"{dim}d option {option} = {value_}, {n} steps")
