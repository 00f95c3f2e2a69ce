"""Options set between two runs of a context: the state, ghosts included, against the oracle.  The ghosts after a
run that ends in a device error."""
import numpy as np
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


@pytest.mark.parametrize("stop_rule", [0, 1])
def test_1d_ghosts_after_a_refused_state(stop_rule):
    """A run that ends with a latched device error leaves the ghosts filled from its last state, wherever in the
    call the error is found."""
    p = _periodic(1)
    p.state[7, :, :, 30] = 0.05  # a negative pressure
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        with pytest.raises(L.QasError) as e:
            ctx.run(max_steps=40, flg=p.flg, cfl=p.cfl, stop_rule=stop_rule, dtrec=100.0)
        assert e.value.status == L.QAS_ERR_NONFINITE
        out = ctx.download(p.state.shape)
    n = p.nxm
    assert not np.array_equal(out, p.state, equal_nan=True)
    assert_bitwise(out[..., :4], out[..., n:n + 4], "lower ghosts")
    assert_bitwise(out[..., n + 4:], out[..., 4:8], "upper ghosts")
