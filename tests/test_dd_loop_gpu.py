"""The slabs' loop control over many steps: the largest CFL maximum reaches every slab whatever the order in which
their streams run on, so the split run keeps the single domain's dt, time and state."""
import pytest

from qasmhd_b200 import lib as L
from qasmhd_b200 import problems as P
from tests.cases import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nparts", [2, 3, 5])
@pytest.mark.parametrize("make", [lambda: P.orszag_tang(32, nym=64), lambda: P.kelvin_helmholtz(3, 10, nzm=40, mach=0.3)],
                         ids=["2d", "3d"])
def test_many_steps(make, nparts):
    p = make()
    with L.Context.from_problem(p) as ctx:
        ctx.upload(p.state)
        one = ctx.run(max_steps=60, flg=1, cfl=p.cfl)
        want = ctx.download(p.state.shape)
    for _ in range(8):
        with L.Decomposition(p, nparts) as dd:
            dd.upload(p.state)
            info = dd.run(max_steps=60, flg=1, cfl=p.cfl)
            out = dd.download()
        assert (info.dt, info.tim, info.n) == (one.dt, one.tim, one.n)
        assert_bitwise(out, want, f"{p.name} x{nparts}")
