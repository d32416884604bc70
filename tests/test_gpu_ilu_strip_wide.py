"""Strip applies where the width of the grid changes their launch: rows whose two
inboxes leave the ring its depth (one launch for both sweeps), rows with room
for one (a launch per sweep), and rows too wide for any (every hand-over through
global memory). Equal bit for bit to the data-flow apply, three applies in a
row."""
import pytest

from specs import BURGERS, NS, Spec
from test_gpu_ilu_strips import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kw", [dict(pde=NS, p=2, nx=60, ny=9), dict(pde=NS, p=2, nx=250, ny=9),
                                dict(pde=NS, p=2, nx=340, ny=17), dict(pde=BURGERS, p=4, nx=500, ny=19),
                                dict(pde=BURGERS, p=2, nx=1400, ny=5), dict(pde=BURGERS, p=1, nx=3000, ny=17)],
                         ids=str)
def test_widths(kw, precision):
    ctx = Spec(g=1, **kw).context()
    check(ctx, ctx.layout.n_dof, precision)
    ctx.close()
