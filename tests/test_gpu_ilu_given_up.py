"""A strip apply that is given up leaves NaN in y, not what y held before: with
the error flag already set (every later apply ends at once), and when a wait
runs out because the strip below never runs. The flag cleared and the exchange
rows reset, the same plan gives the result of before bit for bit."""
import pytest
import torch

from linalg_calls import StripGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side_by_side", [False, True])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("bs,nx,ny", [(4, 21, 70), (9, 5, 3), (9, 40, 33), (16, 1, 9), (25, 19, 4), (36, 7, 20),
                                      (36, 800, 2)])  # the last: rows too wide for an inbox
def test_set_flag(bs, nx, ny, f32, side_by_side):
    g = StripGrid(bs, nx, ny, f32)
    want, y = torch.zeros_like(g.x), torch.full_like(g.x, 7.0)
    assert g.apply(want, side_by_side) == 0 and torch.isfinite(want).all()
    g.err.fill_(1)
    assert g.apply(y, side_by_side) == 1
    assert torch.isnan(y).all()
    g.err.zero_()
    g.pack()
    assert g.apply(y, side_by_side) == 0
    assert torch.equal(y.view(torch.int64), want.view(torch.int64))


@pytest.mark.parametrize("side_by_side", [False, True])
def test_wait_that_runs_out(side_by_side):
    bs, nx, ny = 9, 37, 30
    g = StripGrid(bs, nx, ny, False)
    y = torch.full_like(g.x, 7.0)
    assert g.apply(y, side_by_side, first=1) == 1  # nothing hands strip 1 its row below
    skipped = nx * g.strips[0][5] * bs
    assert (y[:skipped] == 7.0).all()
    assert torch.isnan(y[skipped:]).all()
