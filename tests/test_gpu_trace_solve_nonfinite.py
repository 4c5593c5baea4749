"""An overflowed condensed block reaches the trace solve as an infinity in a
row of tt.  The row's equilibration factor is then 1 / Inf = 0 and the row
holds 0 * Inf = NaN: the solve reports a singular front, or the NaN reaches x;
it never returns DDHDG_OK with a finite x, whichever kernel holds the row
(boundary cell, interior cell read by its parent, panel fronts)."""

import numpy as np
import pytest

from ddhdg_b200 import _lib
from tests.test_gpu_trace_solve import _setup

pytestmark = pytest.mark.gpu

SOLVER_ERROR = 8  # DDHDG_SOLVER_ERROR


def _solve(g, torch, tt, rhs, fl, dv, x):
    r = g.L.ddhdg_solve_condensed(g._ctx, tt.data_ptr(), rhs.data_ptr(), fl.data_ptr(), dv.data_ptr(),
                                  x.data_ptr(), 0, g._sp())
    torch.cuda.synchronize()
    return r


# (2, 1, 3): one cell of 48 eliminated dofs (panel kernel); (2, 4, 1) and
# (3, 4, 1): boundary and interior cells of the one-CTA kernel; (3, 3, 2):
# boundary cells of the panel kernel
@pytest.mark.parametrize("dim,m,k", [(1, 5, 2), (2, 4, 1), (2, 1, 3), (2, 6, 2), (3, 4, 1), (3, 3, 2)])
def test_an_infinite_row_is_never_hidden(dim, m, k):
    torch, g = _setup(dim, m, k)
    tt, rhs, fl, dv = g.assemble_condense()
    x = torch.empty(g.nfaces * 3 * g.nf, dtype=torch.float64, device=g.device)
    flags = fl.cpu().numpy()
    rng = np.random.default_rng(7)
    cells = sorted({0, g.ncells // 2, g.ncells - 1, int(rng.integers(g.ncells))})
    for cell in cells:
        free = np.flatnonzero(flags[cell] == 0)
        for row in {int(free[0]), int(free[-1]), int(rng.choice(free))}:
            for col, val in ((row, np.inf), (int(rng.choice(free)), -np.inf)):
                bad = tt.clone()
                bad[cell, row, col] = val
                x.fill_(float("nan"))
                r = _solve(g, torch, bad, rhs, fl, dv, x)
                assert r in (0, SOLVER_ERROR)
                assert r == SOLVER_ERROR or not torch.isfinite(x).all(), (cell, row, col, val)
    # the context still solves the unharmed system
    x.fill_(float("nan"))
    _lib.check(_solve(g, torch, tt, rhs, fl, dv, x), "solve_condensed")
    assert torch.isfinite(x).all()
