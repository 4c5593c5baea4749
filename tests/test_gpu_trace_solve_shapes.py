"""Trace solve (ddhdg_solve_condensed) at the sizes where its kernels change:
fronts around the register-array sizes of the one-CTA kernel, odd and ragged
meshes, boundary cells that eliminate more than 36 dofs, separators around
the 32-column panel, the 64 x 64 update tile, and the rows that one CTA of
the panel kernel holds (512; 2 and 4 CTAs per cluster beyond).

The tolerance is on the normwise backward error of the row-equilibrated
system D A x = D b (D = 1 / max |row|, the scaling the solver applies): LU
with partial pivoting gives max|D(A x - b)| <= c n eps g (|D A| |x| + |D b|)
in the maximum norm with element growth g; n eps is below 3e-11 for the
largest system here, and 1e-10 allows for a growth of a few."""

import numpy as np
import pytest

from tests.test_gpu_trace_solve import _csr, _setup
from ddhdg_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,m,k", [(1, 1, 2), (1, 2, 1), (1, 37, 3), (2, 1, 3), (2, 2, 2), (2, 3, 3), (2, 5, 2),
                                     (2, 7, 1), (2, 11, 1), (2, 21, 3), (2, 33, 2), (2, 59, 2), (2, 120, 2),
                                     (3, 1, 2), (3, 2, 1), (3, 3, 2), (3, 5, 1), (3, 7, 1)])
def test_solution_satisfies_the_assembled_system(dim, m, k):
    torch, g = _setup(dim, m, k)
    tt, rhs, fl, dv = g.assemble_condense()
    A, b = _csr(torch, g, tt, rhs, fl, dv)
    x = torch.full((A.shape[0],), float("nan"), dtype=torch.float64, device=g.device)
    for rep in range(3):  # eager, captured, replayed
        _lib.check(g.L.ddhdg_solve_condensed(g._ctx, tt.data_ptr(), rhs.data_ptr(), fl.data_ptr(), dv.data_ptr(),
                                             x.data_ptr(), 0, g._sp()), "solve_condensed")
        torch.cuda.synchronize()
        xg = x.cpu().numpy()
        assert np.isfinite(xg).all()
        D = 1.0 / abs(A).max(axis=1).toarray().ravel()
        norm = (D * np.asarray(abs(A).sum(axis=1)).ravel()).max()
        scale = norm * np.abs(xg).max() + np.abs(D * b).max()
        assert np.abs(D * (A @ xg - b)).max() <= 1e-10 * scale


@pytest.mark.parametrize("dim,m,k", [(2, 32, 2), (2, 33, 1), (3, 6, 1)])
def test_repeated_solves_give_the_same_bits(dim, m, k):
    """Every kernel is deterministic; the last panels of these fronts hold
    fewer than 32 columns (72 = 32 + 32 + 8 eliminated dofs and the like)."""
    torch, g = _setup(dim, m, k)
    tt, rhs, fl, dv = g.assemble_condense()
    x = torch.empty(g.sizes().n_trace_dofs, dtype=torch.float64, device=g.device)
    ref = None
    for rep in range(40):
        x.fill_(float("nan"))
        _lib.check(g.L.ddhdg_solve_condensed(g._ctx, tt.data_ptr(), rhs.data_ptr(), fl.data_ptr(), dv.data_ptr(),
                                             x.data_ptr(), 0, g._sp()), "solve_condensed")
        if ref is None:
            ref = x.clone()
        assert torch.equal(x, ref)
