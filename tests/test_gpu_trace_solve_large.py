"""Trace solve (ddhdg_solve_condensed) beyond the sizes of
test_gpu_trace_solve_shapes.py, without the assembled matrix: the residual is
summed from the cells' blocks.  The bound is the one of that file, on the
normwise backward error of the row-equilibrated system."""

import pytest

from ddhdg_b200 import _lib
from tests import cases

pytestmark = pytest.mark.gpu


def _setup(n, k):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from ddhdg_b200.solver import NPSolver

    pb, prm, adim = cases.diode(dim=len(n), m=2, k=k)
    pb.mesh.n = tuple(n)
    g = NPSolver(pb, prm, adim)
    g.compute_local_charge_neutrality()
    for c in (1, 2):
        _lib.check(g.L.ddhdg_project_density(g._ctx, c, 0.0, g.cell_state.data_ptr(),
                                             g.trace_state.data_ptr(), g._sp()), "project_density")
    return torch, g


def _backward_error(torch, g, tt, rhs, fl, dv, x):
    """max |D (A x - b)| / (max row sum of |D A| max |x| + max |D b|)"""
    nd = 3 * g.nf
    faces = torch.as_tensor(g.cell_faces, device=g.device, dtype=torch.int64)
    dofs = (faces[:, :, None] * nd + torch.arange(nd, device=g.device)).reshape(g.ncells, -1)
    free = fl == 0
    n = x.numel()

    def add(cell_values):
        return torch.zeros(n, dtype=torch.float64, device=g.device).index_add_(0, dofs.reshape(-1),
                                                                               cell_values.reshape(-1))

    xl = x[dofs]
    res = add(torch.where(free, torch.bmm(tt, xl[:, :, None])[:, :, 0] - rhs, xl - dv))
    b = add(torch.where(free, rhs, dv))
    sums = add(torch.where(free, tt.abs().sum(2), torch.ones_like(xl)))
    top = torch.zeros(n, dtype=torch.float64, device=g.device).scatter_reduce_(
        0, dofs.reshape(-1), torch.where(free, tt.abs().amax(2), torch.ones_like(xl)).reshape(-1), "amax")
    scale = (sums / top).max() * x.abs().max() + (b / top).abs().max()
    return float((res / top).abs().max() / scale)


# - a rod whose 65 600 cells each eliminate four faces, 48 dofs: more fronts of
#   the panel kernels at one height than a launch has room for in its y
#   dimension
# - 11^3: fronts of 432 and 792 eliminated dofs above the 288 and 576 rows that
#   a column tile of the triangular solves holds (blocks of rows, products
#   between them), beside kept dofs
# - 40 x 19 x 19: fronts of 4332 eliminated dofs, the root and its two children
#   (4332 kept dofs each), whose LU is the library's
@pytest.mark.parametrize("n,k", [((65600, 1, 1), 1), ((11, 11, 11), 1), ((40, 19, 19), 1)])
def test_solution_satisfies_the_cells_equations(n, k):
    torch, g = _setup(n, k)
    tt, rhs, fl, dv = g.assemble_condense()
    x = torch.empty(g.nfaces * 3 * g.nf, dtype=torch.float64, device=g.device)
    for rep in range(3):  # eager, captured, replayed
        x.fill_(float("nan"))
        _lib.check(g.L.ddhdg_solve_condensed(g._ctx, tt.data_ptr(), rhs.data_ptr(), fl.data_ptr(), dv.data_ptr(),
                                             x.data_ptr(), 0, g._sp()), "solve_condensed")
        torch.cuda.synchronize()
        assert torch.isfinite(x).all()
        assert _backward_error(torch, g, tt, rhs, fl, dv, x) <= 1e-10
