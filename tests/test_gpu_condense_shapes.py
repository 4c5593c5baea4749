"""Condensation launches at the sizes where their shape changes: the register
kernel's wide form above eight cells per SM (1184 cells on 148 SMs), fewer
cells than SMs, and host-buffer chunks in whole waves.  The per-cell
arithmetic is the same in every launch shape, so the outputs are bitwise those
of the batched launch and of the host-buffer calls."""

import numpy as np
import pytest

from ddhdg_b200.problem import Precision
from tests import cases

pytestmark = pytest.mark.gpu


def _solver(dim, m, k, prec=Precision.fp64, seed=5):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from ddhdg_b200 import _lib
    from ddhdg_b200.solver import NPSolver

    pb, prm, adim = cases.diode(dim=dim, m=m, k=k, precision=prec)
    g = NPSolver(pb, prm, adim)
    g.compute_local_charge_neutrality()
    for c in (1, 2):
        _lib.check(g.L.ddhdg_project_density(g._ctx, c, 0.0, g.cell_state.data_ptr(), g.trace_state.data_ptr(),
                                             g._sp()), "project_density")
    rng = np.random.default_rng(seed)
    cell, trace = g.get_cell_state(), g.get_trace_state()
    g.set_state(cell * (1 + 1e-3 * rng.standard_normal(cell.shape)),
                trace * (1 + 1e-3 * rng.standard_normal(trace.shape)))
    return torch, g


@pytest.mark.parametrize("dim,m,k,prec", [(1, 1, 3, Precision.fp64), (1, 147, 1, Precision.fp64),
                                          (1, 1184, 2, Precision.fp64), (1, 1185, 2, Precision.fp64),
                                          (1, 2400, 3, Precision.fp64), (2, 34, 1, Precision.fp64),
                                          (2, 35, 1, Precision.fp64), (2, 35, 1, Precision.mixed),
                                          (2, 36, 2, Precision.fp64), (2, 13, 3, Precision.fp64),
                                          (3, 3, 2, Precision.fp64), (3, 11, 1, Precision.fp64)])
def test_launch_shapes_give_the_batched_bits(dim, m, k, prec):
    torch, g = _solver(dim, m, k, prec)
    from ddhdg_b200.batch import CondenseBatch

    for thermo in (False, True):
        ref = g.assemble_condense(thermo)
        assert torch.isfinite(ref[0]).all()
        b = CondenseBatch([g], thermo=thermo)
        b.condense()
        for x, y in zip(ref, (b.tt[0], b.rhs[0], b.dflag[0], b.dval[0])):
            assert torch.equal(x, y.view(x.shape))
        b.close()


@pytest.mark.parametrize("dim,m,k", [(2, 30, 1), (2, 80, 1), (2, 75, 2), (1, 5000, 3)])
def test_host_chunks_give_the_device_bits(dim, m, k):
    torch, g = _solver(dim, m, k)
    from ddhdg_b200 import _lib

    tt, rhs, fl, dv = g.assemble_condense()
    out = [torch.full_like(tt, float("nan")), torch.full_like(rhs, float("nan")), torch.zeros_like(fl),
           torch.full_like(dv, float("nan"))]
    cell, trace = g.cell_state.cpu().pin_memory(), g.trace_state.cpu().pin_memory()
    _lib.check(g.L.ddhdg_assemble_condense_host(g._ctx, cell.data_ptr(), trace.data_ptr(), 0,
                                                *[t.data_ptr() for t in out], g._sp()), "assemble_condense_host")
    torch.cuda.synchronize()
    for x, y in zip((tt, rhs, fl, dv), out):
        assert torch.equal(x, y)
