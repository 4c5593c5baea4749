"""Host-buffer calls whose chunks are whole waves of each form of the
condensation (3D and mixed register kernel, CTA-per-cell kernel with and
without drift columns, both modes): meshes of less than a wave, of a few and
of many ragged ones.  The outputs are the bits of the device-array calls."""

import pytest

from ddhdg_b200 import _lib
from ddhdg_b200.problem import Precision
from tests.test_gpu_condense_shapes import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,m,k,prec", [(1, 3, 2, Precision.fp64), (2, 60, 2, Precision.mixed),
                                          (2, 90, 1, Precision.mixed), (2, 23, 3, Precision.fp64),
                                          (2, 51, 3, Precision.fp64), (3, 13, 1, Precision.fp64),
                                          (3, 13, 1, Precision.mixed), (3, 6, 2, Precision.fp64)])
def test_chunks_of_every_form_give_the_device_bits(dim, m, k, prec):
    torch, g = _solver(dim, m, k, prec)
    cell, trace = g.cell_state.cpu().pin_memory(), g.trace_state.cpu().pin_memory()
    upd = (1e-3 * torch.randn(g.nfaces * 3 * g.nf, dtype=torch.float64,
                              generator=torch.Generator().manual_seed(1))).pin_memory()
    for thermo in (False, True):
        ref = g.assemble_condense(thermo)
        du = g.reconstruct(upd.numpy().reshape(g.nfaces, 3, g.nf), thermo=thermo).clone()
        out = [torch.full_like(ref[0], float("nan")), torch.full_like(ref[1], float("nan")), torch.zeros_like(ref[2]),
               torch.full_like(ref[3], float("nan"))]
        host = torch.full((du.numel(),), float("nan"), dtype=torch.float64).pin_memory()
        _lib.check(g.L.ddhdg_assemble_condense_host(g._ctx, cell.data_ptr(), trace.data_ptr(), int(thermo),
                                                    *[t.data_ptr() for t in out], g._sp()), "assemble_condense_host")
        _lib.check(g.L.ddhdg_reconstruct_host(g._ctx, upd.data_ptr(), int(thermo), host.data_ptr(), g._sp()),
                   "reconstruct_host")
        torch.cuda.synchronize()
        for x, y in zip(ref, out):
            assert torch.equal(x, y)
        assert torch.equal(du.cpu().reshape(-1), host)
