"""The pivots' reciprocal (hdg_reciprocal.cuh) over the whole range of FP64,
and trace systems whose pivots are subnormal with a finite reciprocal.

Bound: the approximation's relative error of at most 2^-20 is squared by each
of two Newton steps, so that before the last rounding it is below 2^-79; the
rounding is half an ulp.  Subnormal results are rounded twice: one ulp."""

import numpy as np
import pytest

from ddhdg_b200 import _lib
from tests import device_probe
from tests.test_gpu_trace_solve import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scaled", [0, 1])
def test_reciprocal_over_all_exponents(tmp_path, scaled):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    L = device_probe.load(tmp_path)
    rng = np.random.default_rng(3)
    e = np.repeat(np.arange(-1074, 1024), 64)
    with np.errstate(over="ignore"):
        x = np.ldexp(rng.uniform(1, 2, e.size), e) * rng.choice([-1., 1.], e.size)
    x = np.concatenate([x, np.ldexp(1., np.arange(-1074, 1024)), np.nextafter(np.ldexp(1., np.arange(-1073, 1024)), 0),
                        [np.finfo(float).max, -np.finfo(float).max, np.finfo(float).tiny]])
    x = x[np.isfinite(x) & (x != 0)]
    if scaled:  # the range of the scaled form
        x = x[np.abs(x) < 2.0 ** 960]
    sp = np.array([0., -0., np.inf, -np.inf, np.nan])
    allx = np.ascontiguousarray(np.concatenate([x, sp]))
    r = np.empty_like(allx)
    assert L.probe_reciprocal(device_probe.dptr(allx), device_probe.dptr(r), allx.size, scaled) == 0
    z = r[x.size:]
    assert (z[:2] == 0).all() and np.isnan(z[4])
    # the scaled form leaves infinities to its caller's check
    assert np.isnan(z[2:4]).all() if scaled else (z[2:4] == 0).all()
    r = r[:x.size]
    exact = 1 / x.astype(np.longdouble)
    with np.errstate(over="ignore", divide="ignore"):
        d = 1 / x
    over = np.isinf(d)
    assert (r[over] == d[over]).all()
    sub = ~over & (np.abs(d) < np.finfo(float).tiny)
    ulps = np.abs(r.astype(np.longdouble)[~over] - exact[~over]) / np.spacing(np.abs(d[~over])).astype(np.longdouble)
    assert (ulps[~sub[~over]] <= 0.5 + 2.0 ** -25).all()
    assert (ulps[sub[~over]] <= 1).all()


# one cell without Dirichlet rows: 6, 24, 48 and 162 eliminated dofs (the
# one-CTA kernel and one or more panels).  The last row is the first one plus
# s on the diagonal, so that s = 2^-1023 is the last pivot: x = 1 there,
# exactly (all products are powers of two).
@pytest.mark.parametrize("dim,k", [(1, 1), (2, 1), (2, 3), (3, 2)])
def test_subnormal_pivots_are_accepted(dim, k):
    torch, g = _setup(dim, 1, k)
    n = g.nfaces * 3 * g.nf
    s = 2.0 ** -1023
    tt = torch.eye(n, dtype=torch.float64)
    tt[n - 1, 0], tt[n - 1, n - 1] = 1.0, s
    rhs = torch.ones(n, dtype=torch.float64)
    rhs[0], rhs[n - 1] = 0.0, s
    want = torch.ones(n, dtype=torch.float64)
    want[0] = 0.0
    tt, rhs = tt.to(g.device), rhs.to(g.device)
    fl = torch.zeros(n, dtype=torch.int32, device=g.device)
    dv = torch.zeros(n, dtype=torch.float64, device=g.device)
    x = torch.full((n,), float("nan"), dtype=torch.float64, device=g.device)
    _lib.check(g.L.ddhdg_solve_condensed(g._ctx, tt.data_ptr(), rhs.data_ptr(), fl.data_ptr(), dv.data_ptr(),
                                         x.data_ptr(), 0, g._sp()), "solve_condensed")
    torch.cuda.synchronize()
    # x is in global dof order; the cell's faces are numbered by axis, as
    # its local ones
    assert torch.equal(x.cpu(), want)
