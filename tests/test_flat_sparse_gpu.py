"""Parallel scans within slices whose few detector rows lie far apart: the forward
projection follows their rays, the backprojection runs slice by slice. Against the FP64
oracle; stacked items, additive calls, angle ranges and batched SIRT (rays writing the
residual the slice kernels read) equal the plain calls."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tests.helpers import TOL_ADJOINT, TOL_ORACLE, adjoint_error, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _scan(nz, rows, angles, n=13):
    vg = ts.volume(shape=(nz, n, n + 4), size=(nz, n, n + 4))
    return vg, ts.parallel(angles=angles, shape=(rows, 2 * n), size=(nz, 2 * n))


def test_the_forward_kernel_follows_the_rows(native_lib):
    """Angles of one axis permutation: rays take two launches (copy, rays), line sums
    three (copy, lines, rows)."""
    for nz, rows, launches in ((200, 8, 2), (200, 40, 2), (200, 200, 3), (200, 100, 3), (60, 3, 3),
                               (400, 9, 2), (512, 32, 3)):
        A = ts.operator(*_scan(nz, rows, [-0.3, 0.0, 0.25]))
        assert A.projector.stats(0)["fp_launches"] == launches, (nz, rows)


@pytest.mark.parametrize("nz, rows", [(200, 8), (200, 41), (300, 2), (131, 17)])
def test_projections(native_lib, nz, rows):
    from tomosipo_gb300.sirt import BatchedSirt, sirt

    vg, pg = _scan(nz, rows, np.linspace(0.1, 3.1, 11))
    A = ts.operator(vg, pg)
    stats = A.projector.stats(0)
    assert (stats["fp_kernel"], stats["bp_matched_kernel"]) == (0, 3)
    g = torch.Generator().manual_seed(5)
    x = torch.rand((3,) + A.domain_shape, generator=g).cuda()
    w = torch.rand(A.range_shape, generator=g).cuda()
    y = torch.empty((3,) + A.range_shape, device="cuda")
    A._apply_batch(x, y)
    assert torch.equal(y, torch.stack([A(v) for v in x]))
    assert rel_l2(y[0].cpu().numpy(), orc.fp(vg, pg, x[0].cpu().numpy())) <= TOL_ORACLE
    Atw = A.T(w)
    assert rel_l2(Atw.cpu().numpy(), orc.bp_matched(vg, pg, w.cpu().numpy())) <= TOL_ORACLE
    assert adjoint_error(y[0].cpu().numpy(), w.cpu().numpy(), x[0].cpu().numpy(),
                         Atw.cpu().numpy()) <= TOL_ADJOINT
    out = torch.ones_like(w)
    ts.operator(vg, pg, additive=True)(x[0], out=out)
    assert torch.equal(out, torch.ones_like(w) + y[0])
    b = BatchedSirt([(A, y[0]), (A, y[1])])
    b.run(3, graph=False)
    for k in range(2):
        assert torch.equal(b.x[k], sirt(A, y[k], 3))
    b.close()
