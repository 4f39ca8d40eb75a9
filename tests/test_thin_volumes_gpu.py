"""Volumes thin along z and wide keep the voxel-pair backprojector: where the default
changes, and that kernel against the FP64 oracle, for cones and parallel scans, plain
and with a supersampled detector, and in batched SIRT."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tests.helpers import TOL_ORACLE, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _scan(scan, nz, ny, nx, rows, cols, angles=3):
    vg = ts.volume(shape=(nz, ny, nx), size=(nz / 64, ny / 64, nx / 64))
    size = (1.2 * nz / 64, 1.5 * max(nx, ny) / 64)
    if scan == "parallel":
        return vg, ts.parallel(angles=np.linspace(0.1, 3, angles), shape=(rows, cols), size=size)
    far = 4 * max(nx, ny) / 64
    return vg, ts.cone(angles=np.linspace(0.1, 6, angles), shape=(rows, cols), size=size,
                       src_orig_dist=far, src_det_dist=far)


@pytest.mark.parametrize("scan, nz, n, kernel", [
    ("cone", 48, 181, 2), ("cone", 16, 182, 1), ("cone", 48, 182, 1), ("cone", 49, 400, 2),
    ("parallel", 16, 181, 3), ("parallel", 16, 182, 1), ("parallel", 17, 256, 3),
    ("parallel", 32, 500, 3), ("parallel", 32, 512, 1), ("parallel", 33, 512, 3)])
def test_where_the_default_changes(native_lib, scan, nz, n, kernel):
    A = ts.operator(*_scan(scan, nz, n, n, 4, 8))
    assert A.projector.stats(0)["bp_matched_kernel"] == kernel


@pytest.mark.parametrize("ss", [1, 2])
@pytest.mark.parametrize("scan", ["cone", "parallel"])
def test_voxel_pair_kernel(native_lib, scan, ss):
    from tomosipo_gb300.sirt import BatchedSirt, sirt

    vg, pg = _scan(scan, 3, 262, 255, 3, 270)
    A = ts.operator(vg, pg, detector_supersampling=ss)
    assert A.projector.stats(0)["bp_matched_kernel"] == 1
    y = torch.rand(A.range_shape, generator=torch.Generator().manual_seed(3))
    ref = orc.bp_matched(vg, pg, y.numpy(), det_ss=ss)
    x = A.T(y.cuda())
    assert rel_l2(x.cpu().numpy(), ref) <= TOL_ORACLE
    out = x.clone()
    ts.operator(vg, pg, detector_supersampling=ss, additive=True).T(y.cuda(), out=out)
    assert rel_l2(out.cpu().numpy(), 2 * ref) <= TOL_ORACLE
    if ss == 1:
        b = BatchedSirt([(A, y.cuda()), (A, 2 * y.cuda())])
        b.run(2, graph=False)
        assert torch.equal(b.x[0], sirt(A, y.cuda(), 2))
        assert torch.equal(b.x[1], sirt(A, 2 * y.cuda(), 2))
        b.close()
