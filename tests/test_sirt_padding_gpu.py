"""Batched SIRT whose tuning changes between iterations, with detectors that end inside the
volume's shadow: voxels beyond them read the padding of the residual's layout."""
import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300.sirt import BatchedSirt, sirt

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scan", ["parallel", "cone"])
@pytest.mark.parametrize("rows", [6, 17])
def test_padding_after_a_change(native_lib, scan, rows):
    nz, n = 40, 20
    vg = ts.volume(shape=(nz, n, n), size=(nz, n, n))
    pg = (ts.parallel(angles=9, shape=(rows, 30), size=(0.6 * nz, 30)) if scan == "parallel" else
          ts.cone(angles=9, shape=(rows, 30), size=(0.6 * nz, 30), src_orig_dist=150, src_det_dist=150))
    A = ts.operator(vg, pg)
    y = torch.rand(A.range_shape, generator=torch.Generator().manual_seed(1)).cuda()
    b = BatchedSirt([(A, y)])
    R, C = b.R[0].clone(), b.C[0].clone()
    x = None
    for kernel in (1, 0, 1, 0):
        A.projector.set_tuning(0, bp_kernel=kernel)
        b.run(2, graph=False)
        x = sirt(A, y, 2, x_init=x, R=R, C=C)
        assert torch.equal(b.x[0], x), kernel
    b.close()
