"""Batched SIRT whose jobs' tuning changes between iterations: each backprojector reads
the residual in a layout of its own, whose padding must be zero. Equal to the plain loop
under the same tunings."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300.sirt import BatchedSirt, sirt

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scan", ["parallel", "cone"])
@pytest.mark.parametrize("jobs, shape", [(1, (20, 24, 22)), (3, (20, 24, 22)), (3, (3, 190, 185))])
def test_kernels_in_turn(native_lib, scan, jobs, shape):
    nz, ny, nx = shape
    vg = ts.volume(shape=shape, size=(nz / 24, ny / 24, nx / 24))
    det, size = (nz + 4, int(1.3 * nx)), (1.5 * nz / 24, 1.6 * nx / 24)
    pg = (ts.parallel(angles=7, shape=det, size=size) if scan == "parallel" else
          ts.cone(angles=7, shape=det, size=size, src_orig_dist=5 * nx / 24, src_det_dist=5 * nx / 24))
    ops = [ts.operator(vg, pg) for _ in range(jobs)]
    g = torch.Generator().manual_seed(1)
    ys = [torch.rand(A.range_shape, generator=g).cuda() for A in ops]
    b = BatchedSirt(list(zip(ops, ys)))
    first = ops[0].projector.get_tuning(0)["bp_kernel"]
    xs = [None] * jobs
    R = [(r.clone(), c.clone()) for r, c in zip(b.R, b.C)]
    for kernel in (first, 1 - first, first, 1 - first):
        for A in ops:
            A.projector.set_tuning(0, bp_kernel=kernel)
        b.run(2, graph=False)
        for k, A in enumerate(ops):
            xs[k] = sirt(A, ys[k], 2, x_init=xs[k], R=R[k][0], C=R[k][1])
            assert torch.equal(b.x[k], xs[k]), (kernel, k)
    b.close()
