"""Which bilinear backprojector runs: lanes along z with a scratch volume (three
launches), or one thread per 16 voxels along z from a quad copy (two). Both against the
FP64 oracle, and FDK's weights on both, where the choice changes: few and many angles,
heights that fill their lanes and heights that do not, rows finer than the voxels, and
slices that few threads cover."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import fdk_oracle
from oracle import oracle as orc
from tests.helpers import TOL_ORACLE, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _scan(nz, ny, nx, rows, angles, scan, cols=None):
    vg = ts.volume(shape=(nz, ny, nx), size=(nz / 64, ny / 64, nx / 64))
    t = np.linspace(0, 2 * np.pi, angles, endpoint=False) + 0.1
    shape, size = (rows, cols or max(nx, ny)), (1.1 * nz / 64, 1.4 * max(nx, ny) / 64)
    if scan == "parallel":
        return vg, ts.parallel(angles=t, shape=shape, size=size)
    far = 4 * max(nx, ny) / 64 + nz / 16
    return vg, ts.cone(angles=t, shape=shape, size=size, src_orig_dist=far, src_det_dist=far)


# name: nz, ny, nx, rows, angles; launches of the cone and the parallel scan
CASES = {
    "few_angles": ((96, 150, 160, 96, 2), 2, 2),
    "one_angle": ((128, 130, 150, 100, 1), 2, 2),
    "more_angles": ((128, 130, 150, 100, 60), 3, 3),
    "idle_lanes": ((40, 300, 310, 40, 40), 2, 3),
    "two_ranges_idle": ((176, 300, 300, 20, 16), 2, 3),
    "fine_rows": ((64, 150, 160, 400, 24), 2, 2),
    "few_threads": ((33, 20, 21, 30, 3), 3, 3),
    "thin": ((20, 190, 180, 20, 12), 2, 2),
}


@pytest.mark.parametrize("scan", ["cone", "parallel"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_both_paths(native_lib, name, scan):
    sizes, cone, parallel = CASES[name]
    vg, pg = _scan(*sizes, scan)
    A = ts.operator(vg, pg, backprojector="bilinear")
    launches = A.projector.stats(0)["bp_bilinear_launches"]
    assert launches == (cone if scan == "cone" else parallel)
    y = torch.rand(A.range_shape, generator=torch.Generator().manual_seed(5))
    ref = orc.bp_bilinear(vg, pg, y.numpy())
    x = A.T(y.cuda())
    assert rel_l2(x.cpu().numpy(), ref) <= TOL_ORACLE
    acc = x.clone()
    ts.operator(vg, pg, backprojector="bilinear", additive=True).T(y.cuda(), out=acc)
    assert rel_l2(acc.cpu().numpy(), 2 * ref) <= TOL_ORACLE


@pytest.mark.parametrize("sizes", [(40, 44, 40, 40, 3), (64, 130, 128, 40, 2), (40, 60, 64, 160, 5)])
def test_fdk(native_lib, sizes):
    from tomosipo_gb300.fdk import fdk_reconstruct

    vg, pg = _scan(*sizes, "cone", cols=48)
    rows, angles = sizes[3:]
    y = torch.rand((rows, angles, 48), generator=torch.Generator().manual_seed(7))
    ref = fdk_oracle.fdk(vg, pg, y.numpy())
    assert rel_l2(fdk_reconstruct(vg, pg, y.cuda()).cpu().numpy(), ref) <= TOL_ORACLE
