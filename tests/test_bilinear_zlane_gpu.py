"""The bilinear backprojector's z-lane kernel at the sizes where its launch
changes (voxels along z per lane, several ranges, ragged blocks of voxel columns,
more angles than one list, thin wide volumes that keep one thread per column),
with detectors that end inside the volume's shadow (clamped rows, columns off the
detector), against the FP64 oracle, setting and adding; and FDK against the FP64
FDK at several z extents."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import fdk_oracle
from oracle import oracle as orc
from tests.helpers import TOL_ORACLE, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def _scan(nz, ny, nx, rows, cols, scan="cone", height=1.3, width=1.6, angles=11):
    vg = ts.volume(shape=(nz, ny, nx), size=(nz / 32, ny / 32, nx / 32))
    size = (height * nz / 32, width * max(nx, ny) / 32)
    t = np.linspace(0, 2 * np.pi, angles, endpoint=False) + 0.1
    if scan == "parallel":
        return vg, ts.parallel(angles=t, shape=(rows, cols), size=size)
    far = 3 + nz / 16
    return vg, ts.cone(angles=t, shape=(rows, cols), size=size, src_orig_dist=far, src_det_dist=far)


def _check(dev, vg, pg):
    A = ts.operator(vg, pg, backprojector="bilinear")
    y = torch.rand(A.range_shape, generator=torch.Generator().manual_seed(5)).to(dev)
    ref = orc.bp_bilinear(vg, pg, y.cpu().numpy())
    x = A.T(y)
    assert rel_l2(x.cpu().numpy(), ref) <= TOL_ORACLE
    B = ts.operator(vg, pg, backprojector="bilinear", additive=True)
    acc = x.clone()
    B.T(y, out=acc)
    assert rel_l2(acc.cpu().numpy(), 2 * ref) <= TOL_ORACLE


@pytest.mark.parametrize("scan", ["cone", "parallel"])
@pytest.mark.parametrize("nz", [1, 31, 33, 65, 97, 129, 160, 161, 193, 321])
def test_z_extents(dev, nz, scan):
    _check(dev, *_scan(nz, 6, 9, max(2, nz), 17, scan))


@pytest.mark.parametrize("nz, ny, nx, angles", [(20, 1, 1, 3), (20, 5, 101, 40), (20, 101, 3, 33),
                                                (12, 184, 190, 70), (33, 184, 190, 5)])
def test_blocks_and_lists(dev, nz, ny, nx, angles):
    _check(dev, *_scan(nz, ny, nx, nz + 3, 2 * max(nx, ny), angles=angles))


@pytest.mark.parametrize("height, width", [(0.4, 1.6), (1.4, 0.5), (0.3, 0.3), (2.5, 2.5)])
@pytest.mark.parametrize("scan", ["cone", "parallel"])
def test_small_and_large_detectors(dev, height, width, scan):
    _check(dev, *_scan(70, 14, 16, 40, 25, scan, height, width))


@pytest.mark.parametrize("nz", [5, 40, 170])
def test_fdk(dev, nz):
    from tomosipo_gb300.fdk import fdk_reconstruct

    vg, pg = _scan(nz, 12, 14, nz, 24)
    y = torch.rand((nz, 11, 24), generator=torch.Generator().manual_seed(7)).to(dev)
    ref = fdk_oracle.fdk(vg, pg, y.cpu().numpy())
    assert rel_l2(fdk_reconstruct(vg, pg, y).cpu().numpy(), ref) <= TOL_ORACLE
