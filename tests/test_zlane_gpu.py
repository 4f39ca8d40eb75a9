"""The z-lane matched backprojector at the sizes where its launch changes: the
voxels along z per lane (1 to 8, several ranges), ragged windows and planes,
detectors that end inside the volume's shadow (clamped rows), rows finer than
the voxels (the four-row and the general row sums, and scans that mix them with
coarser rows), and stacked items. Against the FP64 oracle at the parity
tolerance; stacked items equal each item alone."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tests.helpers import TOL_ORACLE, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def _scan(nz, ny, nx, rows, cols, height, angles=7):
    vg = ts.volume(shape=(nz, ny, nx), size=(nz / 32, ny / 32, nx / 32))
    pg = ts.cone(angles=np.linspace(0, 2 * np.pi, angles, endpoint=False) + 0.1,
                 shape=(rows, cols), size=(height * nz / 32, 1.5 * nx / 32),
                 src_orig_dist=3 + nz / 16, src_det_dist=3 + nz / 16)
    return vg, pg


def _check(dev, vg, pg):
    A = ts.operator(vg, pg)
    assert A.projector.get_tuning(dev.index)["bp_kernel"] == 1
    y = torch.rand(A.range_shape, generator=torch.Generator().manual_seed(5)).to(dev)
    ref = orc.bp_matched(vg, pg, y.cpu().numpy())
    assert rel_l2(A.T(y).cpu().numpy(), ref) <= TOL_ORACLE


@pytest.mark.parametrize("nz", [1, 31, 33, 65, 96, 127, 129, 161, 193, 225, 256, 257, 321, 515])
def test_z_extents(dev, nz):
    _check(dev, *_scan(nz, 9, 13, max(4, int(0.9 * nz)), 21, 1.3))


@pytest.mark.parametrize("ny, nx", [(1, 1), (3, 17), (17, 3), (8, 5), (34, 41)])
def test_windows_and_planes(dev, ny, nx):
    _check(dev, *_scan(40, ny, nx, 44, 2 * nx + 5, 1.3))


@pytest.mark.parametrize("nz", [20, 70, 140, 250])
@pytest.mark.parametrize("height, fine", [(0.5, 0.8), (1.4, 1.2), (1.2, 1.9), (1.2, 3.5), (0.6, 2.2)])
def test_rows(dev, nz, height, fine):
    """height: detector over volume; fine: detector rows per voxel of height."""
    _check(dev, *_scan(nz, 10, 12, max(3, int(height * nz * fine)), 19, height))


@pytest.mark.parametrize("nz", [12, 100, 230])
def test_stacked_items_equal_each_alone(dev, nz):
    vg, pg = _scan(nz, 11, 14, nz, 23, 1.3)
    A = ts.operator(vg, pg)
    B = ts.operator(vg, pg, additive=True)
    y = torch.rand((5,) + A.range_shape, generator=torch.Generator().manual_seed(6)).to(dev)
    out = torch.full((5,) + A.domain_shape, 2.0, device=dev)
    A.T._apply_batch(y, out)
    alone = torch.stack([A.T(v) for v in y])
    assert torch.equal(out, alone)
    B.T._apply_batch(y, out)
    assert torch.equal(out, alone + alone)
