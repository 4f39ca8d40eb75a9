"""Matched backprojection on a supersampled detector (its kernels read the spread
sinogram from the caller's): every kernel that reads it, at factors that do not
divide the tiles' sizes, against the FP64 oracle, set and added."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tests.helpers import TOL_ORACLE, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _cone(angles, shape, size):
    return ts.cone(angles=angles, shape=shape, size=size, src_orig_dist=4.0, src_det_dist=6.0)


CASES = {
    # z-lane kernel, rows finer than the voxels
    "zlane": (ts.volume(shape=(33, 17, 21), size=(1, 0.6, 0.7)),
              _cone(5, (34, 23), (1.7, 1.3)), 3),
    # volume thin along z and wide: voxel-pair kernel
    "voxel_pair": (ts.volume(shape=(3, 190, 187), size=(0.02, 1, 1)),
                   _cone(3, (3, 203), (0.05, 2.2)), 2),
    # rays within one slice, rows coarser than the voxels and finer
    "flat_coarse": (ts.volume(shape=(37, 19, 18), size=1),
                    ts.parallel(angles=6, shape=(11, 35), size=(1.1, 1.5)), 2),
    "flat_fine": (ts.volume(shape=(9, 19, 18), size=1),
                  ts.parallel(angles=6, shape=(11, 35), size=(1.1, 1.5)), 5),
    # tilted detector
    "tilted": (ts.volume(shape=(17, 16, 15), size=1),
               ts.rotate(pos=0, axis=(0.2, 1.0, 0.1), angles=0.3)
               * _cone(4, (13, 19), (1.9, 2.1)).to_vec(), 4),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_supersampled_backprojection(name, native_lib):
    vg, pg, d = CASES[name]
    A = ts.operator(vg, pg, detector_supersampling=d)
    y = np.random.default_rng(3).standard_normal(A.range_shape).astype(np.float32)
    ref = orc.bp_matched(vg, pg, y, det_ss=d)
    yt = torch.from_numpy(y).cuda()
    x = A.T(yt)
    assert rel_l2(x.cpu().numpy(), ref) <= TOL_ORACLE
    out = x.clone()
    ts.operator(vg, pg, detector_supersampling=d, additive=True).T(yt, out=out)
    assert rel_l2(out.cpu().numpy(), 2 * ref) <= TOL_ORACLE
