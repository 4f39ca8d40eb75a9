"""Parallel scans just outside the slice kernels' condition (one ray leaves its slice by
1e-9 of a voxel): the ray kernel under its schedules and copy layouts, and the voxel-pair
and z-lane backprojectors with rows as far apart as the voxels, finer (their four-row
paths) and much finer (their row loops). The forms of tests that the slice kernels took
over."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tests.helpers import TOL_ADJOINT, TOL_ORACLE, adjoint_error, rel_l2
from tests.test_tuning_gpu import BP_TUNINGS, TUNINGS

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _leaving(pg):
    v = pg.to_vec()
    ray = np.array(v.ray_dir, dtype=np.float64)
    ray[len(ray) // 2, 0] = 1e-9
    return ts.parallel_vec(shape=v.det_shape, ray_dir=ray, det_pos=v.det_pos, det_v=v.det_v,
                           det_u=v.det_u)


CASES = {
    "ragged": (ts.volume(shape=(40, 33, 47), size=(1.0, 0.9, 1.2)),
               ts.parallel(angles=31, shape=(70, 53), size=(1.6, 1.9))),
    "fine_rows": (ts.volume(shape=24, size=1), ts.parallel(angles=12, shape=(80, 36), size=(1.2, 1.5))),
    "rows_finer_than_voxels": (ts.volume(shape=24, size=1),
                               ts.parallel(angles=12, shape=(36, 36), size=(1.0, 1.5))),
    "aniso": (ts.volume(shape=(20, 28, 36), size=(0.7, 1.1, 1.3), pos=(0.05, -0.1, 0.2)),
              ts.parallel(angles=np.linspace(0.1, 3.0, 13), shape=(17, 29), size=(1.2, 2.1))),
    "45deg": (ts.volume(shape=32, size=1),
              ts.parallel(angles=[np.pi / 4, 3 * np.pi / 4, 0.0], shape=(32, 48), size=(1, 1.5))),
    "small_detector": (ts.volume(shape=32, size=1),
                       ts.parallel(angles=9, shape=(8, 8), size=(0.3, 0.3))),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_schedules_and_backprojectors(native_lib, name):
    dev = torch.device("cuda", 0)
    vg, pg = CASES[name]
    pg = _leaving(pg)
    A = ts.operator(vg, pg)
    g = torch.Generator().manual_seed(3)
    x = torch.rand(A.domain_shape, generator=g)
    y = torch.rand(A.range_shape, generator=g)
    assert A.projector.stats(0)["fp_kernel"] == 0
    Ax = A(x.to(dev))
    assert rel_l2(Ax.cpu().numpy(), orc.fp(vg, pg, x.numpy())) <= TOL_ORACLE
    default = A.projector.get_tuning(0)
    for t in TUNINGS:
        A.projector.set_tuning(0, **t)
        assert torch.equal(A(x.to(dev)), Ax), t
    A.projector.set_tuning(0, **default)
    ref = orc.bp_matched(vg, pg, y.numpy())
    for t in BP_TUNINGS:
        A.projector.set_tuning(0, **t)
        assert A.projector.stats(0)["bp_matched_kernel"] == 1 + t["bp_kernel"]
        Aty = A.T(y.to(dev)).cpu().numpy()
        assert rel_l2(Aty, ref) <= TOL_ORACLE, t
        assert adjoint_error(Ax.cpu().numpy(), y.numpy(), x.numpy(), Aty) <= TOL_ADJOINT, t
