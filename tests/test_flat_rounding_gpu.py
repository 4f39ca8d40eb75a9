"""Line sums of the slice forward projector (flat.cu) round once per plane: a plane's
sample is formed before it is added, so a large pair of voxels that cancels in one
plane leaves what the other planes added."""
import numpy as np
import pytest

import tomosipo_gb300 as ts

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [5, 40, 100, 140, 260])
@pytest.mark.parametrize("axis", [1, 2])  # the rays' axis: y or x
def test_cancelling_voxels_keep_the_sum(native_lib, nz, axis):
    """Rays along an axis, 3/4 of a voxel from one line of voxels and 1/4 from the
    next. Every plane but the last two adds 2^-10 (both voxels 2^-10); in the last
    two, voxels a = 2^21 and b = 1 - 3 a give 3/4 a + 1/4 b = 1/4. Products, samples and
    sums are exact in single precision, so the projection is (n - 2) 2^-10 + 1/2
    exactly; a running sum that takes a's product first (1.6e6, spacing 1/8) loses
    the small terms."""
    n, cols = 66, 3
    other = 3 - axis
    shape = [nz, 0, 0]
    shape[axis], shape[other] = n, 4
    vg = ts.volume(shape=shape, size=shape)
    ray, u = np.zeros((1, 3)), np.zeros((1, 3))
    ray[0, axis], u[0, other] = 1.0, 1.0
    # voxel centres of the short axis lie at -1.5, -0.5, 0.5, 1.5: the middle column
    # passes at -0.25
    pg = ts.parallel_vec(shape=(nz, cols), ray_dir=ray, det_pos=-0.25 * u,
                         det_v=np.array([[1.0, 0.0, 0.0]]), det_u=u)
    x = np.full(shape, 2.0 ** -10, np.float32)
    big = 2.0 ** 21
    line = [slice(None)] * 3
    for k in (n - 2, n - 1):
        line[axis] = k
        line[other] = 1
        x[tuple(line)] = big
        line[other] = 2
        x[tuple(line)] = 1.0 - 3.0 * big
    A = ts.operator(vg, pg)
    y = A(torch.from_numpy(x).cuda()).cpu().numpy()
    assert (y[:, 0, 1] == (n - 2) * 2.0 ** -10 + 0.5).all(), y[:, 0, 1]
