"""Scans whose line sums and profiles would take gigabytes (many angles): the slice
kernels work on pieces of the scan in bounded workspaces, and give what scans of fewer
angles give."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from tests.helpers import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_many_angles_of_few_rows(native_lib):
    """30000 angles x 300 columns over 64 slices: 2.3 GB of line sums, in two pieces
    (27904 angles and the rest). The forward projection equals those of the scan's
    halves, which need one piece each."""
    dev = torch.device("cuda", 0)
    n, rows, angles, cols = 8, 8, 30000, 300
    vg = ts.volume(shape=(64, n, n), size=(64, n, n))
    pg = ts.parallel(angles=np.linspace(0, np.pi, angles, endpoint=False), shape=(rows, cols),
                     size=(64, 2 * n))
    A = ts.operator(vg, pg)
    x = torch.rand(A.domain_shape, generator=torch.Generator().manual_seed(1)).to(dev)
    y = A(x)
    half = angles // 2
    halves = [ts.operator(vg, pg[:half]), ts.operator(vg, pg[half:])]
    assert torch.equal(y, torch.cat([B(x) for B in halves], dim=1))
    # the backprojection of four angles' values, around the pieces' border: the four
    # angles' own, up to the order of about 150 terms a voxel (37 columns an angle, each
    # rounding 2^-24 / sqrt(3): 3.4e-7 between two orders)
    some = [5, 27903, 27904, 29999]
    y4 = torch.rand((rows, 4, cols), generator=torch.Generator().manual_seed(2)).to(dev)
    y.zero_()
    y[:, some] = y4
    vec = pg.to_vec()
    pg4 = ts.parallel_vec(shape=vec.det_shape, **{
        k: np.asarray(getattr(vec, k))[some] for k in ("ray_dir", "det_pos", "det_v", "det_u")})
    back4 = ts.operator(vg, pg4).T(y4)
    back = A.T(y)
    assert rel_l2(back.cpu().numpy(), back4.cpu().numpy()) <= 2e-6
    acc = torch.ones_like(back)
    ts.operator(vg, pg, additive=True).T(y, out=acc)
    assert torch.equal(acc, torch.ones_like(back) + back)
    stats = A.projector.stats(dev.index)
    small = 1 << 20  # the volume's copies
    assert stats["fp_workspace_bytes"] <= (2 << 30) + small
    assert stats["bp_workspace_bytes"] <= (2 << 30) + small
    assert stats["fp_launches"] == stats["bp_matched_launches"] == 5
