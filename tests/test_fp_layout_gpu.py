"""The forward projector's default copy layout: single voxels where detector rows lie 4 to
28 voxels apart, pairs where they are nearer or farther; both give the same sinogram."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tests.helpers import TOL_ORACLE, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pitch, pairs", [(0.5, 1), (1.0, 1), (3.0, 1), (4.0, 0), (16.0, 0),
                                          (27.0, 0), (32.0, 1)])
def test_rows_apart(native_lib, pitch, pairs):
    n, rows = 14, max(2, int(120 / pitch))
    vg = ts.volume(shape=(120, n, n + 2), size=(120, n, n + 2))
    pg = ts.cone(angles=np.linspace(0.1, 6, 9), shape=(rows, 20), size=(rows * pitch, 24),
                 src_orig_dist=400, src_det_dist=400)
    A = ts.operator(vg, pg)
    assert A.projector.get_tuning(0)["fp_pair_layout"] == pairs
    x = torch.rand(A.domain_shape, generator=torch.Generator().manual_seed(4))
    y = A(x.cuda())
    assert rel_l2(y.cpu().numpy(), orc.fp(vg, pg, x.numpy())) <= TOL_ORACLE
    A.projector.set_tuning(0, fp_pair_layout=1 - pairs)
    assert torch.equal(A(x.cuda()), y)
