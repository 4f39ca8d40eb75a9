"""Bilinear and FDK backprojection with a workspace that starts on 8 bytes but not on 16:
sizes that would read 16-byte quads from it (few angles; thin, wide volumes) and sizes
that read pairs give what an aligned workspace gives."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300 import _native
from tests.helpers import TOL_ORACLE, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scan", ["cone", "parallel"])
@pytest.mark.parametrize("shape, angles, launches", [((128, 70, 65), 1, 2), ((9, 190, 185), 3, 2),
                                                     ((40, 20, 24), 8, 3)])
def test_workspace_on_eight_bytes(native_lib, scan, shape, angles, launches):
    nz, ny, nx = shape
    vg = ts.volume(shape=shape, size=(nz / 32, ny / 32, nx / 32))
    t = np.linspace(0.1, 6, angles)
    det, size = (nz + 2, nx + 30), (1.2 * nz / 32, 1.5 * nx / 32)
    pg = (ts.parallel(angles=t, shape=det, size=size) if scan == "parallel" else
          ts.cone(angles=t, shape=det, size=size, src_orig_dist=nz / 8 + 9, src_det_dist=nz / 8 + 10))
    A = ts.operator(vg, pg, backprojector="bilinear")
    assert A.projector.stats(0)["bp_bilinear_launches"] == launches
    lib, h = _native.load(), A.projector.handle(0)
    y = torch.rand(A.range_shape, generator=torch.Generator().manual_seed(2)).cuda()
    w = torch.rand(angles, generator=torch.Generator().manual_seed(3)).cuda()
    need = lib.tsgb_bp_workspace_bytes(h, 1)
    ws = torch.empty(need + 8, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    out = {}
    for offset in (0, 8):
        x, q = torch.ones(shape, device="cuda"), torch.ones(shape, device="cuda")
        at = ws.data_ptr() + offset
        _native.check(lib.tsgb_direct_bp(h, x.data_ptr(), y.data_ptr(), 1, 1, at, need, stream), "bp")
        if scan == "cone":
            _native.check(lib.tsgb_fdk_backproject(h, q.data_ptr(), y.data_ptr(), w.data_ptr(), 0,
                                                   at, need, stream), "fdk")
        out[offset] = x.cpu().numpy(), q.cpu().numpy()
    for got, want in zip(out[8], out[0]):
        assert rel_l2(got, want) <= TOL_ORACLE
