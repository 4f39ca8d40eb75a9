"""Workspaces of the C entry points that start on 8 bytes but not on 16: the kernels
that would read them 16 bytes at a time (parallel scans within one slice, stacked
items of the z-lane backprojector) give the results of an aligned workspace."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300 import _native
from tests.helpers import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def _calls(A, dev, n, offset):
    """Both projections of n stacked items with the workspace offset bytes from an
    allocation's start."""
    lib, h = _native.load(), A.projector.handle(dev.index)
    g = torch.Generator().manual_seed(7)
    x = torch.rand((n,) + A.domain_shape, generator=g).to(dev)
    y = torch.rand((n,) + A.range_shape, generator=g).to(dev)
    Ax, Aty = torch.empty_like(y), torch.empty_like(x)
    stream = torch.cuda.current_stream(dev).cuda_stream
    for forward in (True, False):
        need = (lib.tsgb_fp_batch_workspace_bytes(h, n) if forward
                else lib.tsgb_bp_batch_workspace_bytes(h, n, 0))
        ws = torch.empty(need + offset, dtype=torch.uint8, device=dev)
        at = ws.data_ptr() + offset
        assert ws.data_ptr() % 256 == 0
        if forward:
            rc = lib.tsgb_direct_fp_batch(h, x.data_ptr(), Ax.data_ptr(), n, 0, at, need, stream)
        else:
            rc = lib.tsgb_direct_bp_batch(h, Aty.data_ptr(), y.data_ptr(), n, 0, 0, at, need, stream)
        _native.check(rc, "batch")
        torch.cuda.synchronize()
    return Ax, Aty


@pytest.mark.parametrize("scan", ["parallel", "cone"])
@pytest.mark.parametrize("nz", [20, 61, 100, 140, 260])
@pytest.mark.parametrize("n", [1, 3])
def test_workspace_on_eight_bytes(dev, scan, nz, n):
    vg = ts.volume(shape=(nz, 14, 17), size=(nz / 16, 14 / 16, 17 / 16))
    shape, size = (nz + 3, 25), (1.1 * nz / 16, 1.6)
    pg = (ts.parallel(angles=np.linspace(0.1, 3, 12), shape=shape, size=size) if scan == "parallel"
          else ts.cone(angles=12, shape=shape, size=size, src_orig_dist=20, src_det_dist=21))
    A = ts.operator(vg, pg)
    want = _calls(A, dev, n, 0)
    got = _calls(A, dev, n, 8)
    assert torch.equal(got[0], want[0])
    # (another split of the angles: the same sums in another order)
    assert rel_l2(got[1].cpu().numpy(), want[1].cpu().numpy()) <= 1e-6
