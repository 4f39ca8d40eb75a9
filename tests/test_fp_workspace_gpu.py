"""A forward projection's workspace holds what it touches (parallel scans within one
slice: one volume copy and the line sums); batched SIRT's holds its backprojection too."""
import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300 import _native
from tomosipo_gb300.sirt import SirtJobState

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_a_projection_takes_its_own_need(native_lib):
    dev = torch.device("cuda", 0)
    nz, n, angles, cols = 40, 60, 12, 90
    A = ts.operator(ts.volume(shape=(nz, n, n), size=1),
                    ts.parallel(angles=angles, shape=(nz, cols), size=(1, 1.5)))
    x = torch.rand(A.domain_shape, device=dev)
    y = A(x)

    def up(floats):
        return (4 * floats + 255) // 256 * 256

    own = up((n + 4) * (n + 4) * nz) + up(angles * cols * nz)
    job = up(angles * cols * nz) + 2 * up(n * n * nz)  # profiles, a scratch volume per pass
    assert own < job
    nbytes = A.projector.workspace_bytes(dev.index, True)
    assert nbytes == own
    assert A.projector.stats(dev.index)["fp_workspace_bytes"] == job
    assert SirtJobState(A, y).ws.numel() * 4 == job
    # nothing is written past it
    lib, h = _native.load(), A.projector.handle(dev.index)
    ws = torch.full((nbytes + 4096,), 91, dtype=torch.uint8, device=dev)
    out = torch.empty_like(y)
    stream = torch.cuda.current_stream(dev).cuda_stream
    _native.check(lib.tsgb_direct_fp(h, x.data_ptr(), out.data_ptr(), 0, ws.data_ptr(), nbytes,
                                     stream), "tsgb_direct_fp")
    assert torch.equal(out, y) and bool((ws[nbytes:] == 91).all())
    assert lib.tsgb_direct_fp(h, x.data_ptr(), out.data_ptr(), 0, ws.data_ptr(), nbytes - 1,
                              stream) == -3
