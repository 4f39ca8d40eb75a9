"""The tuning's bp_kernel on parallel scans whose rays stay in one slice: 1 runs the
slice kernels, 0 the voxel-pair kernel (its two-row, four-row and row-loop paths),
for single calls, stacked items and batched SIRT; a workspace sized for the slice kernels
stays enough."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tomosipo_gb300 import _native
from tests.helpers import TOL_ADJOINT, TOL_ORACLE, adjoint_error, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def test_kernel_zero_is_the_voxel_pair_kernel(dev):
    """Angles of one pass: the slice kernels take three launches (profiles, windows,
    output), the voxel-pair kernel two (weights, one pass)."""
    vg = ts.volume(shape=(20, 12, 14), size=(20, 12, 14))
    A = ts.operator(vg, ts.parallel(angles=[-0.3, 0.0, 0.2], shape=(20, 20), size=(20, 20)))
    launches = {}
    for kernel in (1, 0):
        A.projector.set_tuning(dev.index, bp_kernel=kernel)
        launches[kernel] = A.projector.stats(dev.index)["bp_matched_launches"]
    assert launches == {1: 3, 0: 2}


# rows of the detector over 24 slices: coarser than the voxels, four rows a voxel, more
@pytest.mark.parametrize("rows", [17, 24, 36, 80])
def test_both_kernels(dev, rows):
    from tomosipo_gb300.sirt import BatchedSirt, sirt

    vg = ts.volume(shape=(24, 17, 21), size=(24, 17, 21))
    pg = ts.parallel(angles=11, shape=(rows, 30), size=(26, 30))
    A = ts.operator(vg, pg)
    g = torch.Generator().manual_seed(2)
    x = torch.rand((3,) + A.domain_shape, generator=g).to(dev)
    y = torch.rand((3,) + A.range_shape, generator=g).to(dev)
    ref = orc.bp_matched(vg, pg, y[0].cpu().numpy())
    Ax = A(x[0])
    fp_sizes, sizes = set(), []
    for kernel, path in ((1, 3), (0, 1)):
        A.projector.set_tuning(dev.index, bp_kernel=kernel)
        stats = A.projector.stats(dev.index)
        assert (stats["fp_kernel"], stats["bp_matched_kernel"]) == (1, path)
        fp_sizes.add(stats["fp_workspace_bytes"])
        sizes.append(stats["bp_workspace_bytes"])
        Aty = A.T(y[0])
        assert rel_l2(Aty.cpu().numpy(), ref) <= TOL_ORACLE
        assert adjoint_error(Ax.cpu().numpy(), y[0].cpu().numpy(), x[0].cpu().numpy(),
                             Aty.cpu().numpy()) <= TOL_ADJOINT
        assert torch.equal(A(x[0]), Ax)
        back = torch.empty_like(x)
        A.T._apply_batch(y, back)
        assert rel_l2(back[0].cpu().numpy(), Aty.cpu().numpy()) <= 1e-6
        b = BatchedSirt([(A, y[0]), (A, y[1])])
        b.run(2, graph=False)
        for k in range(2):
            assert torch.equal(b.x[k], sirt(A, y[k], 2))
        b.close()
    assert len(fp_sizes) == 1
    # (tuning 0 now) the workspace that tuning 1 asked for
    lib, h = _native.load(), A.projector.handle(dev.index)
    ws = torch.empty(max(sizes), dtype=torch.uint8, device=dev)
    out = torch.empty_like(x[0])
    stream = torch.cuda.current_stream(dev).cuda_stream
    for nbytes, rc in ((sizes[0], 0), (sizes[0] - 1, -3)):
        assert lib.tsgb_direct_bp(h, out.data_ptr(), y[0].data_ptr(), 0, 0, ws.data_ptr(), nbytes,
                                  stream) == rc
    assert rel_l2(out.cpu().numpy(), ref) <= TOL_ORACLE
    A.projector.set_tuning(dev.index, bp_kernel=1)
    if sizes[0] < 8 * (rows + 4) * 11 * 30:  # no row pairs fit: the slice kernels ran
        assert torch.equal(out, A.T(y[0]))
