"""Parallel scans whose detector covers a part of the volume along z: the slice kernels
(flat.cu) work on the slices the rows interpolate and no others. Detectors at the
bottom, in the middle, at the top and beside the volume, moving along z, one row;
against the FP64 oracle, with workspaces sized by those slices; additive calls, angle
ranges, stacked items and batched SIRT."""
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


def _scan(nz, rows, pitch, first, angles=7, move=0.0, n=12):
    """Voxels of size 1; detector rows of height pitch, the first row's centre at voxel
    `first` along z (0: the first slice's centre), the detector rising by `move` voxels
    over the scan."""
    vg = ts.volume(shape=(nz, n, n + 3), size=(nz, n, n + 3))
    pg = ts.parallel(angles=np.linspace(0.1, 3.0, angles), shape=(rows, 2 * n),
                     size=(rows * pitch, 2 * n)).to_vec()
    z = np.zeros((angles, 3))
    z[:, 0] = first + (rows - 1) / 2 * pitch - (nz - 1) / 2 + np.linspace(0, move, angles)
    return vg, ts.parallel_vec(shape=pg.det_shape, ray_dir=pg.ray_dir,
                               det_pos=np.asarray(pg.det_pos) + z, det_v=pg.det_v, det_u=pg.det_u)


CASES = {  # nz, rows, pitch, first, move
    "bottom": (300, 20, 1.0, -3.3, 0.0),
    "bottom_edge": (200, 2, 1.0, -0.5, 0.0),
    "middle": (300, 40, 1.1, 101.7, 0.0),
    "middle_whole_slices": (300, 64, 1.0, 100.0, 0.0),
    "sixty_two_slices": (200, 61, 1.0, 64.0, 0.0),
    "fine_rows": (260, 90, 0.3, 200.2, 0.0),
    "coarse_rows": (400, 9, 6.5, 150.4, 0.0),
    "top": (300, 20, 1.0, 290.2, 0.0),
    "top_edge": (200, 1, 1.0, 199.5, 0.0),
    "one_row": (513, 1, 1.0, 255.5, 0.0),
    "one_coarse_row": (513, 1, 40.0, 17.0, 0.0),
    "below": (150, 10, 1.0, -40.0, 0.0),
    "above": (150, 10, 1.0, 170.0, 0.0),
    "rising": (400, 12, 1.0, 50.0, 150.0),
    "rising_out": (150, 12, 1.0, 100.0, 90.0),
}


def _slices(nz, rows, pitch, first, move):
    """An upper bound of the slices the rows interpolate, with one to spare on each
    side, in steps of 64."""
    lo, hi = np.clip([first - 1, first + (rows - 1) * pitch + move + 1], 0, nz - 1)
    return min(nz, (int(np.ceil(hi) - np.floor(lo)) + 1 + 63) // 64 * 64)


@pytest.mark.parametrize("name", sorted(CASES))
def test_projections_and_workspaces(dev, name):
    nz, rows, pitch, first, move = CASES[name]
    vg, pg = _scan(nz, rows, pitch, first, move=move)
    A = ts.operator(vg, pg)
    gen = torch.Generator().manual_seed(5)
    x = torch.rand(A.domain_shape, generator=gen).to(dev)
    y = torch.rand(A.range_shape, generator=gen).to(dev)
    Ax, Aty = A(x), A.T(y)
    ref = orc.fp(vg, pg, x.cpu().numpy())
    assert rel_l2(Ax.cpu().numpy(), ref) <= TOL_ORACLE
    assert rel_l2(Aty.cpu().numpy(), orc.bp_matched(vg, pg, y.cpu().numpy())) <= TOL_ORACLE
    if np.any(ref):
        assert adjoint_error(Ax.cpu().numpy(), y.cpu().numpy(), x.cpu().numpy(),
                             Aty.cpu().numpy()) <= TOL_ADJOINT
    else:
        assert not Ax.any() and not Aty.any()
    B = ts.operator(vg, pg, additive=True)
    out = torch.ones_like(y)
    B(x, out=out)
    assert torch.equal(out, torch.ones_like(y) + Ax)
    acc = torch.ones_like(x)
    B.T(y, out=acc)
    assert torch.equal(acc, torch.ones_like(x) + Aty)
    # workspaces: copy, line sums (profiles) and two scratch volumes of those slices
    _, ny, nx = A.domain_shape
    _, angles, cols = A.range_shape
    n = (_slices(nz, rows, pitch, first, move) + 3) // 4 * 4
    volume, lines = 4 * n * (ny + 4) * (nx + 4), 4 * n * angles * cols
    pairs = 8 * (rows + 4) * angles * cols
    stats = A.projector.stats(dev.index)
    if 2 * rows >= n or n <= 64:  # (few rows over many slices follow their rays)
        assert stats["fp_workspace_bytes"] <= max(lines + 2 * volume, 4 * nz * ny * nx) + 4 * 256
    assert stats["bp_workspace_bytes"] <= max(lines + 2 * volume, pairs) + 4 * 256


@pytest.mark.parametrize("name", ["middle", "top", "rising", "below"])
def test_ranges_items_and_sirt(dev, name):
    from tomosipo_gb300.sirt import BatchedSirt, sirt

    nz, rows, pitch, first, move = CASES[name]
    vg, pg = _scan(nz, rows, pitch, first, move=move)
    A = ts.operator(vg, pg)
    g = torch.Generator().manual_seed(6)
    x = torch.rand((3,) + A.domain_shape, generator=g).to(dev)
    y = torch.empty((3,) + A.range_shape, device=dev)
    A._apply_batch(x, y)
    assert torch.equal(y, torch.stack([A(v) for v in x]))
    back = torch.full_like(x, 7.0)
    A.T._apply_batch(y, back)
    assert torch.equal(back, torch.stack([A.T(v) for v in y]))
    # two angle ranges
    lib, h = _native.load(), A.projector.handle(dev.index)
    stream = torch.cuda.current_stream(dev).cuda_stream
    part, sums = torch.empty_like(y[0]), torch.empty_like(x[0])
    nfp, nbp = (A.projector.workspace_bytes(dev.index, f) for f in (True, False))
    ws = torch.empty(max(nfp, nbp), dtype=torch.uint8, device=dev)
    for k, (a, b) in enumerate(((0, 3), (3, 7))):
        _native.check(lib.tsgb_direct_fp_angles(h, x[0].data_ptr(), part.data_ptr(), 0, a, b, k,
                                                ws.data_ptr(), nfp, stream), "fp")
    assert torch.equal(part, y[0])
    for k, (a, b) in enumerate(((0, 3), (3, 7))):
        _native.check(lib.tsgb_direct_bp_angles(h, sums.data_ptr(), y[0].data_ptr(), k, a, b,
                                                ws.data_ptr(), nbp, stream), "bp")
    assert rel_l2(sums.cpu().numpy(), back[0].cpu().numpy()) <= 1e-6
    b = BatchedSirt([(A, y[0]), (A, y[1])])
    b.run(3, graph=False)
    for k in range(2):
        assert torch.equal(b.x[k], sirt(A, y[k], 3))
    b.close()
