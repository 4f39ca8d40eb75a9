"""Parallel beams whose rays stay in one volume slice (flat.cu): both
projections at the sizes where their launches change (voxels along z per lane,
several z ranges, angles split between warps, thin wide volumes that keep the
voxel-pair backprojector), over the forms the path takes (rows coarser and finer
than the voxels, det_v or the rays reversed, detectors off centre or moving along
z, anisotropic and moved volumes, one angle), against the FP64 oracle; stacked
items, additive calls and batched SIRT equal the plain calls; and a scan just
outside the path's condition agrees with one inside it."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from oracle import oracle as orc
from tests.helpers import TOL_ADJOINT, TOL_ORACLE, adjoint_error, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _flat_workspace(A):
    """Forward workspaces of the flat path: volume copy with a border of 2 and the
    line sums, or what batched SIRT's backprojection keeps there (resampled
    sinogram and scratch volumes; thin wide volumes: sum and scratch volumes)."""
    (nz, ny, nx), (_, angles, cols) = A.domain_shape, A.range_shape
    zs = (nz + 3) // 4 * 4

    def r(n):
        return (4 * n + 255) // 256 * 256

    lines = r(angles * cols * zs)
    return ([r((ny + 4) * (nx + 4) * zs) + lines] + [lines + k * r(ny * nx * zs) for k in (1, 2)]
            + [3 * r(nz * ny * nx)])


@pytest.fixture(scope="module")
def dev(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def _scan(nz, ny, nx, rows, cols, height=1.0, angles=9):
    vg = ts.volume(shape=(nz, ny, nx), size=(nz / 32, ny / 32, nx / 32))
    pg = ts.parallel(angles=np.linspace(0, np.pi, angles, endpoint=False) + 0.1,
                     shape=(rows, cols), size=(height * nz / 32, 1.4 * max(nx, ny) / 32))
    return vg, pg


def _check(dev, vg, pg, flat=True):
    A = ts.operator(vg, pg)
    got = A.projector.stats(dev.index)["fp_workspace_bytes"]
    assert (got in _flat_workspace(A)) == flat
    gen = torch.Generator().manual_seed(5)
    x = torch.rand(A.domain_shape, generator=gen).to(dev)
    y = torch.rand(A.range_shape, generator=gen).to(dev)
    Ax, Aty = A(x).cpu().numpy(), A.T(y).cpu().numpy()
    assert rel_l2(Ax, orc.fp(vg, pg, x.cpu().numpy())) <= TOL_ORACLE
    assert rel_l2(Aty, orc.bp_matched(vg, pg, y.cpu().numpy())) <= TOL_ORACLE
    assert adjoint_error(Ax, y.cpu().numpy(), x.cpu().numpy(), Aty) <= TOL_ADJOINT
    B = ts.operator(vg, pg, additive=True)
    out = torch.ones_like(y)
    B(x, out=out)
    assert torch.equal(out, torch.ones_like(y) + A(x))
    acc = torch.ones_like(x)
    B.T(y, out=acc)
    assert rel_l2(acc.cpu().numpy() - 1, Aty) <= 1e-5


@pytest.mark.parametrize("nz", [1, 2, 31, 33, 64, 65, 127, 129, 255, 257, 300])
def test_z_extents(dev, nz):
    _check(dev, *_scan(nz, 11, 14, max(1, int(0.9 * nz)), 21))


@pytest.mark.parametrize("nz, n", [(192, 12), (193, 12), (385, 9), (140, 190)])
def test_ranges_of_three_runs(dev, nz, n):
    """Around the heights where the backprojector's z ranges are 192 voxels, not 256."""
    _check(dev, *_scan(nz, n, n - 1, nz + 3, int(1.4 * n), angles=5))


@pytest.mark.parametrize("nz, ny, nx", [(20, 1, 1), (20, 3, 70), (20, 70, 3), (40, 120, 130),
                                        (70, 130, 140), (130, 100, 90), (16, 190, 180), (17, 190, 180)])
def test_planes_and_splits(dev, nz, ny, nx):
    _check(dev, *_scan(nz, ny, nx, nz, int(1.4 * max(nx, ny)), angles=40))


@pytest.mark.parametrize("rows", [3, 20, 37, 75, 160])
@pytest.mark.parametrize("height", [0.4, 1.0, 1.7])
def test_rows(dev, rows, height):
    _check(dev, *_scan(36, 10, 12, rows, 19, height))


def _forms():
    vg, pg = _scan(24, 17, 21, 26, 33, 1.1, 10)
    v = pg.to_vec()
    z = np.zeros((10, 3))
    z[:, 0] = np.linspace(-0.2, 0.3, 10)

    def vec(ray_dir=v.ray_dir, det_pos=v.det_pos, det_v=v.det_v, det_u=v.det_u):
        return ts.parallel_vec(shape=v.det_shape, ray_dir=ray_dir, det_pos=det_pos, det_v=det_v,
                               det_u=det_u)

    return {
        "rows_reversed": (vg, vec(det_v=-np.asarray(v.det_v))),
        "rays_reversed": (vg, vec(ray_dir=-3.0 * np.asarray(v.ray_dir))),
        "columns_reversed": (vg, vec(det_u=-np.asarray(v.det_u))),
        "moving_along_z": (vg, vec(det_pos=np.asarray(v.det_pos) + z)),
        "off_centre": (vg, vec(det_pos=np.asarray(v.det_pos) + 0.3 * np.asarray(v.det_u) * 7)),
        "sheared_detector": (vg, vec(det_u=np.asarray(v.det_u) + 0.4 * np.asarray(v.ray_dir) / 32)),
        "anisotropic_moved": (ts.volume(shape=(24, 17, 21), size=(1.0, 0.4, 0.9), pos=(0.1, -0.05, 0.2)),
                              pg),
        "one_angle": (vg, ts.parallel(angles=[0.3], shape=(26, 33), size=(0.8, 1.0))),
        "axis_angles": (vg, ts.parallel(angles=[0.0, np.pi / 2, np.pi], shape=(26, 33), size=(0.8, 1.0))),
    }


@pytest.mark.parametrize("name", sorted(_forms()))
def test_forms(dev, name):
    _check(dev, *_forms()[name])


def test_next_to_the_condition(dev):
    """A ray leaving its slice, or a detector column rising along u, by 1e-9 of
    a voxel takes the general kernels, and the results agree."""
    vg, pg = _scan(24, 17, 21, 26, 33, 1.1, 10)
    v = pg.to_vec()
    tilt = np.zeros((10, 3))
    tilt[4, 0] = 1e-9
    A = ts.operator(vg, pg)
    x = torch.rand(A.domain_shape, generator=torch.Generator().manual_seed(1)).to(dev)
    y = torch.rand(A.range_shape, generator=torch.Generator().manual_seed(2)).to(dev)
    for name in ("ray_dir", "det_u"):
        args = {k: np.asarray(getattr(v, k)) for k in ("ray_dir", "det_pos", "det_v", "det_u")}
        args[name] = args[name] + tilt * (1.0 if name == "ray_dir" else 1 / 32)
        near = ts.parallel_vec(shape=v.det_shape, **args)
        B = ts.operator(vg, near)
        _check(dev, vg, near, flat=False)
        assert rel_l2(A(x).cpu().numpy(), B(x).cpu().numpy()) <= TOL_ORACLE
        assert rel_l2(A.T(y).cpu().numpy(), B.T(y).cpu().numpy()) <= TOL_ORACLE


@pytest.mark.parametrize("nz, n", [(12, 20), (70, 33), (16, 184)])
def test_stacked_items_and_batched_sirt(dev, nz, n):
    from tomosipo_gb300.sirt import BatchedSirt, sirt

    vg, pg = _scan(nz, n, n, nz, int(1.4 * n), angles=30)
    A = ts.operator(vg, pg)
    x = torch.rand((3,) + A.domain_shape, generator=torch.Generator().manual_seed(6)).to(dev)
    y = torch.empty((3,) + A.range_shape, device=dev)
    A._apply_batch(x, y)
    assert torch.equal(y, torch.stack([A(v) for v in x]))
    back = torch.empty_like(x)
    A.T._apply_batch(y, back)
    assert torch.equal(back, torch.stack([A.T(v) for v in y]))
    b = BatchedSirt([(A, y[0]), (A, y[1])])
    b.run(3, graph=False)
    for k in range(2):
        assert torch.equal(b.x[k], sirt(A, y[k], 3))
    b.close()


def test_non_finite_voxels_stay_in_their_rays(dev):
    """An infinite voxel makes the rays that sample it non-finite and no others."""
    vg, pg = _scan(20, 15, 18, 20, 24, angles=6)
    A = ts.operator(vg, pg)
    x = torch.rand(A.domain_shape, generator=torch.Generator().manual_seed(3))
    w = torch.zeros_like(x)
    w[7, 4, 11] = 1.0
    hit = torch.from_numpy(orc.fp(vg, pg, w.numpy())) > 1e-6
    x[7, 4, 11] = float("inf")
    y = A(x.to(dev)).cpu()
    assert not torch.isfinite(y[hit]).any()
    miss = torch.from_numpy(orc.fp(vg, pg, torch.nn.functional.max_pool3d(
        w[None], 3, 1, 1)[0].numpy())) == 0
    assert torch.isfinite(y[miss]).all()
