"""The autotuner times what differs: no forward schedule and two backprojectors on scans
that run slice by slice, and no two shapes of one launch on the others."""
import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300 import autotune as at

torch = pytest.importorskip("torch")


def _run(nz, most):
    """Voxels along z per lane, at most ``most``, in ranges of near-equal length."""
    lanes = -(-nz // 32)
    return -(-lanes // -(-lanes // most))


@pytest.mark.parametrize("nz", [1, 32, 33, 64, 65, 96, 128, 129, 160, 224, 225, 256, 257, 300, 512])
def test_shapes_with_launches_of_their_own(nz):
    chosen = at.bp_candidates(2, nz)
    assert set(map(str, chosen)) <= set(map(str, at.BP_CANDIDATES))
    # a shape's launch: voxels per lane, and the window where lanes hold 8
    launches = {}
    for k in range(7):
        run = _run(nz, {5: 4, 6: 2}.get(k, 8))
        launches.setdefault((run, k if run == 8 and k in (3, 4) else 0), []).append(k)
    shapes = [c["bp_shape"] for c in chosen if c["bp_kernel"] == 1]
    assert len(shapes) == len(set(shapes)) and len(chosen) == len(shapes) + 1
    assert all(sum(k in shapes for k in group) == 1 for group in launches.values())


def test_one_kernel_or_none():
    assert at.bp_candidates(0, 100) == ()
    assert [(c["bp_kernel"], c["bp_shape"]) for c in at.bp_candidates(3, 256)] == [(0, 0), (1, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("scan, trials, bp_trials", [("parallel", 1, 2), ("cone", 14, 2)])
def test_autotune_times_each_launch_once(native_lib, scan, trials, bp_trials):
    vg = ts.volume(shape=(40, 20, 22), size=1)
    pg = (ts.parallel(angles=9, shape=(40, 30), size=1.4) if scan == "parallel"
          else ts.cone(angles=9, shape=(40, 30), size=1.4, cone_angle=0.3))
    A = ts.operator(vg, pg)
    at._cache.pop(at.geometry_key(A.projector), None)
    r = at.autotune(A)
    at._cache.pop(at.geometry_key(A.projector), None)
    assert (r["trials"], r["bp_trials"]) == (trials, bp_trials)
    assert A.projector.get_tuning(0) == r["tuning"]
