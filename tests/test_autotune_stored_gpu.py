"""Stored tunings that were timed when slice scans had one backprojector: their bp_kernel 0
does not select the voxel-pair kernel there; on other scans, and in tunings stored since,
it does."""
import json

import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300 import autotune as at

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scan, since, kernel", [("parallel", False, 3), ("parallel", True, 1),
                                                 ("cone", False, 1)])
def test_stored_kernel(native_lib, tmp_path, scan, since, kernel):
    vg = ts.volume(shape=(20, 21, 22), size=1)
    pg = (ts.parallel(angles=5, shape=(20, 30), size=1.4) if scan == "parallel"
          else ts.cone(angles=5, shape=(20, 30), size=1.4, cone_angle=0.3))
    A = ts.operator(vg, pg)
    key = at.geometry_key(A.projector)
    stored = {"tuning": dict(A.projector.get_tuning(0), bp_kernel=0, bp_shape=0), "ms": 1.0,
              "default_ms": 1.0, "trials": 14}
    if since:
        stored["bp_candidates"] = 2
    path = tmp_path / "tuning.json"
    path.write_text(json.dumps({key: stored}))
    at._cache.pop(key, None)
    for cache_path in (str(path), None):  # from the file, then from memory
        assert at.autotune(A, cache_path=cache_path)["cached"]
        assert A.projector.stats(0)["bp_matched_kernel"] == kernel
        A.projector.set_tuning(0, bp_kernel=1)
    at._cache.pop(key, None)
