"""Parallel scans at the limits of the slice kernels (flat.cu): sizes beyond their
32-bit offsets keep the general kernels."""
import numpy as np
import pytest

import tomosipo_gb300 as ts

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def test_wide_planes_keep_the_general_kernels(dev):
    """One plane of voxels whose ray kernel's copy has fewer than 2^31 elements, but
    whose slice copy, with a border on both in-slice axes, has more: the plan (no
    projection is run) takes the ray kernel, whose workspace is a copy of pairs."""
    n = 40000
    A = ts.operator(ts.volume(shape=(n, 1, n)), ts.parallel(angles=[0.0], shape=(4, 8)))
    stats = A.projector.stats(dev.index)
    assert stats["layouts"] == 1
    assert stats["fp_workspace_bytes"] == 8 * (((n + 4) ** 2 + 31) // 32 * 32)
