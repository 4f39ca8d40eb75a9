"""Operator calls on device tensors the kernels take as they are skip the links;
everything else goes through them. Both give the same results, conversions and
errors for every form of input and output."""
import numpy as np
import pytest

import tomosipo_gb300 as ts
from tomosipo_gb300.links.base import link
from tomosipo_gb300.projector import device_ready, direct_bp, direct_fp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(native_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


def _linked(op, forward, src, additive=False, out=None, kind="matched"):
    """The same projection through the links."""
    vg, pg = op.astra_compat_vg, op.astra_compat_pg
    if out is None:
        out = torch.zeros(op.range_shape if forward else op.domain_shape, device=src.device)
    if forward:
        direct_fp(op.projector, link(vg, src), link(pg, out), additive=additive)
    else:
        direct_bp(op.projector, link(vg, out), link(pg, src), additive=additive, bp_kind=kind)
    return out


def _forms(t):
    wide = torch.zeros(t.shape[:-1] + (2 * t.shape[-1],), device=t.device)
    wide[..., ::2] = t
    return {
        "plain": (t, True),
        "requires_grad": (t.clone().requires_grad_(), True),
        "view_with_offset": (torch.cat([t[:1], t])[1:], True),
        "parameter": (torch.nn.Parameter(t.clone()), False),
        "strided": (wide[..., ::2], False),
        "transposed": (t.transpose(0, 2).contiguous().transpose(0, 2), False),
        "double": (t.double(), False),
    }


@pytest.mark.filterwarnings("ignore:The parameter initial_value")
@pytest.mark.parametrize("kind", ["matched", "bilinear"])
@pytest.mark.parametrize("scan", ["parallel", "cone"])
def test_forms_equal_the_links(dev, scan, kind):
    vg = ts.volume(shape=(9, 12, 14), size=1)
    pg = (ts.parallel(angles=7, shape=(10, 20), size=1.5) if scan == "parallel"
          else ts.cone(angles=7, shape=(10, 20), size=1.5, cone_angle=0.4))
    for additive in (False, True):
        A = ts.operator(vg, pg, additive=additive, backprojector=kind)
        for forward, op, shape, out_shape in ((True, A, A.domain_shape, A.range_shape),
                                              (False, A.T, A.range_shape, A.domain_shape)):
            t = torch.rand(shape, generator=torch.Generator().manual_seed(1)).to(dev)
            for name, (src, ready) in _forms(t).items():
                assert device_ready(src) == ready, name
                ref = _linked(A, forward, src, additive, kind=kind)
                with torch.no_grad():
                    assert torch.equal(op(src), ref), name
                    out = torch.full(out_shape, 2.0, device=dev)
                    want = _linked(A, forward, src, additive, out.clone(), kind)
                    assert op(src, out=out) is out and torch.equal(out, want), name


def test_refusals_stay(dev):
    A = ts.operator(ts.volume(shape=(4, 5, 6)), ts.parallel(angles=3, shape=(4, 8)))
    x = torch.ones(A.domain_shape, device=dev)
    with pytest.raises(ValueError):
        A(torch.ones((4, 5, 7), device=dev))
    with pytest.raises(ValueError):
        A(x, out=torch.ones((4, 3, 9), device=dev))
    with pytest.raises(ValueError):
        A(x, out=torch.ones(A.range_shape))  # another device
    with pytest.raises(ValueError):
        A(x, out=np.ones(A.range_shape, np.float32))
    assert not device_ready(torch.ones(3)) and not device_ready(np.ones(3))
