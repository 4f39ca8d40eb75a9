"""Timed workloads of the projection path, through the package's public calls.

``listed()`` are the fixed cases, ``draw`` gives more of the same ranges,
``prepare`` / ``run`` make a case's inputs and do one pass of it, ``work`` says
what a pass cannot do without, and ``exact`` computes the same outputs in 64
bits with plain torch, from the discretisation's definition (Joseph's method
on the planes of an angle's dominant axis, and its transpose).

A case: ``scan`` (parallel, cone, helical, tilted), ``op`` (fp, bp, grad, sirt,
fdk), the volume's and detector's shapes, the number of angles, ``start`` (the
first angle), ``height`` and ``width`` (the detector's extent at the rotation
axis over the volume's), ``batch`` (stacked volumes), ``iters`` (SIRT
iterations) and ``ss`` (detector supersampling).
"""
import math

import numpy as np
import torch

import tomosipo_gb300 as ts
from tomosipo_gb300.fdk import fdk_reconstruct
from tomosipo_gb300.sirt import sirt
from tomosipo_gb300.torch_support import to_autograd

SQRT2 = math.sqrt(2.0)
DISTANCE = 2 * SQRT2  # source to axis and axis to detector of ts.cone(size=sqrt(2), cone_angle=0.5)
EXACT_SAMPLES = 2.5e10  # ray samples that exact() computes within a few seconds


def _case(name, scan, op, vol, det, angles, height, width, start=0.05, batch=1, iters=0, ss=1):
    return {"name": name, "scan": scan, "op": op, "nz": vol[0], "ny": vol[1], "nx": vol[2],
            "rows": det[0], "cols": det[1], "angles": angles, "height": height, "width": width,
            "start": start, "batch": batch, "iters": iters, "ss": ss}


def listed():
    return [
        # the smallest scan of the benchmark configurations, as one layer of a
        # learned reconstruction: projection and its gradient; launches count
        _case("parallel_grad_64", "parallel", "grad", (64, 64, 64), (64, 96), 96, 1.0, 1.5),
        # a small cone scan reconstructed with a few SIRT iterations
        _case("cone_sirt_96", "cone", "sirt", (96, 96, 96), (96, 144), 120, SQRT2, SQRT2, iters=4),
        # the medium cone scan of the benchmark configurations, each direction
        _case("cone_fp_256", "cone", "fp", (256, 256, 256), (256, 384), 360, SQRT2, SQRT2),
        _case("cone_bp_256", "cone", "bp", (256, 256, 256), (256, 384), 360, SQRT2, SQRT2),
        # the headline cone scan, each direction
        _case("cone_fp_512", "cone", "fp", (512, 512, 512), (512, 768), 1024, SQRT2, SQRT2,
              start=0.0),
        _case("cone_bp_512", "cone", "bp", (512, 512, 512), (512, 768), 1024, SQRT2, SQRT2,
              start=0.0),
        # a synchrotron-style parallel scan of odd sizes, both directions
        _case("parallel_grad_odd", "parallel", "grad", (203, 397, 421), (211, 563), 401, 1.0, 1.35),
        # the learned primal-dual network's projector calls: a batch of 8 volumes
        _case("lpd_grad_128", "cone", "grad", (128, 128, 128), (128, 192), 128, SQRT2, SQRT2,
              batch=8),
        # a helical scan with jittered source and detector, both directions
        _case("helical_grad_odd", "helical", "grad", (170, 190, 181), (173, 259), 257, SQRT2,
              SQRT2),
        # a scan whose detector is tilted out of the z axis, both directions
        _case("tilted_grad_odd", "tilted", "grad", (120, 152, 161), (131, 219), 180, SQRT2, SQRT2),
        # an analytic reconstruction
        _case("fdk_320", "cone", "fdk", (320, 320, 320), (320, 480), 500, SQRT2, SQRT2),
        # 2 x 2 rays per detector pixel, both directions
        _case("cone_ss2_grad", "cone", "grad", (128, 160, 160), (128, 240), 200, SQRT2, SQRT2,
              ss=2),
    ]


def draw(rng):
    """One more case of the listed ones' ranges."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    scan, op = rng.choice([("parallel", "fp"), ("parallel", "bp"), ("parallel", "grad"),
                           ("cone", "fp"), ("cone", "bp"), ("cone", "grad"), ("cone", "sirt"),
                           ("cone", "fdk"), ("helical", "fp"), ("helical", "bp"),
                           ("tilted", "grad")])
    hi = {"tilted": 200, "helical": 320}.get(scan, 448)
    nx = size(64, hi)
    ny = max(48, int(nx * rng.uniform(0.8, 1.1)))
    nz = max(32, int(nx * rng.uniform(0.4, 1.1)))
    rows = max(32, int(nz * rng.uniform(0.8, 1.2)))
    cols = max(48, int(nx * rng.uniform(1.1, 1.6)))
    angles = int(rng.uniform(0.6, 1.8) * nx) + 1
    height, width = (1.0, rng.uniform(1.2, 1.5)) if scan == "parallel" else (SQRT2, SQRT2)
    ss = 2 if op == "grad" and scan == "cone" and nx <= 200 and rng.random() < 0.4 else 1
    batch = rng.randint(2, 8) if op == "grad" and ss == 1 and nx <= 150 else 1
    iters = rng.randint(2, 4) if op == "sirt" else 0
    return {"scan": scan, "op": op, "nz": nz, "ny": ny, "nx": nx, "rows": rows, "cols": cols,
            "angles": angles, "height": height, "width": width,
            "start": rng.uniform(0.02, 0.7), "batch": batch, "iters": iters, "ss": ss}


# ------------------------------------------------------------------ geometry
def _extent(case):
    """(volume size, detector size at the axis), world units: the volume is 1 wide along x."""
    voxel = 1.0 / case["nx"]
    vol = tuple(case[k] * voxel for k in ("nz", "ny", "nx"))
    return vol, (case["height"] * vol[0], case["width"] * vol[2])


def _angles(case):
    if case["scan"] == "parallel":
        span = math.pi
    else:
        span = 3 * math.pi if case["scan"] == "helical" else 2 * math.pi
    return np.linspace(0.0, span, case["angles"], endpoint=False) + case["start"]


def _vectors(case):
    """(first, det_pos, det_v, det_u) per angle, (z, y, x): first is the source
    position, or the ray direction of a parallel beam."""
    (height, width) = _extent(case)[1]
    t = _angles(case)
    c, s, zero = np.cos(t), np.sin(t), np.zeros_like(t)
    sv, su = height / case["rows"], width / case["cols"]
    if case["scan"] == "parallel":
        first, det = np.stack([zero, -c, s], 1), np.zeros((len(t), 3))
        grow = 1.0
    else:
        first = np.stack([zero, -c * DISTANCE, s * DISTANCE], 1)
        # circular and tilted scans have the detector on the axis, helical
        # ones as far behind it as the source is in front
        behind = DISTANCE if case["scan"] == "helical" else 0.0
        det = np.stack([zero, c * behind, -s * behind], 1)
        grow = 1.0 + behind / DISTANCE
    v = np.stack([zero + sv * grow, zero, zero], 1)
    u = np.stack([zero, s * su * grow, c * su * grow], 1)
    if case["scan"] == "helical":
        rise = 0.5 * _extent(case)[0][0] * (t - t.mean()) / (2 * math.pi)
        jitter = np.random.default_rng(11).normal(0.0, 0.5 / case["nx"], (2, len(t), 3))
        first = first + np.stack([rise, zero, zero], 1) + jitter[0]
        det = det + np.stack([rise, zero, zero], 1) + jitter[1]
    if case["scan"] == "tilted":
        axis = np.array([1.0, 0.3, -0.2]) / math.sqrt(1.13)
        k = np.array([[0, -axis[2], axis[1]], [axis[2], 0, -axis[0]], [-axis[1], axis[0], 0]])
        # the scan turned 0.4 rad about an axis near y and x, out of the z axis
        k = k[:, [1, 0, 2]][[1, 0, 2]]
        turn = np.eye(3) + math.sin(0.4) * k + (1 - math.cos(0.4)) * k @ k
        first, det, v, u = (a @ turn.T for a in (first, det, v, u))
    return first, det, v, u


def _geometries(case):
    vol_size, (height, width) = _extent(case)
    vg = ts.volume(shape=(case["nz"], case["ny"], case["nx"]), size=vol_size)
    shape = (case["rows"], case["cols"])
    if case["scan"] == "parallel":
        return vg, ts.parallel(angles=_angles(case), shape=shape, size=(height, width))
    if case["scan"] == "cone":
        return vg, ts.cone(angles=_angles(case), shape=shape, size=(height, width),
                           src_orig_dist=DISTANCE, src_det_dist=DISTANCE)
    first, det, v, u = _vectors(case)
    return vg, ts.cone_vec(shape=shape, src_pos=first, det_pos=det, det_v=v, det_u=u)


# -------------------------------------------------------------------- inputs
def _volume(case, gen):
    """Ellipsoids of densities 0.1 .. 1 with a little texture."""
    dev = gen.device
    z, y, x = (torch.linspace(-1, 1, case[k], device=dev) for k in ("nz", "ny", "nx"))
    out = torch.empty((case["nz"], case["ny"], case["nx"]), device=dev)
    out.uniform_(0.0, 0.02, generator=gen)
    p = torch.rand((8, 7), generator=gen, device=dev).tolist()
    for cz, cy, cx, rz, ry, rx, rho in p:
        r = [0.15 + 0.4 * a for a in (rz, ry, rx)]
        m = [1.2 * (a - 0.5) for a in (cz, cy, cx)]
        inside = (((z - m[0]) / r[0]) ** 2)[:, None, None] + (((y - m[1]) / r[1]) ** 2)[None, :, None] \
            + (((x - m[2]) / r[2]) ** 2)[None, None, :] < 1
        out.add_(inside, alpha=0.1 + 0.9 * rho)
    return out


def _sinogram(case, gen):
    """Smooth traces of a few objects turning with the scan, well inside the
    volume's shadow, and noise that grows with the signal."""
    dev = gen.device
    t = torch.as_tensor(_angles(case), dtype=torch.float32, device=dev)
    v = torch.linspace(-1, 1, case["rows"], device=dev)
    u = torch.linspace(-1, 1, case["cols"], device=dev)
    out = torch.zeros((case["rows"], case["angles"], case["cols"]), device=dev)
    for r, phase, row, wv, wu, a in torch.rand((6, 6), generator=gen, device=dev).tolist():
        centre = 0.3 * r * torch.cos(t + 6.28 * phase)
        gv = torch.exp(-(((v - 0.5 * (row - 0.5)) / (0.05 + 0.1 * wv)) ** 2))
        gu = torch.exp(-(((u[None, :] - centre[:, None]) / (0.04 + 0.08 * wu)) ** 2))
        out.addcmul_(gv[:, None, None] * (0.2 + 0.8 * a), gu[None])
    noise = torch.empty_like(out).normal_(0.0, 1.0, generator=gen)
    return out.addcmul_(noise, out, value=0.03)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["op"] == "grad":
        x = torch.stack([_volume(case, gen) for _ in range(case["batch"])])[:, None]
        g = torch.stack([_sinogram(case, gen) for _ in range(case["batch"])])[:, None]
        return (x, g) if case["batch"] > 1 else (x[0, 0].clone(), g[0, 0].clone())
    if case["op"] == "fp":
        return (_volume(case, gen),)
    return (_sinogram(case, gen),)


def prepare(case, seed):
    vg, pg = _geometries(case)
    state = {"case": case, "vg": vg, "pg": pg,
             "A": ts.operator(vg, pg, detector_supersampling=case["ss"]),
             "inputs": _inputs(case, seed)}
    if case["op"] == "grad":
        state["layer"] = to_autograd(state["A"], num_extra_dims=2 if case["batch"] > 1 else 0)
        state["inputs"][0].requires_grad_()
    return state


def run(state):
    op, A, inputs = state["case"]["op"], state["A"], state["inputs"]
    if op == "fp":
        return A(inputs[0])
    if op == "bp":
        return A.T(inputs[0])
    if op == "grad":
        x, g = inputs
        y = state["layer"](x)
        (dx,) = torch.autograd.grad(y, x, g)
        return {"y": y.detach(), "dx": dx}
    if op == "sirt":
        return sirt(A, inputs[0], state["case"]["iters"])
    return fdk_reconstruct(state["vg"], state["pg"], inputs[0], projector=A.projector)


def work(case):
    """Each input read once and each output written once; per voxel and angle
    the multiply-adds of interpolating it (two in the slice, and two along z
    where the rays leave it)."""
    vol = case["nz"] * case["ny"] * case["nx"] * case["batch"]
    sino = case["rows"] * case["angles"] * case["cols"] * case["batch"]
    passes = {"fp": 1, "bp": 1, "grad": 2, "sirt": 2 * (case["iters"] + 1), "fdk": 1}[case["op"]]
    # a gradient pass reads and writes one volume and one sinogram each way
    moved = 2 * (vol + sino) if case["op"] == "grad" else vol + sino
    per = 4 if case["scan"] == "parallel" else 8
    return {"bytes": 4 * moved, "flops": per * vol * case["angles"] * case["ss"] ** 2 * passes}


# --------------------------------------------------------------- 64-bit answer
class _Exact:
    """The projector's definition in 64 bits: an angle's rays are sampled on
    every voxel-centre plane of its dominant axis (the largest component, in
    voxels, of the ray through the detector's centre) by bilinear
    interpolation, times the ray's length between planes."""

    def __init__(self, case):
        self.dev = torch.device("cuda")
        self.case, ss = case, case["ss"]
        first, det, v, u = _vectors(case)
        self.rows, self.cols = case["rows"] * ss, case["cols"] * ss
        self.shape = (case["nz"], case["ny"], case["nx"])
        vol_size = _extent(case)[0]
        self.vs = [vol_size[i] / self.shape[i] for i in range(3)]
        # world position w -> voxel index
        self.low = [-0.5 * vol_size[i] + 0.5 * self.vs[i] for i in range(3)]
        self.first, self.det, self.v, self.u = first, det, v / ss, u / ss

    def rays(self, t):
        """Dominant axis, in-plane axes, and per pixel the position on plane 0
        and the step per plane along them, and the length of a step."""
        parallel = self.case["scan"] == "parallel"
        f, d = self.first[t], self.det[t]
        centre = [(f[i] if parallel else d[i] - f[i]) / self.vs[i] for i in range(3)]
        k = max(range(3), key=lambda i: abs(centre[i]))
        rest = [i for i in range(3) if i != k]
        r = torch.arange(self.rows, device=self.dev, dtype=torch.float64) + 0.5 - self.rows / 2
        c = torch.arange(self.cols, device=self.dev, dtype=torch.float64) + 0.5 - self.cols / 2
        pix = [((d[i] + r[:, None] * self.v[t, i] + c[None, :] * self.u[t, i]) - self.low[i])
               / self.vs[i] for i in range(3)]
        if parallel:
            way = [torch.full_like(pix[i], f[i] / self.vs[i]) for i in range(3)]
        else:
            src = [(f[i] - self.low[i]) / self.vs[i] for i in range(3)]
            way = [pix[i] - src[i] for i in range(3)]
        slope = [way[i] / way[k] for i in rest]
        start = [pix[i] - pix[k] * m for i, m in zip(rest, slope)]
        length = torch.sqrt(self.vs[k] ** 2 + sum((self.vs[i] * m) ** 2
                                                  for i, m in zip(rest, slope)))
        return k, rest, start, slope, length

    def taps(self, t):
        """(flat voxel indices, weights) of every sample of angle t, in slabs
        of planes; the last step's length comes with them."""
        k, rest, start, slope, length = self.rays(t)
        n = self.shape
        stride = (n[1] * n[2], n[2], 1)
        per = max(1, int(2 ** 25 // (self.rows * self.cols)))
        for p0 in range(0, n[k], per):
            plane = torch.arange(p0, min(n[k], p0 + per), device=self.dev, dtype=torch.float64)
            qa = start[0][None] + plane[:, None, None] * slope[0][None]
            qb = start[1][None] + plane[:, None, None] * slope[1][None]
            ia, ib = torch.floor(qa), torch.floor(qb)
            fa, fb = qa - ia, qb - ib
            ia, ib = ia.long(), ib.long()
            base = plane.long()[:, None, None] * stride[k]
            for da in (0, 1):
                for db in (0, 1):
                    i, j = ia + da, ib + db
                    inside = (i >= 0) & (i < n[rest[0]]) & (j >= 0) & (j < n[rest[1]])
                    w = (fa if da else 1 - fa) * (fb if db else 1 - fb) * length[None] * inside
                    at = base + i.clamp(0, n[rest[0]] - 1) * stride[rest[0]] \
                        + j.clamp(0, n[rest[1]] - 1) * stride[rest[1]]
                    yield at, w

    def forward(self, x):
        x = x.double().reshape(-1)
        ss = self.case["ss"]
        out = torch.zeros((self.rows, self.case["angles"], self.cols), device=self.dev,
                          dtype=torch.float64)
        for t in range(self.case["angles"]):
            for at, w in self.taps(t):
                out[:, t] += (x[at] * w).sum(0)
        if ss > 1:
            out = out.reshape(self.case["rows"], ss, -1, self.case["cols"], ss).mean((1, 4))
        return out

    def back(self, y):
        y, ss = y.double(), self.case["ss"]
        if ss > 1:
            y = y.repeat_interleave(ss, 0).repeat_interleave(ss, 2) / ss ** 2
        out = torch.zeros(self.shape, device=self.dev, dtype=torch.float64).reshape(-1)
        for t in range(self.case["angles"]):
            for at, w in self.taps(t):
                out.index_add_(0, at.reshape(-1), (w * y[:, t][None]).reshape(-1))
        return out.reshape(self.shape)

    def sirt(self, y):
        def inverse(a):
            return torch.clamp(1 / a, max=1e8)

        ones = torch.ones((), device=self.dev, dtype=torch.float64)
        R = inverse(self.forward(ones.expand(self.shape)))
        C = inverse(self.back(ones.expand(y.shape)))
        x = torch.zeros(self.shape, device=self.dev, dtype=torch.float64)
        for _ in range(self.case["iters"]):
            x = x + C * self.back(R * (y.double() - self.forward(x)))
        return x

    def fdk(self, y):
        """Feldkamp, Davis and Kress: cosine weights, the ramp filter on the
        virtual detector through the volume's anchor voxel (index n // 2), and
        the depth-weighted bilinear backprojection."""
        n, cols, rows = self.shape, self.cols, self.rows
        anchor = np.array([self.low[i] + (n[i] // 2) * self.vs[i] for i in range(3)])
        ramp = np.zeros(2 * cols)
        odd = np.arange(1, cols, 2)
        ramp[0] = 0.25
        ramp[odd] = ramp[2 * cols - odd] = -1 / (math.pi * odd) ** 2
        ramp = torch.fft.rfft(torch.from_numpy(ramp).to(self.dev)).real
        rel = self.first - anchor
        beta = np.unwrap(np.arctan2(rel[:, 1], rel[:, 2]))
        dbeta = np.abs(np.gradient(beta))
        out = torch.zeros(n, device=self.dev, dtype=torch.float64)
        r = torch.arange(rows, device=self.dev, dtype=torch.float64) + 0.5 - rows / 2
        c = torch.arange(cols, device=self.dev, dtype=torch.float64) + 0.5 - cols / 2
        at = [self.low[i] + self.vs[i] * torch.arange(n[i], device=self.dev, dtype=torch.float64)
              for i in range(3)]
        for t in range(self.case["angles"]):
            S, D, V, U = self.first[t], self.det[t], self.v[t], self.u[t]
            normal = np.cross(U, V)
            normal /= np.linalg.norm(normal)
            normal *= np.sign((D - S) @ normal)
            sdd, sod = (D - S) @ normal, (anchor - S) @ normal
            dist = torch.sqrt(sum((D[i] - S[i] + r[:, None] * V[i] + c[None, :] * U[i]) ** 2
                                  for i in range(3)))
            q = torch.fft.rfft(y[:, t].double() * sdd / dist, n=2 * cols)
            pitch = np.linalg.norm(U) * sod / sdd
            q = torch.fft.irfft(q * ramp / pitch, n=2 * cols)[:, :cols]
            q = torch.nn.functional.pad(q, (1, 2, 1, 2))
            # the scan's normal lies in the slice, det_v along z: u and the depth need y, x only
            depth = (at[1] - S[1])[:, None] * normal[1] + (at[2] - S[2])[None, :] * normal[2]
            grow = sdd / depth
            iu = ((S[1] + grow * (at[1] - S[1])[:, None] - D[1]) * U[1]
                  + (S[2] + grow * (at[2] - S[2])[None, :] - D[2]) * U[2]) / (U @ U) + cols / 2 - 0.5
            iv = (S[0] + grow[None] * (at[0] - S[0])[:, None, None] - D[0]) / V[0] + rows / 2 - 0.5
            iu = iu.clamp(-1, cols)[None].expand(n)
            iv = iv.clamp(-1, rows)
            u0, v0 = torch.floor(iu), torch.floor(iv)
            fu, fv = iu - u0, iv - v0
            base = (v0.long() + 1) * q.shape[1] + u0.long() + 1
            q = q.contiguous().reshape(-1)
            wide = cols + 3
            top = q[base] * (1 - fu) + q[base + 1] * fu
            low = q[base + wide] * (1 - fu) + q[base + wide + 1] * fu
            out += (top * (1 - fv) + low * fv) * (0.5 * dbeta[t] * (sod / depth) ** 2)[None]
        return out


def exact(case, seed):
    ss2 = case["ss"] ** 2
    samples = case["rows"] * case["cols"] * ss2 * case["angles"] * case["ny"] * case["batch"]
    samples *= {"grad": 2, "sirt": 2 * (case["iters"] + 1)}.get(case["op"], 1)
    if samples > EXACT_SAMPLES:
        return None
    inputs = _inputs(case, seed)
    e = _Exact(case)
    if case["op"] == "fp":
        return e.forward(inputs[0])
    if case["op"] == "bp":
        return e.back(inputs[0])
    if case["op"] == "sirt":
        return e.sirt(inputs[0])
    if case["op"] == "fdk":
        return e.fdk(inputs[0])
    x, g = inputs
    if case["batch"] == 1:
        return {"y": e.forward(x), "dx": e.back(g)}
    return {"y": torch.stack([e.forward(a[0]) for a in x])[:, None],
            "dx": torch.stack([e.back(a[0]) for a in g])[:, None]}
