"""The calls that the solver's time is measured on, and what each stands for in use.

A case is one call sequence through the public Python interface (``vfs_b200.stereotgv``):

  form    "host"   one pair, default settings, images and results in host memory, as a program
                   written for the reference class calls it
          "device" one pair, frames already on the GPU, the disparity left there
          "batch"  several pairs in one ``StereoBatch.solve_device``
  fused   the handle's solve path (False: the default path)
  half    FP16 storage (fused path only)
  masked  solveStereoForwardMasked or solveStereoForward
  warm    pyramid level a warm start begins at (-1: every frame solved from zero)
  sizes   "WxH*N" terms joined by "+"

Scenes, fields, solver settings and pyramid depths are those of ``vfs_b200.synth``: 163 degree
fisheye masks, 3 warps x 50 iterations per level.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vfs_b200 import synth
from vfs_b200.stereotgv import StereoBatch, StereoTgv

DEV = "cuda"


def _case(name, form, sizes, fused, half, masked=True, warm=-1):
    return dict(name=name, form=form, sizes=sizes, fused=fused, half=half, masked=masked, warm=warm)


def listed():
    return [
        # the demo program's frame size, ported from the reference without any change
        _case("host 424x400", "host", "424x400*1", False, False),
        # the camera's native frame, the same way
        _case("host 848x800", "host", "848x800*1", False, False),
        # the class's unmasked solve on the default path, frames on the GPU
        _case("unmasked 640x480", "device", "640x480*1", False, False, masked=False),
        # one camera on the fused path, exact and FP16 storage
        _case("fp32 848x800", "device", "848x800*1", True, False),
        _case("fp16 848x800", "device", "848x800*1", True, True),
        # thumbnails: launches and latency only
        _case("fp16 96x64", "device", "96x64*1", True, True),
        # a cropped frame of odd size
        _case("fp16 531x397", "device", "531x397*1", True, True),
        # a sensor larger than the ones the tests use
        _case("fp16 1280x1024", "device", "1280x1024*1", True, True),
        # a camera stream that continues from its last frame and skips the coarsest levels
        _case("warm fp16 424x400", "device", "424x400*1", True, True, warm=1),
        # the benchmark's batch: eight cameras of one rig
        _case("batch fp16 8x848x800", "batch", "848x800*8", True, True),
        # cameras of three sizes with exact storage
        _case("batch fp32 mixed", "batch", "848x800*8+640x480*4+424x400*4", True, False),
    ]


def draw(rng):
    form = rng.choice(["host", "device", "device", "device", "batch"])
    fused = form == "batch" or (form == "device" and rng.random() < 0.8)
    half = fused and rng.random() < 0.6

    def size(lo, hi):
        w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return w, max(48, int(round(w * rng.uniform(0.65, 1.0))))

    if form == "batch":
        terms = []
        for _ in range(rng.randint(1, 3)):
            w, h = size(96, 848)
            terms.append("%dx%d*%d" % (w, h, rng.randint(1, 4)))
        sizes = "+".join(terms)
    else:
        w, h = size(80, 848 if not fused else 1280)
        sizes = "%dx%d*1" % (w, h)
    masked = rng.random() < 0.85
    warm = rng.choice([-1, -1, 0, 1]) if form == "device" and fused and masked else -1
    return dict(form=form, sizes=sizes, fused=fused, half=half, masked=masked, warm=warm)


def _sizes(case):
    out = []
    for term in case["sizes"].split("+"):
        wh, n = term.split("*")
        w, h = wh.split("x")
        out += [(int(w), int(h))] * int(n)
    return out


def _frames(case, seed):
    """Per pair: (fields, frames), one frame more than a solve needs with a warm start.  Pairs
    of one size are frames of one rig's stream (the same calibration, other images)."""
    sizes = _sizes(case)
    per_pair = 2 if case["warm"] >= 0 else 1
    streams = {}
    for k, wh in enumerate(dict.fromkeys(sizes)):
        fields, frames = synth.make_sequence_gpu(wh[0], wh[1], 1000 * (seed % 1000003) + k + 1,
                                                 sizes.count(wh) * per_pair)
        streams[wh] = (fields, frames)
    out, used = [], {}
    for wh in sizes:
        i = used.get(wh, 0)
        used[wh] = i + per_pair
        out.append((wh, streams[wh][0], streams[wh][1][i:i + per_pair]))
    return out


def _levels(w, h):
    n = synth.n_levels_for(w)
    while n > 1 and min(w, h) >> (n - 1) < 16:
        n -= 1
    return n


_STREAM = []


def _stream():
    """The program's one stream: it solves frame after frame."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def _solver(wh, fields, case, stream):
    sp = synth.SOLVER_PARAMS
    s = StereoTgv()
    if case["fused"]:
        s.set_solve_path(True, case["half"])
    s.limitRange = synth.LIMIT_RANGE
    s.initialize(wh[0], wh[1], sp["beta"], sp["gamma"], sp["alpha0"], sp["alpha1"], sp["timestep_lambda"],
                 sp["lambda_"], _levels(*wh), sp["fScale"], sp["nWarpIters"], sp["nSolverIters"])
    s.copyMaskToDevice(fields["mask"])
    s.loadVectorFields(fields["tv"], fields["cv"])
    if stream is not None:
        s.set_stream(stream)
    if case["warm"] >= 0:
        s.set_warm_start(case["warm"])
    return s


def prepare(case, seed):
    pairs = _frames(case, seed)
    if case["form"] == "host":
        wh, fields, frames = pairs[0]
        return dict(case=case, solver=_solver(wh, fields, case, None), frame=frames[0])
    stream = _stream()
    solvers = [_solver(wh, fields, case, stream) for wh, fields, _ in pairs]
    frames = [[tuple(torch.from_numpy(i).cuda() for i in f) for f in fr] for _, _, fr in pairs]
    outs = [torch.empty((h, w), dtype=torch.float32, device=DEV) for (w, h), _, _ in pairs]
    torch.cuda.synchronize()
    st = dict(case=case, solvers=solvers, frames=[f[-1] for f in frames], outs=outs, stream=stream)
    if case["form"] == "batch":
        st["batch"] = StereoBatch(half_storage=case["half"], stream=stream)
        for s in solvers:
            st["batch"].add(s)
    elif case["warm"] >= 0:  # the stream's earlier frame
        solvers[0].copy_images_from_device(*frames[0][0])
        solvers[0].solveStereoForwardMasked()
        torch.cuda.synchronize()
    return st


def run(state):
    case = state["case"]
    if case["form"] == "batch":
        state["batch"].solve_device(state["frames"], state["outs"], masked=case["masked"])
        return state["outs"]
    if case["form"] == "host":
        s = state["solver"]
        s.copyImagesToDevice(*state["frame"])
        (s.solveStereoForwardMasked if case["masked"] else s.solveStereoForward)()
        return [s.copy1DDisparityToHost(), s.copyDisparityToHost()]
    s = state["solvers"][0]
    s.copy_images_from_device(*state["frames"][0])
    (s.solveStereoForwardMasked if case["masked"] else s.solveStereoForward)()
    s.copy_1d_disparity_to_device(state["outs"][0])
    return state["outs"]


def work(case):
    """Bytes: both images and the fields in, the disparity out, each once.  Operations: what one
    primal-dual iteration, one warp and one level need per pixel that is solved (about 100
    in the dual, threshold and primal steps; 400 per warp with its 5x5 median)."""
    sp = synth.SOLVER_PARAMS
    nbytes = flops = 0
    for w, h in _sizes(case):
        n = _levels(w, h)
        top = min(case["warm"], n - 1) if case["warm"] >= 0 else n - 1
        px = sum((w >> l) * (h >> l) for l in range(top + 1))
        r = w * (163.0 / 360.0 if case["masked"] else 1 / 2.2)  # the solved disc, cut by the frame
        rows = (min(w, 2 * math.sqrt(max(0.0, r * r - (y - h / 2) ** 2))) for y in range(h))
        on = sum(rows) / (w * h)
        nbytes += w * h * (2 + 4 + 8 + 8 + 4)
        flops += px * sp["nWarpIters"] * (on * sp["nSolverIters"] * 100 + 400)
        if case["form"] == "host":
            nbytes += w * h * 8
    return dict(bytes=nbytes, flops=flops)


# ---- the same solve in 64 bits, in plain torch ------------------------------------------
def _tex(img, x, y):
    """Bilinear sample at normalised coordinates with mirror addressing; the sampler's
    coordinates have 21 fractional bits and its weights 8."""
    h, w = img.shape[:2]

    def axis(t, n):
        t = torch.floor(t * 2 ** 21) / 2 ** 21 * n - 0.5
        i = torch.floor(t)
        a = torch.floor((t - i) * 256 + 0.5) / 256
        i = i.long()

        def fold(k):
            k = torch.remainder(k, 2 * n)
            return torch.where(k >= n, 2 * n - 1 - k, k)
        return fold(i), fold(i + 1), a

    x0, x1, a = axis(x, w)
    y0, y1, b = axis(y, h)
    if img.dim() == 3:
        a, b = a[..., None], b[..., None]
    return (img[y0, x0] * (1 - a) + img[y0, x1] * a) * (1 - b) + (img[y1, x0] * (1 - a) + img[y1, x1] * a) * b


class _Exact:
    """The coarse-to-fine solve on float64 planes, with the full-size pitched buffers whose
    values the masked form leaves in place."""

    def __init__(self, wh, fields, case):
        self.w, self.h = wh
        self.masked, self.warm = case["masked"], case["warm"]
        self.n = _levels(*wh)
        self.geo = []
        w, h = wh
        for _ in range(self.n):
            self.geo.append((w, h, (w + 31) // 32 * 32))
            w, h = int(w / 2), int(h / 2)
        self.full = self.geo[0][2] * self.geo[0][1]
        f64 = dict(dtype=torch.float64, device=DEV)
        self.f64 = f64
        self.cv = torch.tensor(fields["cv"], **f64)
        self.tv = [torch.tensor(fields["tv"], **f64)]
        self.on = [torch.tensor(fields["mask"], device=DEV) != 0]
        for w, h, _ in self.geo[1:]:
            self.tv.append(self.down(self.tv[-1], w, h))
            src = self.on[-1]  # the sampler's nearest texel, found from single-precision coordinates
            at = [torch.floor((torch.arange(n, dtype=torch.float32, device=DEV) + 0.5) * (torch.ones(1, device=DEV) / n)
                              .float() * 2 ** 21).double() / 2 ** 21 * m for n, m in ((h, src.shape[0]), (w, src.shape[1]))]
            self.on.append(src[at[0].long()][:, at[1].long()])
        self.buf = {k: torch.zeros(self.full, **f64) for k in ("u", "us", "ub", "ubs", "vx", "vy", "vxs", "vys",
                                                               "tpx", "tpy")}
        self.have_prev = False

    def centres(self, w, h):
        y, x = torch.meshgrid(torch.arange(h, **self.f64), torch.arange(w, **self.f64), indexing="ij")
        return (x + 0.5) / w, (y + 0.5) / h

    def down(self, img, w, h):
        x, y = self.centres(w, h)
        dx, dy = 0.25 / w, 0.25 / h
        return 0.25 * (_tex(img, x - dx, y) + _tex(img, x + dx, y) + _tex(img, x, y - dy) + _tex(img, x, y + dy))

    def view(self, name, l):
        w, h, s = self.geo[l]
        return self.buf[name][:h * s].view(h, s)[:, :w]

    def swap(self, *pairs):
        for a, b in pairs:
            self.buf[a], self.buf[b] = self.buf[b], self.buf[a]

    def flat(self, img, l, fill=0.0):
        w, h, s = self.geo[l]
        out = torch.full((h, s), fill, dtype=img.dtype, device=DEV)
        out[:, :w] = img
        return out.view(-1)

    def tensor(self, i0, l):
        sp = synth.SOLVER_PARAMS
        w, h, _ = self.geo[l]
        x, y = self.centres(w, h)
        dx, dy = 1.0 / w, 1.0 / h
        g = 0.25 * _tex(i0, x, y)
        for sx, sy, k in ((-1, -1, 16), (-1, 1, 16), (1, -1, 16), (1, 1, 16), (-1, 0, 8), (1, 0, 8), (0, -1, 8),
                          (0, 1, 8)):
            g = g + _tex(i0, x + sx * dx, y + sy * dy) / k
        if self.masked:
            g = torch.where(self.on[l], g, torch.zeros_like(g))
        c11, c01, c10 = _tex(g, x + dx, y + dy), _tex(g, x, y + dy), _tex(g, x + dx, y)
        gx, gy = c11 - c01, c11 - c10
        mag = torch.sqrt(gx * gx + gy * gy)
        flat = mag < 1e-8
        nx = torch.where(flat, torch.ones_like(gx), gx / mag)
        ny = torch.where(flat, torch.zeros_like(gy), gy / mag)
        wt = torch.clamp(torch.exp(-sp["beta"] * mag ** sp["gamma"]), min=1e-8)
        a, b, c = wt * nx * nx + ny * ny, wt * ny * ny + nx * nx, wt * nx * ny - nx * ny
        keep = torch.arange(w, device=DEV) < (h + 31) // 32 * 32
        keep = (keep & self.on[l]) if self.masked else keep.expand(h, w)
        z = torch.zeros_like(a)
        return [torch.where(keep, t, z) for t in (a, b, c)]

    def median(self, u):
        h, w = u.shape
        rows, cols = torch.arange(-2, h + 2, device=DEV), torch.arange(-2, w + 2, device=DEV)
        p = u[rows.clamp(0, h - 1)][:, cols.clamp(0, w - 1)]
        out = ((rows < 0) | (rows >= h))[:, None] & ((cols < 0) | (cols >= w))[None]
        p = torch.where(out, torch.zeros_like(p), p)
        taps = torch.stack([p[j:j + h, i:i + w] for j in range(5) for i in range(5)], -1)
        return taps.sort(-1).values[..., 12]

    def iterate(self, l, abc, iu, iz):
        sp = synth.SOLVER_PARAMS
        a0, a1, lam = sp["alpha0"], sp["alpha1"], sp["lambda_"]
        w, h, s = self.geo[l]
        n = h * s
        a, b, c = (self.flat(t, l) for t in abc)
        iu, iz = self.flat(iu, l), self.flat(iz, l)
        ones = torch.ones((h, w), dtype=torch.bool, device=DEV)
        inside = self.flat(ones, l, False)
        pos = torch.arange(n, device=DEV)
        col, row = pos % s, pos // s
        eu = (a * a + b * b + 2 * c * c + (a + c) ** 2 + (b + c) ** 2) * a1 * a1
        e1 = a1 * a1 * (b * b + c * c) + 4 * a0 * a0
        e2 = a1 * a1 * (a * a + c * c) + 4 * a0 * a0
        ru = torch.where(eu == 0, torch.ones_like(eu), 1 / eu)

        def west(t, k=1):
            return torch.cat([t.new_zeros(k), t[:-k]])

        def east(t, k=1):
            return torch.cat([t[k:], t.new_zeros(k)])

        if self.masked:
            on = self.flat(self.on[l], l, False)
            r, d, lf, up = east(on), east(on, s), west(on), west(on, s)
            r, lf = r & (col + 1 < w), lf & (col > 0)
            use_r, use_d, zr, zd, has_l, has_u = r, d, ~r, ~d, lf, up
            both_x, neg_x, both_y, neg_y = lf & r, ~r, up & d, ~d
            write = on
        else:
            rad = torch.sqrt((row - h / 2.0) ** 2 + (col - w / 2.0) ** 2)
            on = inside & ~(rad >= w / 2.2)
            use_r, use_d, zr, zd = col + 1 < w, row + 1 < h, col == w - 1, row == h - 1
            has_l, has_u = col > 0, row > 0
            both_x, neg_x, both_y, neg_y = has_l, ~has_l & zr, has_u, ~has_u & zd
            write = inside
        zero = torch.zeros(n, **self.f64)
        px, py, qx, qy, qz, qw = (zero.clone() for _ in range(6))
        B = self.buf
        for k in ("vx", "vy"):
            self.view(k, l).zero_()
        lamru = lam * ru
        tau = sigma = 1.0
        for _ in range(sp["nSolverIters"]):
            mu = 1 / math.sqrt(1 + 0.7 * tau * sp["timestep_lambda"]) if sigma < 1000 else 1.0
            ub, vx, vy, u = B["ub"][:n], B["vx"][:n], B["vy"][:n], B["u"][:n]

            def grad(t, use, k):
                return torch.where(use, east(t, k) - t, t - west(t, k))
            gx, gy = grad(ub, use_r, 1) - vx, grad(ub, use_d, s) - vy
            tx, ty = px + a1 * sigma / 3 * (a * gx + c * gy), py + a1 * sigma / 3 * (c * gx + b * gy)
            m = torch.clamp(torch.sqrt(tx * tx + ty * ty), min=1)
            px, py = torch.where(on, tx / m, zero), torch.where(on, ty / m, zero)
            k = a0 * sigma / 2
            t1, t2 = qx + k * grad(vx, use_r, 1), qy + k * grad(vy, use_d, s)
            t3, t4 = qz + k * grad(vx, use_d, s), qw + k * grad(vy, use_r, 1)
            m = torch.clamp(torch.sqrt(t1 * t1 + t2 * t2 + t3 * t3 + t4 * t4), min=1)
            qx, qy, qz, qw = (torch.where(on, t / m, zero) for t in (t1, t2, t3, t4))
            tpx = torch.where(write, a * px + c * py, B["tpx"][:n])
            tpy = torch.where(write, c * px + b * py, B["tpy"][:n])
            B["tpx"][:n], B["tpy"][:n] = tpx, tpy
            dx = torch.where(both_x, tpx - west(tpx), torch.where(neg_x, -west(tpx), tpx))
            dy = torch.where(both_y, tpy - west(tpy, s), torch.where(neg_y, -west(tpy, s), tpy))
            dun = ub + tau * ru * (dx + dy) - u
            rho = iu * dun + iz
            lt = tau * lamru
            up = lt * iu * iu
            newton = torch.where(iu == 0, dun, dun - rho / iu)
            new = u + torch.where(rho < -up, dun + lt * iu, torch.where(rho > up, dun - lt * iu, newton))
            qcx, qcw = torch.where(zr, zero, qx), torch.where(zr, zero, qw)
            qcy, qcz = torch.where(zd, zero, qy), torch.where(zd, zero, qz)
            gx = qcx - torch.where(has_l, west(qx), zero) + qcz - torch.where(has_u, west(qz, s), zero)
            gy = qcw - torch.where(has_l, west(qw), zero) + qcy - torch.where(has_u, west(qy, s), zero)
            nvx = vx + tau / e1 * (a1 * tpx + a0 * gx)
            nvy = vy + tau / e2 * (a1 * tpy + a0 * gy)
            for name, t in (("us", new), ("ubs", new + mu * (new - ub)), ("vxs", nvx + mu * (nvx - vx)),
                            ("vys", nvy + mu * (nvy - vy))):
                B[name][:n] = torch.where(write, torch.where(on, t, zero), B[name][:n])
            self.swap(("u", "us"), ("ub", "ubs"), ("vx", "vxs"), ("vy", "vys"))
            sigma, tau = sigma / mu, tau * mu

    def solve(self, i0, i1):
        sp = synth.SOLVER_PARAMS
        i0 = [torch.tensor(i0, **self.f64) / 256]
        i1 = torch.tensor(i1, **self.f64) / 256
        x, y = self.centres(self.w, self.h)
        i1 = [_tex(i1, x + self.cv[..., 0] / self.w, y + self.cv[..., 1] / self.h)]
        for w, h, _ in self.geo[1:]:
            i0.append(self.down(i0[-1], w, h))
            i1.append(self.down(i1[-1], w, h))
        B = self.buf
        top = self.n - 1
        if self.warm >= 0 and self.have_prev:
            top = min(self.warm, top)
            for l in range(1, top + 1):
                w, h, _ = self.geo[l]
                self.view("us", l).copy_(self.down(self.view("u", l - 1), w, h) / sp["fScale"])
                self.swap(("u", "us"))
            self.view("ub", top).copy_(self.view("u", top))
        else:
            B["u"].zero_()
            B["ub"].zero_()
        uv = self.view("u", top)[..., None] * self.tv[top]
        for l in range(top, -1, -1):
            w, h, _ = self.geo[l]
            x, y = self.centres(w, h)
            abc = self.tensor(i0[l], l)
            tv = self.tv[l]
            r = torch.sqrt((tv * tv).sum(-1))
            dx, dy = tv[..., 0] / r / w, tv[..., 1] / r / h
            for _ in range(sp["nWarpIters"]):
                wx, wy = x + uv[..., 0] / w, y + uv[..., 1] / h
                tv2, warped = _tex(tv, wx, wy), _tex(i1[l], wx, wy)

                def slope(t):
                    return (_tex(t, x - 2 * dx, y - 2 * dy) - 8 * _tex(t, x - dx, y - dy)
                            + 8 * _tex(t, x + dx, y + dy) - _tex(t, x + 2 * dx, y + 2 * dy)) / 12
                iu = 0.5 * (slope(i0[l]) + slope(warped))
                iz = _tex(warped, x, y) - _tex(i0[l], x, y)
                last = self.view("u", l).clone()
                self.iterate(l, abc, iu, iz)
                u = self.view("u", l)
                if self.masked:
                    u = self.median(u)
                    self.swap(("u", "us"))
                d = torch.clamp(u - last, max=synth.LIMIT_RANGE)
                self.view("u", l).copy_(last + d)
                self.view("ub", l).copy_(last + d)
                uv = uv + d[..., None] * tv2
            if l > 0:
                w, h, _ = self.geo[l - 1]
                x, y = self.centres(w, h)
                self.view("us", l - 1).copy_(_tex(self.view("u", l), x, y) * sp["fScale"])
                self.view("ubs", l - 1).copy_(_tex(self.view("ub", l), x, y) * sp["fScale"])
                uv = _tex(uv, x, y) * sp["fScale"]
                self.swap(("u", "us"), ("ub", "ubs"))
        self.have_prev = True
        return self.view("u", 0).clone(), uv


def exact(case, seed):
    outs = []
    for wh, fields, frames in _frames(case, seed):
        e = _Exact(wh, fields, case)
        for f in frames:
            u, uv = e.solve(*f)
        outs.append(u)
        if case["form"] == "host":
            outs.append(uv)
    return outs
