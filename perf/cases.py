"""Performance cases of the projection, SIRT, sparse-matrix and U-Net paths.

Each case is one pass through a public entry point: the drop-in classes of
``futhark`` (forwardprojection, backprojection, SIRT, SIRT3D), the batched
solver, the CSR system matrix and the U-Net warm starter.  Sizes are those of
the repository's configurations, tests and benchmark, or ragged ones between
them; ``draw`` spreads more cases over the same ranges.

Images are seeded random-ellipse phantoms.  Sinograms that are reconstructed
are the ellipses' analytic line integrals with 1 % Gaussian noise, so they do
not depend on any projector.  ``exact`` restates each operation in 64 bits
with plain torch; rays within 2^-12 of an axis take the column (forward) and
the detector (backward) that the float32 expressions of the reference choose
(forwardprojection.fut:31-56, backprojection.fut:22-65), because there the
rounding of those expressions is part of the operation's definition.
"""
import math
import os
import random

import numpy as np
import torch

import futhark.backprojection
import futhark.backprojection_sparse
import futhark.forwardprojection
import futhark.forwardprojection_sparse
import futhark.SIRT
import futhark.SIRT3D
from synkrotomo_gb300 import runtime as rt
from synkrotomo_gb300.unet import UNet

CHECKPOINT = os.path.join("synkrotomo_gb300", "checkpoints", "unet_n256_a180_noisefree.npz")
BATCH_SIZES = (128, 256, 384, 512)
BATCH_ANGLES = (60, 90, 180, 360)
LAYERS = ((1, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 256), (256, 256), (384, 128),
          (128, 128), (192, 64), (64, 64), (96, 32), (32, 32))


def listed():
    return [
        # sparse-view data (the reference's *_sparse programs: 1-95 angles): a
        # handful of small launches, latency decides
        {"name": "fp_sparse_512x30", "op": "fp", "size": 512, "angles": 30, "det": 725, "dr": 1.0, "arc": "pi"},
        # the geometry of the reference's shipped dataset fpinputf32rad512
        {"name": "fp_512x805", "op": "fp", "size": 512, "angles": 805, "det": 725, "dr": 1.0, "arc": "quarter"},
        # the dense projector microbench, the largest single projection
        {"name": "fp_2048x2048", "op": "fp", "size": 2048, "angles": 2048, "det": 2897, "dr": 1.0, "arc": "pi"},
        {"name": "bp_sparse_512x60", "op": "bp", "size": 512, "angles": 60, "det": 725, "dr": 1.0, "arc": "pi"},
        # a ragged size on a detector of half-pixel pitch over a limited arc
        {"name": "bp_362x271_fine", "op": "bp", "size": 362, "angles": 271, "det": 1025, "dr": 0.5, "arc": "limited"},
        {"name": "bp_2048x2048", "op": "bp", "size": 2048, "angles": 2048, "det": 2897, "dr": 1.0, "arc": "pi"},
        # the plain SIRT configuration: many short iterations on one small slice
        {"name": "sirt_128x128", "op": "sirt", "size": 128, "angles": 128, "det": 182, "iterations": 200},
        # a share of the slice-stack configuration (512 x 512 slices, 360 angles)
        {"name": "sirt3d_512x360x16", "op": "sirt3d", "size": 512, "angles": 360, "det": 725, "slices": 16,
         "iterations": 10},
        # the uneven batch: problems of different size and angle count in one call
        {"name": "sirt_batch_8", "op": "batch", "problems": 8, "pick": 3, "iterations": 20},
        # the precomputed system matrix: A x and A^T y, once each
        {"name": "csr_512x512", "op": "csr", "size": 512, "angles": 512, "det": 725},
        # the trained warm starter on a few sinograms
        {"name": "unet_forward_8", "op": "unet_forward", "size": 256, "batch": 8},
        # one training step at the training configuration's batch
        {"name": "unet_train_32", "op": "unet_train", "size": 256, "batch": 32},
    ]


def _log_even(rng, lo, hi):
    return 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("fp", "fp", "bp", "bp", "sirt", "sirt", "sirt3d", "sirt3d", "batch", "csr", "unet_forward",
                     "unet_train"))
    if op in ("fp", "bp"):
        size = _log_even(rng, 64, 2048)
        dr = rng.choice((1.0, 1.0, 1.0, 1.0, 0.5, 1.5))
        det = int(math.ceil(size * math.sqrt(2.0) / dr)) + rng.choice((0, 1, 7))
        return {"op": op, "size": size, "angles": _log_int(rng, 1, 2048), "det": det, "dr": dr,
                "arc": rng.choice(("pi", "pi", "limited", "quarter"))}
    if op in ("sirt", "sirt3d"):
        size = _log_even(rng, 48, 512)
        det = int(math.ceil(size * math.sqrt(2.0))) + rng.choice((0, 1))
        case = {"op": op, "size": size, "angles": _log_int(rng, 30, 360), "det": det}
        if op == "sirt3d":
            case["slices"] = _log_int(rng, 2, 32)
        per = size * size * case["angles"] * case.get("slices", 1)
        # at most the work of the listed stack
        case["iterations"] = max(1, min(_log_int(rng, 5, 200), int(1.5e10 / per)))
        return case
    if op == "batch":
        return {"op": op, "problems": rng.randint(3, 8), "pick": rng.randint(10, 10 ** 6),
                "iterations": rng.randint(5, 20)}
    if op == "csr":
        size = _log_even(rng, 64, 512)
        return {"op": op, "size": size, "angles": _log_int(rng, 30, 512),
                "det": int(math.ceil(size * math.sqrt(2.0)))}
    return {"op": op, "size": 256, "batch": rng.randint(1, 32)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _angles(count, arc="pi"):
    first, span = {"pi": (0.0, math.pi), "limited": (0.0, 2.0 * math.pi / 3.0),
                   "quarter": (math.pi / 4.0, math.pi / 2.0)}[arc]
    return (first + np.linspace(0.0, span, count, endpoint=False)).astype(np.float32)


def _rhozero(det, dr=1.0):
    return float(np.float32(-(det - 1) / 2.0 * dr))


def _ellipses(size, rng, count=10):
    """Rows (cx, cy, ax, ay, phi, value) of a random-ellipse phantom."""
    half = size / 2.0
    c = rng.uniform(-0.6, 0.6, (count, 2)) * half
    a = rng.uniform(0.05, 0.4, (count, 2)) * half
    return np.column_stack([c, a, rng.uniform(0.0, math.pi, count), rng.uniform(0.0, 1.0, count)])


def _phantom(size, ellipses):
    """The phantom's pixels, float32 [size*size] on the GPU."""
    co = torch.arange(size, dtype=torch.float64, device="cuda") - size / 2.0 + 0.5
    y, x = co[:, None], co[None, :]
    img = torch.zeros(size, size, dtype=torch.float64, device="cuda")
    for cx, cy, ax, ay, phi, val in ellipses:
        c, s = math.cos(phi), math.sin(phi)
        u = (x - cx) * c + (y - cy) * s
        v = (y - cy) * c - (x - cx) * s
        img += val * ((u / ax) ** 2 + (v / ay) ** 2 <= 1.0)
    return img.float().reshape(-1)


def _sinogram(angles, det, ellipses, gen):
    """The phantom's line integrals over rho = x cos - y sin with 1 % noise,
    float32 [a*det] on the GPU."""
    th = torch.from_numpy(angles.astype(np.float64)).cuda()[:, None]
    rho = _rhozero(det) + torch.arange(det, dtype=torch.float64, device="cuda")[None, :]
    b = torch.zeros(th.shape[0], det, dtype=torch.float64, device="cuda")
    for cx, cy, ax, ay, phi, val in ellipses:
        t = rho - (cx * torch.cos(th) - cy * torch.sin(th))
        # the line's normal is (cos, -sin); in the ellipse's axes it is turned by phi
        nu = torch.cos(th) * math.cos(phi) - torch.sin(th) * math.sin(phi)
        nv = -torch.sin(th) * math.cos(phi) - torch.cos(th) * math.sin(phi)
        s2 = (ax * nu) ** 2 + (ay * nv) ** 2
        b += val * 2.0 * ax * ay * torch.sqrt(torch.clamp(s2 - t * t, min=0.0)) / s2
    noise = torch.randn(b.shape, generator=gen, device="cuda", dtype=torch.float32)
    return (b.float() + 0.01 * float(b.max()) * noise).reshape(-1)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _batch_specs(case):
    r = random.Random(int(case["pick"]))
    specs = []
    for _ in range(case["problems"]):
        size, a = r.choice(BATCH_SIZES), r.choice(BATCH_ANGLES)
        arc = "limited" if r.random() < 0.25 else "pi"
        specs.append((size, a, int(math.ceil(size * math.sqrt(2.0))), arc))
    return specs


def _data(case, seed):
    """The input arrays of a case, made from the seed."""
    rng, gen, op = np.random.default_rng(int(seed)), _gen(seed), case["op"]
    if op in ("fp", "bp"):
        ang = _angles(case["angles"], case["arc"])
        if op == "fp":
            x = _phantom(case["size"], _ellipses(case["size"], rng))
        else:
            x = torch.rand(case["angles"] * case["det"], generator=gen, device="cuda", dtype=torch.float32)
        return ang, x
    if op in ("sirt", "sirt3d"):
        ang = _angles(case["angles"])
        b = [_sinogram(ang, case["det"], _ellipses(case["size"], rng), gen) for _ in range(case.get("slices", 1))]
        return ang, torch.cat(b)
    if op == "batch":
        return [(_angles(a, arc), _sinogram(_angles(a, arc), det, _ellipses(size, rng), gen))
                for size, a, det, arc in _batch_specs(case)]
    if op == "csr":
        return (_angles(case["angles"]), _phantom(case["size"], _ellipses(case["size"], rng)),
                torch.rand(case["angles"] * case["det"], generator=gen, device="cuda", dtype=torch.float32))
    # U-Net: a phantom as the target, a smoothed and noisy one as the input
    n, batch = case["size"], case["batch"]
    t = torch.stack([_phantom(n, _ellipses(n, rng)).view(n, n) for _ in range(batch)])
    x = torch.nn.functional.avg_pool2d(t[:, None], 5, 1, 2)[:, 0]
    x = x + 0.02 * torch.randn(x.shape, generator=gen, device="cuda")
    return x.contiguous(), t.contiguous()


def _unet_params(case, seed):
    """The network's flat FP32 parameters: the trained checkpoint for the
    forward pass, a seeded He-normal start for training."""
    if case["op"] == "unet_forward":
        z = np.load(CHECKPOINT)
        bf16 = np.concatenate([m for i, (ci, co) in enumerate(LAYERS)
                               for m in (np.full(9 * ci * co, i > 0), np.zeros(co, bool))] + [np.zeros(33, bool)])
        flat = np.empty(bf16.size, np.float32)
        flat[bf16] = (z["bf16_weights"].astype(np.uint32) << 16).view(np.float32)
        flat[~bf16] = z["fp32_rest"]
        return torch.from_numpy(flat).cuda()
    gen, parts = _gen(seed + 77), []
    for ci, co in LAYERS:
        parts.append(torch.randn(9 * ci * co, generator=gen, device="cuda") * math.sqrt(2.0 / (9 * ci)))
        parts.append(torch.zeros(co, device="cuda"))
    parts.append(0.01 * torch.randn(32, generator=gen, device="cuda"))
    parts.append(torch.zeros(1, device="cuda"))
    return torch.cat(parts)


# ---------------------------------------------------------------------------
# the measured interface
# ---------------------------------------------------------------------------

def prepare(case, seed):
    op, data = case["op"], _data(case, seed)
    if op in ("fp", "bp"):
        ang, x = data
        mod = {("fp", False): futhark.forwardprojection.forwardprojection,
               ("fp", True): futhark.forwardprojection_sparse.forwardprojection_sparse,
               ("bp", False): futhark.backprojection.backprojection,
               ("bp", True): futhark.backprojection_sparse.backprojection_sparse}[op, case["angles"] <= 95]
        last = case["det"] if op == "fp" else case["size"]
        return {"op": op, "prog": mod(), "args": (torch.from_numpy(ang).cuda(), _rhozero(case["det"], case["dr"]),
                                                  case["dr"], last, x)}
    if op == "sirt":
        ang, b = data
        zero = torch.zeros(case["size"] ** 2, device="cuda")
        return {"op": op, "prog": futhark.SIRT.SIRT(),
                "args": (torch.from_numpy(ang).cuda(), _rhozero(case["det"]), 1.0, zero, b, case["iterations"])}
    if op == "sirt3d":
        ang, b = data
        rhos = (_rhozero(case["det"]) + np.arange(case["det"])).astype(np.float32)
        return {"op": op, "prog": futhark.SIRT3D.SIRT3D(), "slices": case["slices"],
                "args": (torch.from_numpy(ang).cuda(), torch.from_numpy(rhos).cuda(), b, case["iterations"],
                         case["size"])}
    if op == "batch":
        probs = [rt.Problem(torch.from_numpy(ang).cuda(), _rhozero(det), 1.0, det, size, b, case["iterations"])
                 for (size, _, det, _), (ang, b) in zip(_batch_specs(case), data)]
        return {"op": op, "problems": probs}
    if op == "csr":
        ang, x, y = data
        m = rt.SystemMatrix(torch.from_numpy(ang).cuda(), _rhozero(case["det"]), 1.0, case["det"], case["size"])
        return {"op": op, "matrix": m, "x": x, "y": y}
    x, t = data
    net = UNet(case["size"], case["batch"], seed=1)
    net.load(_unet_params(case, seed))
    return {"op": op, "net": net, "x": x, "target": t}


def run(state):
    op = state["op"]
    if op in ("fp", "bp", "sirt"):
        return state["prog"].main(*state["args"]).torch()
    if op == "sirt3d":
        return state["prog"].main(*state["args"], nslices=state["slices"]).torch()
    if op == "batch":
        return [p.out for p in rt.sirt_batch(state["problems"])]
    if op == "csr":
        return [state["matrix"].matvec(state["x"]), state["matrix"].rmatvec(state["y"])]
    if op == "unet_forward":
        return state["net"].forward(state["x"])
    loss = state["net"].train_step(state["x"], state["target"], apply=False)
    return [loss, state["net"].gradients()]


# Operation counts: 14 per ray and frame row and 13 per (pixel, ray)
# evaluation plus 13 per pixel and angle, the reference's expressions (multiply-add = 2).
def _fp_flops(size, a, det):
    return 14.0 * a * det * size


def _bp_flops(size, a, dr=1.0):
    return 13.0 * (1 + math.ceil(math.sqrt(2.0) / dr)) * size * size * a


def work(case):
    op = case["op"]
    if op in ("fp", "bp"):
        n, a, d = case["size"], case["angles"], case["det"]
        return {"bytes": 4.0 * (n * n + a * d + a),
                "flops": _fp_flops(n, a, d) if op == "fp" else _bp_flops(n, a, case["dr"])}
    if op in ("sirt", "sirt3d", "batch"):
        specs = (_batch_specs(case) if op == "batch"
                 else [(case["size"], case["angles"], case["det"], "pi")] * case.get("slices", 1))
        return {"bytes": sum(4.0 * (2 * n * n + a * d) for n, a, d, _ in specs),
                "flops": case["iterations"] * sum(_fp_flops(n, a, d) + _bp_flops(n, a) for n, a, d, _ in specs)}
    if op == "csr":
        n, a, d = case["size"], case["angles"], case["det"]
        # a frame row meets about n*(2/pi)*sqrt(2) of the d rays, 1.41 pixels each
        nnz = 4.0 / math.pi * n * n * a
        return {"bytes": 2 * (8.0 * nnz + 4.0 * (n * n + a * d)) + 8.0 * (n * n + a * d), "flops": 4.0 * nnz}
    px = [case["size"] ** 2 // 4 ** lv for lv in (0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0)]
    conv = sum(18.0 * ci * co * p for (ci, co), p in zip(LAYERS, px)) * case["batch"]
    par = sum(9 * ci * co + co for ci, co in LAYERS) + 33
    io = 8.0 * case["batch"] * case["size"] ** 2
    if op == "unet_forward":
        return {"bytes": io + 4.0 * par, "flops": conv}
    return {"bytes": io + 8.0 * par, "flops": 3 * conv - 18.0 * 32 * px[0] * case["batch"]}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

class _Geometry64:
    """Weights of both projectors, angle by angle, in 64 bits."""

    def __init__(self, angles, rhozero, dr, det, size):
        self.n, self.half, self.det, self.dr, self.rz = size, size // 2, det, dr, rhozero
        self.th = [float(t) for t in angles]
        self.rows = torch.arange(size, device="cuda") - self.half

    def _line(self, k):
        c, s = math.cos(self.th[k]), math.sin(self.th[k])
        c32, s32 = np.float32(c), np.float32(s)
        flat = bool(abs(s32) >= abs(c32))
        slope32 = -(c32 if flat else -s32) / (-s32 if flat else c32)
        near = bool(abs(slope32) < np.float32(1.0 / 4096.0))
        return c, s, flat, near

    def _line32(self, c, s, flat):
        """The float32 line of the reference's frame: (cost, sint, lbase, slope)."""
        one = np.float32(1.0)
        c, s = np.float32(c), np.float32(s)
        q = c / s if flat else s / c
        cost, sint = (-s, c) if flat else (c, -s)
        return cost, sint, np.sqrt(one + q * q), -sint / cost

    def fp(self, k):
        """(flat, [(frame column, weight)] * 2), each [rows, detectors]."""
        c, s, flat, near = self._line(k)
        n, half = self.n, self.half
        r = torch.arange(self.det, device="cuda")
        if near:
            cost, _, lbase, slope = (torch.tensor(v, device="cuda") for v in self._line32(c, s, flat))
            rho = self.rz + r.float() * torch.tensor(np.float32(self.dr), device="cuda")
            xb = (self.rows.float() * slope)[:, None] + (rho / cost)[None, :]
            xt = xb + slope
            pb, pt = torch.floor(xb), torch.floor(xt)
            single = pb == pt
            top = torch.maximum(pb, pt)
            diff = torch.where(single, torch.ones_like(xb), xt - xb)
            wb = torch.where(single, lbase, (top - xb) / diff * lbase).double()
            wt = torch.where(single, torch.zeros_like(wb), ((xt - top) / diff * lbase).double())
            c0, c1 = pb.long() + half, pt.long() + half
        else:
            cost, slope = (-s, c / s) if flat else (c, s / c)
            rho = self.rz + r.double() * self.dr
            x = self.rows.double()[:, None] * slope + (rho / cost)[None, :] + min(slope, 0.0)
            fl = torch.floor(x)
            t = torch.clamp((x - fl + abs(slope) - 1.0) / abs(slope), 0.0, 1.0)
            lbase = math.sqrt(1.0 + slope * slope)
            wb, wt = (1.0 - t) * lbase, t * lbase
            c0 = fl.long() + half
            c1 = c0 + 1
        out = []
        for col, w in ((c0, wb), (c1, wt)):
            ok = (col >= 0) & (col < n)
            out.append((torch.where(ok, col, 0), torch.where(ok, w, 0.0)))
        return flat, out

    def bp(self, k):
        """[(detector, weight)], each [image rows, image columns]."""
        c, s, flat, near = self._line(k)
        n = self.n
        rpp = int(math.ceil(np.float32(math.sqrt(2.0)) / np.float32(self.dr)))
        out = []
        if near:
            f = np.float32(0.70710677)
            cost, sint, lbase, slope = self._line32(c, s, flat)
            g = self.rows.float()
            xmin, ymin = (g[:, None].expand(n, n), g[None, :].expand(n, n)) if flat else (
                g[None, :].expand(n, n), g[:, None].expand(n, n))
            fc, fs, cost, sint, lbase, slope, dr, rz = (
                torch.tensor(np.float32(v), device="cuda") for v in (f * cost, f * sint, cost, sint, lbase, slope,
                                                                     self.dr, self.rz))
            x, y = xmin + 0.5 - fc, ymin + 0.5 - fs
            first = torch.ceil((cost * x + sint * y - rz) / dr)
            base = ymin * slope
            for i in range(rpp):
                sp = first + float(i)
                xb = base + (sp * dr + rz) / cost
                xt = xb + slope
                hi, lo = torch.maximum(xb, xt), torch.minimum(xb, xt)
                inside = torch.minimum(torch.clamp(hi - xmin, min=0.0), torch.clamp(xmin + 1.0 - lo, min=0.0))
                diff = hi - lo
                p = torch.where(diff == 0, torch.ones_like(diff), inside / torch.where(diff == 0, 1.0, diff))
                p = torch.where(inside == 0, torch.zeros_like(p), torch.clamp(p, max=1.0))
                out.append((sp.long(), (p * lbase).double()))
        else:
            g = self.rows.double() + 0.5
            rho = g[None, :] * c - g[:, None] * s
            a, b = max(abs(c), abs(s)), min(abs(c), abs(s))
            first = torch.ceil((rho - math.sqrt(0.5) - self.rz) / self.dr)
            for i in range(rpp):
                d = (first + i) * self.dr + self.rz - rho
                w = torch.clamp(((a + b) / 2.0 - d.abs()) / b, 0.0, 1.0) / a
                out.append(((first + i).long(), w))
        kept = []
        for d, w in out:
            ok = (d >= 0) & (d < self.det)
            kept.append((torch.where(ok, d, 0), torch.where(ok, w, 0.0)))
        return kept

    def project(self, img):
        img = img.double().view(self.n, self.n)
        out = torch.empty(len(self.th), self.det, dtype=torch.float64, device="cuda")
        for k in range(len(self.th)):
            flat, terms = self.fp(k)
            frame = img.t().contiguous() if flat else img
            out[k] = sum((w * frame.gather(1, c)).sum(0) for c, w in terms)
        return out.view(-1)

    def project_t(self, y):
        """The transpose of project (the system matrix's A^T y)."""
        y = y.double().view(len(self.th), self.det)
        acc = [torch.zeros(self.n, self.n, dtype=torch.float64, device="cuda") for _ in range(2)]
        for k in range(len(self.th)):
            flat, terms = self.fp(k)
            for c, w in terms:
                acc[flat].scatter_add_(1, c, w * y[k][None, :])
        return (acc[0] + acc[1].t()).reshape(-1)

    def backproject(self, y):
        y = y.double().view(len(self.th), self.det)
        out = torch.zeros(self.n, self.n, dtype=torch.float64, device="cuda")
        for k in range(len(self.th)):
            for d, w in self.bp(k):
                out += w * y[k][d]
        return out.view(-1)

    def matrices(self):
        """Both projectors as sparse matrices [rays x pixels], [pixels x rays]."""
        n, f, b = self.n, ([], [], []), ([], [], [])
        r = torch.arange(self.det, device="cuda")[None, :]
        j = torch.arange(n, device="cuda")[:, None]
        pix = torch.arange(n * n, device="cuda").view(n, n)
        for k in range(len(self.th)):
            flat, terms = self.fp(k)
            for c, w in terms:
                m = w != 0
                f[0].append((k * self.det + r).expand_as(c)[m])
                f[1].append((c * n + j if flat else j * n + c)[m])
                f[2].append(w[m])
            for d, w in self.bp(k):
                m = w != 0
                b[0].append(pix[m])
                b[1].append((k * self.det + d)[m])
                b[2].append(w[m])
        rays = len(self.th) * self.det

        def csr(t, shape):
            i = torch.stack([torch.cat(t[0]), torch.cat(t[1])])
            return torch.sparse_coo_tensor(i, torch.cat(t[2]), shape).coalesce().to_sparse_csr()

        return csr(f, (rays, n * n)), csr(b, (n * n, rays))


def _sirt64(angles, det, size, b, iterations, slices=1):
    g = _Geometry64(angles, _rhozero(det), 1.0, det, size)
    A, B = g.matrices()

    def inverse(v):
        return torch.where(v != 0, 1.0 / torch.where(v != 0, v, 1.0), 0.0)

    R = inverse(A @ torch.ones(size * size, 1, dtype=torch.float64, device="cuda"))
    C = inverse(B @ torch.ones(len(angles) * det, 1, dtype=torch.float64, device="cuda"))
    b = b.double().view(slices, -1).t().contiguous()
    x = torch.zeros(size * size, slices, dtype=torch.float64, device="cuda")
    for _ in range(iterations):
        x = x + C * (B @ (R * (b - A @ x)))
    return x.t().reshape(-1)


def _unet64(flat, x):
    """The network of the warm starter with 64-bit weights and activations."""
    F, pos, conv = torch.nn.functional, 0, []
    for ci, co in LAYERS:
        w = flat[pos:pos + 9 * ci * co].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        conv.append((w, flat[pos + 9 * ci * co:pos + 9 * ci * co + co]))
        pos += 9 * ci * co + co

    def c(i, v):
        return torch.relu(F.conv2d(v, conv[i][0], conv[i][1], padding=1))

    def up(v):
        return F.interpolate(v, scale_factor=2, mode="nearest")

    x = x[:, None]
    e1 = c(1, c(0, x))
    e2 = c(3, c(2, F.max_pool2d(e1, 2)))
    e3 = c(5, c(4, F.max_pool2d(e2, 2)))
    e4 = c(7, c(6, F.max_pool2d(e3, 2)))
    d3 = c(9, c(8, torch.cat([up(e4), e3], 1)))
    d2 = c(11, c(10, torch.cat([up(d3), e2], 1)))
    d1 = c(13, c(12, torch.cat([up(d2), e1], 1)))
    return (x + flat[pos + 32] + F.conv2d(d1, flat[pos:pos + 32].view(1, 32, 1, 1)))[:, 0]


def exact(case, seed):
    op, data = case["op"], _data(case, seed)
    if op in ("fp", "bp"):
        g = _Geometry64(data[0], _rhozero(case["det"], case["dr"]), case["dr"], case["det"], case["size"])
        return g.project(data[1]) if op == "fp" else g.backproject(data[1])
    if op in ("sirt", "sirt3d"):
        return _sirt64(data[0], case["det"], case["size"], data[1], case["iterations"], case.get("slices", 1))
    if op == "batch":
        return [_sirt64(ang, det, size, b, case["iterations"])
                for (size, _, det, _), (ang, b) in zip(_batch_specs(case), data)]
    if op == "csr":
        g = _Geometry64(data[0], _rhozero(case["det"]), 1.0, case["det"], case["size"])
        return [g.project(data[1]), g.project_t(data[2])]
    x, t = data[0].double(), data[1].double()
    flat = _unet_params(case, seed).double()
    if op == "unet_forward":
        with torch.no_grad():
            return _unet64(flat, x)
    flat.requires_grad_(True)
    loss = torch.mean((_unet64(flat, x) - t) ** 2)
    loss.backward()
    return [loss.detach(), flat.grad]
