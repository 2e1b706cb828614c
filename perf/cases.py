"""Performance cases of the distance-driven projectors.

Every case is one call, or one gradient step, of the public projector classes on synthetic scans:
volumes of seeded random ellipsoids, and sinograms that are the analytic line integrals of such
ellipsoids plus 1 % noise.  ``listed()`` names the cases, ``draw()`` makes more of the same ranges,
``exact()`` evaluates the same operators in float64 with plain torch.

Fields of a case: ``scan`` (parallel, flat, arc or helical), ``what`` (the pass, see ``run``),
``W H D`` voxels of ``dx dx dz`` mm (``D`` = 0: a 2D image), ``Nu Nv`` detector cells of ``du dv`` mm,
``V`` views over ``arc`` turns, ``sod sdd`` mm, ``batch`` volumes, ``dtype`` of the stored data.
"""
import math

import torch

from xrecon_b200 import geometry as G
from xrecon_b200.projector import HelicalProjector3d, Projector2d, Projector3d
from xrecon_b200.ragged import RaggedFBP2d

DEVICE = "cuda"
DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
FROM_IMAGE = ("project", "backproject_t", "backproject_weighted_t")
FROM_SINO = ("project_t", "backproject", "backproject_weighted")


def _case(scan, what, size, cells, views, name=None, dx=1.0, dz=None, du=1.0, dv=None, sod=500.0, sdd=1000.0,
          arc=1.0, batch=1, dtype="float32", parker=False, pitch=0.0):
    c = dict(scan=scan, what=what, W=size[0], H=size[1], D=size[2] if len(size) > 2 else 0,
             Nu=cells[0], Nv=cells[1] if len(cells) > 1 else 0, V=views, dx=dx, dz=dz or dx, du=du, dv=dv or du,
             sod=sod, sdd=sdd, arc=arc, batch=batch, dtype=dtype, parker=parker, pitch=pitch)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One sparse-view projection of a small image, as a data-consistency layer calls it many times: launch latency.
        _case("flat", "project", (64, 64), (96,), 30, "fan_flat_small_project", dx=4.0, du=8.0),
        # The 2D fan-flat configuration: ramp FBP of 720 views of 256 cells to 256 x 256.
        _case("flat", "fbp", (256, 256), (256,), 720, "fan_flat_fbp", dx=1.0, du=2.0),
        # Learned 2D reconstruction: a batch of 512 x 512 slices on a curved 736-cell detector, forward and backward.
        _case("arc", "gradient", (512, 512), (736,), 360, "fan_arc_batch_gradient", dx=0.7, du=1.2858, sod=595.0,
              sdd=1085.6, batch=8),
        # 64 slices of mixed sizes scanned and reconstructed in one persistent launch (16 of them here).
        dict(name="fan_arc_ragged", scan="arc", what="ragged", count=16, geometry=4),
        # The circular FDK configuration.
        _case("flat", "fbp", (256, 256, 64), (384, 96), 720, "cone_flat_fdk", du=1.5),
        # A learned short-scan FDK at odd sizes: Parker weights, forward and the gradient of the sinogram.
        _case("flat", "fbp_gradient", (201, 189, 51), (277, 83), 251, "cone_flat_odd_fdk_gradient", du=2.3, dv=1.5,
              arc=0.66, parker=True),
        # The least-squares configuration: 8 volumes, curved detector, residual and gradient of one step.
        _case("arc", "gradient", (128, 128, 32), (256, 64), 360, "cone_arc_batch_gradient", du=1.5, batch=8),
        # Half-precision storage: simulate a scan and backproject it.
        _case("flat", "project_backproject", (256, 256, 128), (384, 160), 360, "cone_flat_half", du=1.5, dtype="float16"),
        # The largest circular scan, projected and backprojected: the headline workload's two operators.
        _case("flat", "project", (512, 512, 256), (1024, 256), 1440, "cone_flat_large_project", dx=0.75, du=0.8,
              sod=595.0, sdd=1085.0),
        _case("flat", "backproject", (512, 512, 256), (1024, 256), 1440, "cone_flat_large_backproject", dx=0.75,
              du=0.8, sod=595.0, sdd=1085.0),
        # A clinical helical scan, five turns: helical FDK.
        _case("helical", "fbp", (512, 512, 128), (736, 64), 5760, "helical_fdk", dx=0.7, dz=0.8, du=1.2858,
              dv=1.0947, sod=595.0, sdd=1085.6, arc=5.0, pitch=30.7),
        # Iterative helical reconstruction on a coarse grid: residual and gradient of one step.
        _case("helical", "gradient", (160, 160, 48), (240, 32), 720, "helical_gradient", dx=2.2, dz=2.0, du=4.0,
              dv=2.2, sod=595.0, sdd=1085.6, arc=3.0, pitch=30.7),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: 2D, circular 3D, helical or ragged, any size between the smallest and the largest listed."""
    kind = rng.choice(["2d", "2d", "3d", "3d", "3d", "helical", "ragged"])
    if kind == "ragged":
        return dict(scan="arc", what="ragged", count=rng.randint(2, 16), geometry=rng.randrange(1, 10000))
    dtype = rng.choice(["float32"] * 4 + ["float16", "bfloat16"])
    if kind == "2d":
        scan = rng.choice(["flat", "arc", "parallel"])
        n = _log(rng, 64, 512)
        size, cells, views = (n, max(64, int(n * rng.uniform(0.8, 1.0)))), (_log(rng, 96, 736),), _log(rng, 30, 720)
        batch = rng.choice([1, 1, 2, 5, 8])
    else:
        scan = "helical" if kind == "helical" else rng.choice(["flat", "flat", "arc", "parallel"])
        n = _log(rng, 64, 400)
        size = (n, max(48, int(n * rng.uniform(0.8, 1.0))), max(16, int(n * rng.uniform(0.15, 0.5))))
        cells, views = (_log(rng, n, 2 * n), max(24, int(size[2] * rng.uniform(0.7, 1.5)))), _log(rng, 60, 900)
        batch = rng.choice([1, 1, 1, 2, 4])
    what = rng.choice(["project", "gradient", "fbp", "backproject"] * 2 + list(FROM_IMAGE + FROM_SINO)
                      + ["fbp_gradient", "project_backproject"])
    parker = scan in ("flat", "arc") and what in ("fbp", "fbp_gradient") and rng.random() < 0.4
    if what in ("gradient", "fbp_gradient") or scan == "helical":
        dtype = "float32"
    dx = rng.uniform(150.0, 350.0) / size[0]
    sod, sdd = (500.0, 1000.0) if rng.random() < 0.5 else (595.0, 1085.6)
    mag = 1.0 if scan == "parallel" else sdd / sod
    du = size[0] * dx * rng.uniform(1.2, 1.5) * mag / cells[0]
    dz = dx * rng.uniform(0.8, 1.3)
    dv = size[2] * dz * rng.uniform(0.9, 1.3) * mag / cells[1] if len(size) > 2 else du
    arc, pitch = (0.72 if parker else rng.choice([1.0, 1.0, 0.5])), 0.0
    if scan == "helical":
        pitch, arc, dv = size[2] * dz * rng.uniform(0.4, 0.8), rng.choice([2.0, 3.0]), 0.6 * dv
    return _case(scan, what, size, cells, views, dx=dx, dz=dz, du=du, dv=dv, sod=sod, sdd=sdd, arc=arc, batch=batch,
                 dtype=dtype, parker=parker, pitch=pitch)


# ------------------------------------------------------------------ inputs

def _angles(c):
    return (torch.arange(c["V"], dtype=torch.float64) * (2 * math.pi * c["arc"] / c["V"])).float()


def _source_pos(c):
    """[4, V]: the helical source's z, centred on the volume; no flying focal spot."""
    turns = _angles(c).double() / (2 * math.pi)
    z = c["pitch"] * (turns - 0.5 * turns[-1])
    return torch.cat([z[None], torch.zeros(3, c["V"], dtype=torch.float64)]).float()


def _projector(c):
    two = c["D"] == 0
    det = G.Detector2d(c["Nu"], c["du"]) if two else G.Detector3d((c["Nu"], c["Nv"]), (c["du"], c["dv"]))
    vol = G.Volume2d((c["W"], c["H"]), c["dx"]) if two else G.Volume3d((c["W"], c["H"], c["D"]), (c["dx"], c["dx"], c["dz"]))
    if c["scan"] == "helical":
        geo = G.HelicalConeBeam3d(det, c["sod"], c["sdd"], "arc", pitch=c["pitch"])
        return HelicalProjector3d(vol, geo).to(DEVICE)
    if c["scan"] == "parallel":
        geo = (G.ParallelBeam2d if two else G.ParallelBeam3d)(det)
    else:
        geo = (G.FanBeam2d if two else G.ConeBeam3d)(det, c["sod"], c["sdd"], c["scan"])
    return (Projector2d if two else Projector3d)(vol, geo).to(DEVICE)


def _ellipsoids(c, gen, count=12):
    """Per ellipsoid: density, centre [3] and semi-axes [3] in mm, inside the image."""
    ext = torch.tensor([c["W"] * c["dx"], c["H"] * c["dx"], max(1, c["D"]) * c["dz"]]) * 0.5
    r = torch.rand(count, 7, generator=gen)
    density = 0.2 + 0.8 * r[:, 0]
    return density, (r[:, 1:4] * 1.2 - 0.6) * ext * (1.0 if c["D"] else torch.tensor([1.0, 1.0, 0.0])), \
        (0.05 + 0.35 * r[:, 4:7]) * ext


def _volume(c, seed, count=12):
    gen = torch.Generator().manual_seed(seed)
    x = ((torch.arange(c["W"]) + 0.5 - 0.5 * c["W"]) * c["dx"]).to(DEVICE)
    y = ((0.5 * c["H"] - 0.5 - torch.arange(c["H"])) * c["dx"]).to(DEVICE)
    z = ((torch.arange(max(1, c["D"])) + 0.5 - 0.5 * max(1, c["D"])) * c["dz"]).to(DEVICE)
    out = torch.zeros(c["batch"], max(1, c["D"]), c["H"], c["W"], device=DEVICE)
    for b in range(c["batch"]):
        density, centre, axes = _ellipsoids(c, gen, count)
        for d, m, a in zip(density.tolist(), centre.tolist(), axes.tolist()):
            inside = (((z - m[2]) / a[2]) ** 2)[:, None, None] + (((y - m[1]) / a[1]) ** 2)[None, :, None] \
                + (((x - m[0]) / a[0]) ** 2)[None, None, :] <= 1.0
            out[b].add_(inside, alpha=d)
    out = out[:, None] if c["D"] else out
    return out.to(DTYPES[c["dtype"]])


def _sinogram(c, seed, count=12):
    """Line integrals of the ellipsoids from the source to every cell centre, plus 1 % noise."""
    gen = torch.Generator().manual_seed(seed)
    noise = torch.Generator(device=DEVICE).manual_seed(seed + 1)
    beta = _angles(c).to(DEVICE)
    zs = _source_pos(c)[0].to(DEVICE) if c["scan"] == "helical" else torch.zeros_like(beta)
    Nu, Nv = c["Nu"], max(1, c["Nv"])
    u = (torch.arange(Nu, device=DEVICE) + 0.5 - 0.5 * Nu) * c["du"]
    v = (torch.arange(Nv, device=DEVICE) + 0.5 - 0.5 * Nv) * (c["dv"] if c["Nv"] else 0.0)
    out = torch.zeros(c["batch"], c["V"], Nv, Nu, device=DEVICE)
    step = max(1, int(3e7 // (Nu * Nv)))
    for b in range(c["batch"]):
        density, centre, axes = _ellipsoids(c, gen, count)
        for i in range(0, c["V"], step):
            s, k = torch.sin(beta[i:i + step])[:, None, None], torch.cos(beta[i:i + step])[:, None, None]
            z0 = zs[i:i + step, None, None]
            if c["scan"] == "parallel":
                p, d = (u * k, u * s, v[:, None].expand(Nv, Nu) + z0), (s, -k, torch.zeros_like(z0))
            else:
                p = (-s * c["sod"], k * c["sod"], z0)
                a = u / c["sdd"] if c["scan"] != "flat" else torch.atan(u / c["sdd"])
                r = 1.0 if c["scan"] != "flat" else 1.0 / torch.cos(a)
                d = (torch.sin(a) * k * r + s * torch.cos(a) * r, torch.sin(a) * s * r - k * torch.cos(a) * r,
                     (v[:, None] / c["sdd"]).expand(Nv, Nu))
            length = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
            for w, m, ax in zip(density.tolist(), centre.tolist(), axes.tolist()):
                aa = sum((d[q] / ax[q]) ** 2 for q in range(3))
                bb = sum((p[q] - m[q]) * d[q] / ax[q] ** 2 for q in range(3))
                cc = sum(((p[q] - m[q]) / ax[q]) ** 2 for q in range(3)) - 1.0
                out[b, i:i + step].add_(torch.sqrt((bb * bb - aa * cc).clamp_min_(0.0)) / aa * length, alpha=2.0 * w)
    out += torch.randn(out.shape, generator=noise, device=DEVICE) * (0.01 * float(out.max()))
    out = out[:, None] if c["Nv"] else out.transpose(1, 2).contiguous()
    return out.to(DTYPES[c["dtype"]])


def _ragged_instances(c):
    """The fan-arc batch of mixed sizes: N in {128 .. 512} over 512 mm, 180-720 views, 192-736 cells."""
    gen = torch.Generator().manual_seed(c["geometry"])
    got = []
    for _ in range(c["count"]):
        r = torch.rand(5, generator=gen).tolist()
        n = (128, 192, 256, 384, 512)[int(r[0] * 5)]
        sod = 400.0 + 200.0 * r[4]
        got.append(_case("arc", "fbp", (n, n), (int(192 + r[2] * 544),), int(180 + r[1] * 540), dx=512.0 / n,
                         du=1.0 + r[3], sod=sod, sdd=2 * sod))
    return got


def prepare(case, seed):
    c = case
    if c["what"] == "ragged":
        parts = _ragged_instances(c)
        plan = RaggedFBP2d([_projector(p) for p in parts], [_angles(p) for p in parts])
        return dict(what="ragged", plan=plan, images=[_volume(p, 1000 * seed + i)[0, 0] for i, p in enumerate(parts)])
    s = dict(what=c["what"], projector=_projector(c), angles=_angles(c).to(DEVICE), parker=c["parker"],
             extra=(_source_pos(c).to(DEVICE),) if c["scan"] == "helical" else ())
    if c["what"] in FROM_IMAGE + ("gradient", "project_backproject"):
        s["image"] = _volume(c, 1000 * seed)
    if c["what"] in FROM_SINO + ("fbp", "gradient", "fbp_gradient"):
        s["sino"] = _sinogram(c, 1000 * seed + 500)
    if c["what"] == "fbp_gradient":
        s["image"] = _volume(c, 1000 * seed)
    if c["what"] == "gradient":
        s["image"].requires_grad_(True)
    if c["what"] == "fbp_gradient":
        s["sino"].requires_grad_(True)
    return s


OPERATORS = {"project": "projection", "project_t": "projection_t", "backproject": "backprojection",
             "backproject_weighted": "backprojection_weighted", "backproject_t": "backprojection_t",
             "backproject_weighted_t": "backprojection_weighted_t"}


def run(state):
    s, what = state, state["what"]
    if what == "ragged":
        return s["plan"](s["images"])
    P, more = s["projector"], (s["angles"],) + s["extra"]
    if what in FROM_IMAGE:
        return getattr(P, OPERATORS[what])(s["image"], *more)
    if what in FROM_SINO:
        return getattr(P, OPERATORS[what])(s["sino"], *more)
    if what == "project_backproject":
        y = P.projection(s["image"], *more)
        return y, P.backprojection(y, *more)
    options = {"parker": True} if s["parker"] else {}
    if what == "fbp":
        return P.filtered_backprojection(s["sino"], *more, **options)
    if what == "gradient":  # one step of least squares
        y = P.projection(s["image"], *more)
        residual = y - s["sino"]
        loss = 0.5 * (residual * residual).sum()
        return y.detach(), torch.autograd.grad(loss, s["image"])[0]
    recon = P.filtered_backprojection(s["sino"], *more, **options)
    loss = 0.5 * ((recon - s["image"]) ** 2).sum()
    return recon.detach(), torch.autograd.grad(loss, s["sino"])[0]


def _voxel_views(c):
    return c["batch"] * c["W"] * c["H"] * max(1, c["D"]) * c["V"]


def work(case):
    """Images and sinograms read or written once; 4 operations per voxel, view and operator (two multiply-adds: one
    detector column and one row boundary)."""
    c = case
    if c["what"] == "ragged":
        parts = _ragged_instances(c)
        return {"bytes": sum(4.0 * (2 * p["W"] * p["H"] + p["V"] * p["Nu"]) for p in parts),
                "flops": sum(8.0 * _voxel_views(p) for p in parts)}
    size = 4.0 if c["dtype"] == "float32" else 2.0
    image, sino = c["batch"] * c["W"] * c["H"] * max(1, c["D"]), c["batch"] * c["V"] * c["Nu"] * max(1, c["Nv"])
    images, sinos, ops = {"gradient": (2, 2, 2), "fbp_gradient": (2, 2, 2), "project_backproject": (2, 1, 2)}.get(
        c["what"], (1, 1, 1))
    return {"bytes": size * (images * image + sinos * sino), "flops": 4.0 * ops * _voxel_views(c)}


# ------------------------------------------------- the same operators in float64

class _Exact:
    """Distance-driven operators in float64.

    Per view, detector-column boundaries and pixel edges are mapped from the source onto the image axis nearer to the
    detector; a cell's value is the overlap-weighted sum over the lines of pixels parallel to that axis.  Both overlaps
    are differences of a running integral: along the line at the column boundaries, along z at the row boundaries.
    Curved detectors have float32 boundary angles (k - Nu/2) du + beta and float32 axis positions, as the scan's
    definition gives them; a helical scan's are not rounded.
    """

    def __init__(self, c):
        self.c = c
        f = lambda x: float(torch.tensor(x, dtype=torch.float32))  # noqa: E731 - options are float32
        self.two = c["D"] == 0
        self.D, self.Nv = max(1, c["D"]), max(1, c["Nv"])
        self.dx, self.dz = f(c["dx"]), f(c["dz"])
        self.sod, self.sdd = f(c["sod"]), f(c["sdd"])
        self.arc, self.flat = c["scan"] in ("arc", "helical"), c["scan"] == "flat"
        du = c["du"]
        if self.flat:
            du = f(du * c["sod"] / c["sdd"]) if self.two else f(du) * self.sod / self.sdd
        elif self.arc:
            du = f(2.0 * math.atan(du / c["sdd"] / 2.0) if self.two else du / c["sdd"])
        else:
            du = f(du)
        self.du, self.dv = du, f(c["dv"]) * (self.sod / self.sdd if self.flat else 1.0)
        angles = _angles(c)
        cos, sin = torch.cos(angles), torch.sin(angles)
        self.use_x = cos * cos > 0.5
        self.keep = torch.where(self.use_x, cos >= 0, sin >= 0)
        self.angles = angles
        self.zs = _source_pos(c)[0].double() if c["scan"] == "helical" else torch.zeros(c["V"], dtype=torch.float64)
        per = max(c["W"], c["H"]) * c["Nu"] * (max(self.D, self.Nv) + 1)
        n = max(1, int(2.5e7 // per))
        self.chunks = []
        for flag in (True, False):
            idx = torch.nonzero(self.use_x == flag).reshape(-1)
            self.chunks += [(flag, part) for part in idx.split(n)] if len(idx) else []

    def _columns(self, beta, use_x, keep, k, src, centres=False):
        """Axis positions of the column boundaries k, or (x, y) of the column centres."""
        c, par = self.c, self.c["scan"] == "parallel"
        sg = torch.where(keep[:, None], k - 0.5 * c["Nu"], 0.5 * c["Nu"] - k)
        co, si = torch.cos(beta)[:, None], torch.sin(beta)[:, None]
        if self.arc:
            if c["scan"] == "helical":
                a = sg * self.du + beta[:, None]
            else:
                a = (sg.float() * torch.tensor(self.du, dtype=torch.float32) + beta.float()[:, None]).double()
            if centres:
                return torch.sin(a) * self.sdd + src[0], -torch.cos(a) * self.sdd + src[1]
            t = torch.tan(a)
            if c["scan"] == "helical":
                return src[0] + src[1] * t if use_x else src[1] + src[0] / t
            b = beta.float()[:, None]
            sx, sy, t = -torch.sin(b) * self.sod, torch.cos(b) * self.sod, t.float()
            return (sx + sy * t if use_x else sy + sx / t).double()
        u = sg * self.du
        if centres:
            return u * co, u * si
        if par:
            return u / co if use_x else u / si
        return self._map(src, use_x, u * co, u * si)

    @staticmethod
    def _map(src, use_x, x, y):
        return (src[0] * y - src[1] * x) / (y - src[1]) if use_x else (src[1] * x - src[0] * y) / (x - src[0])

    def _views(self, use_x, idx):
        c, dev, par = self.c, DEVICE, self.c["scan"] == "parallel"
        beta, keep = self.angles[idx].double().to(dev), self.keep[idx].to(dev)
        co, si = torch.cos(beta)[:, None], torch.sin(beta)[:, None]
        src = (-si * self.sod, co * self.sod)
        k = torch.arange(c["Nu"] + 1, device=dev, dtype=torch.float64)[None]
        Dk = self._columns(beta, use_x, keep, k, src)
        if par:
            M = torch.ones(len(idx), c["Nu"], device=dev, dtype=torch.float64)
        else:
            cx, cy = self._columns(beta, use_x, keep, k[:, :-1] + 0.5, src, True)
            M = src[1] / (src[1] - cy) if use_x else src[0] / (src[0] - cx)
        L, P = (c["H"], c["W"]) if use_x else (c["W"], c["H"])
        line = torch.arange(L, device=dev, dtype=torch.float64)[None]
        perp = (0.5 * L - line - 0.5) * self.dx if use_x else (line - 0.5 * L + 0.5) * self.dx
        e0, e1 = -0.5 * P * self.dx, 0.5 * P * self.dx
        if par:
            shift = (si / co if use_x else co / si) * perp
            X0, X1, Mv = shift + e0, shift + e1, torch.ones_like(shift)
        else:
            ends = [self._map(src, use_x, torch.full_like(perp, e), perp) if use_x
                    else self._map(src, use_x, perp, torch.full_like(perp, e)) for e in (e0, e1)]
            X0, X1 = ends
            Mv = src[1] / (src[1] - perp) if use_x else src[0] / (src[0] - perp)
        return dict(idx=idx, use_x=use_x, keep=keep, src=src, D=Dk, M=M, X0=X0, xw=(X1 - X0) / P, Mv=Mv, P=P, L=L,
                    zs=self.zs[idx].to(dev)[:, None])

    def _rows(self, v):
        r = torch.arange(self.Nv + 1, device=DEVICE, dtype=torch.float64) - 0.5 * self.Nv
        return v["M"][:, None, :] * (r * self.dv)[None, :, None]  # [n, Nv + 1, Nu], from the source's z

    def overlaps(self, image, v, line_scale):
        """[D, H, W] -> [n, Nv, Nu]: sum over lines of line_scale x pixel overlap x slice overlap (in pixels, slices)."""
        lines = image.permute(1, 0, 2) if v["use_x"] else image.permute(2, 0, 1).flip(2)  # [L, D, P]
        n = len(v["idx"])
        f = ((v["D"][:, None, :] - v["X0"][:, :, None]) / v["xw"][:, :, None]).clamp(0, v["P"])  # [n, L, Nu + 1]
        i = f.floor().clamp_(max=v["P"] - 1)
        run_ = torch.nn.functional.pad(lines.cumsum(2), (1, 0))
        at = i.long()[:, :, None, :].expand(-1, -1, self.D, -1)
        at_edge = torch.gather(run_[None].expand(n, -1, -1, -1), 3, at)
        cut = torch.gather(lines[None].expand(n, -1, -1, -1), 3, at)
        J = (at_edge + (f - i)[:, :, None, :] * cut).diff(dim=3)  # [n, L, D, Nu]
        if not self.two:
            z0 = (-0.5 * self.D * self.dz - v["zs"])[:, :, None, None]
            u = ((self._rows(v)[:, None] / v["Mv"][:, :, None, None] - z0) / self.dz).clamp(0, self.D)
            j = u.floor().clamp_(max=self.D - 1)
            run_ = torch.nn.functional.pad(J.cumsum(2), (0, 0, 1, 0))
            at = j.long()
            J = (torch.gather(run_, 2, at) + (u - j) * torch.gather(J, 2, at)).diff(dim=2)
        return (J * line_scale[:, :, None, None]).sum(1)

    def _view_op(self, image, v, op):
        """project: A.  backproject_t: the transpose of B.  backproject_weighted_t: of Bw, whose pixel weight is in the image."""
        c, par = self.c, self.c["scan"] == "parallel"
        if op == "project" or (par and not self.two):
            depth = 1.0 if self.two else v["Mv"] * self.dz
            y = self.overlaps(image, v, v["xw"] * depth)
            dD = v["D"].diff(dim=1)[:, None]
            if par:
                scale = self.dx / (self.du * (1.0 if self.two else self.dv)) * torch.ones_like(dD)
            else:
                spar, sperp = (v["src"][0], v["src"][1]) if v["use_x"] else (v["src"][1], v["src"][0])
                a = 0.5 * (v["D"][:, 1:] + v["D"][:, :-1])[:, None] - spar[:, None]
                rows = self._rows(v)
                dZ = 1.0 if self.two else rows.diff(dim=1)
                b = 0.0 if self.two else 0.5 * (rows[:, 1:] + rows[:, :-1]) + v["zs"][:, None]
                scale = self.dx / (dD * dZ) * torch.sqrt(a * a + b * b + sperp[:, None] ** 2) / sperp.abs()[:, None]
            y = y * scale
        else:
            if self.c["scan"] == "helical":
                width = self.sod * self.du
            else:
                width = 2.0 * self.sod * math.tan(0.5 * self.du) if self.arc else self.du
            y = self.overlaps(image, v, width * torch.ones_like(v["Mv"]))
        return torch.where(v["keep"][:, None, None], y, y.flip(2))

    def _weight(self, v, k):
        """[H, W] FBP weight of view k of the chunk."""
        c = self.c
        x = (torch.arange(c["W"], device=DEVICE, dtype=torch.float64) + 0.5 - 0.5 * c["W"])[None] * self.dx
        y = (0.5 * c["H"] - 0.5 - torch.arange(c["H"], device=DEVICE, dtype=torch.float64))[:, None] * self.dx
        sx, sy = v["src"][0][k], v["src"][1][k]
        if self.arc:
            return 1.0 / ((sx - x) ** 2 + (sy - y) ** 2)
        return (self.sod / (self.sod - (sx * x + sy * y) / self.sod)) ** 2 if self.flat else torch.ones_like(x + y)

    def from_image(self, image, op):
        """[B, D, H, W] -> [B, V, Nv, Nu]"""
        c = self.c
        out = torch.zeros(c["batch"], c["V"], self.Nv, c["Nu"], device=DEVICE, dtype=torch.float64)
        weighted = op == "backproject_weighted_t" and c["scan"] != "parallel"
        for flag, idx in self.chunks:
            for part in idx.split(1) if weighted else [idx]:
                v = self._views(flag, part)
                for b in range(c["batch"]):
                    x = image[b] * self._weight(v, 0) if weighted else image[b]
                    out[b, part.to(DEVICE)] = self._view_op(x, v, op)
        return out

    def from_sino(self, sino, op):
        """[B, V, Nv, Nu] -> [B, D, H, W]: the transpose, by differentiating the linear operator."""
        c = self.c
        fwd = {"project_t": "project", "backproject": "backproject_t", "backproject_weighted": "backproject_weighted_t"}[op]
        weighted = op == "backproject_weighted" and c["scan"] != "parallel"
        out = torch.zeros(c["batch"], self.D, c["H"], c["W"], device=DEVICE, dtype=torch.float64)
        x = torch.zeros(self.D, c["H"], c["W"], device=DEVICE, dtype=torch.float64, requires_grad=True)
        for flag, idx in self.chunks:
            for part in idx.split(1) if weighted else [idx]:
                with torch.no_grad():
                    v = self._views(flag, part)
                y = self._view_op(x, v, fwd)
                for b in range(c["batch"]):
                    g, = torch.autograd.grad(y, x, sino[b, part.to(DEVICE)], retain_graph=b + 1 < c["batch"])
                    out[b] += g * self._weight(v, 0) if weighted else g
        return out

    # -- FBP
    def _cell_weight(self):
        c, k = self.c, torch.arange(self.c["Nu"], device=DEVICE, dtype=torch.float64) + 0.5 - 0.5 * self.c["Nu"]
        s = k * self.du
        w = torch.ones_like(s)
        if self.flat:
            w = self.sod / torch.sqrt(s * s + self.sod ** 2)
        elif self.arc:
            w = torch.cos(s)
        w = w[None, None].expand(c["V"], self.Nv, -1)
        if c["parker"]:
            gamma = s if self.arc else torch.atan2(s, torch.full_like(s, self.sod))
            beta = (self.angles - self.angles[0]).double().to(DEVICE)[:, None]
            span, gmax = beta[-1].abs(), gamma.abs().max()
            over = torch.clamp((span - math.pi) / 2, min=gmax)
            left, right = 2 * (over - gamma), span - 2 * (over + gamma)
            ramp = lambda t, width: torch.sin(0.5 * math.pi * t / width.clamp(min=1e-7)) ** 2  # noqa: E731
            p = torch.where(beta < left, ramp(beta, left), torch.ones_like(beta))
            p = torch.where(beta > right, ramp(span - beta, span - right), p)
            w = w * p[:, None, :]
        return w

    def _filter(self, rows):
        Nu, n = self.c["Nu"], torch.arange(self.c["Nu"], device=DEVICE, dtype=torch.float64)
        h = torch.where(n % 2 == 1, -1.0 / (math.pi * self.du * n.clamp(min=1)) ** 2, torch.zeros_like(n))
        h[0] = 1.0 / (4.0 * self.du ** 2)
        m = 4 * Nu
        taps = torch.zeros(m, device=DEVICE, dtype=torch.float64)
        taps[:Nu] = h
        taps[m - Nu + 1:] = h[1:].flip(0)
        return torch.fft.irfft(torch.fft.rfft(rows, n=m) * torch.fft.rfft(taps).real, n=m)[..., :Nu]

    def _step(self):
        d = self.angles.double().diff()
        step = float(((d + math.pi) % (2 * math.pi) - math.pi).abs().mean())
        return step if self.c["parker"] else step / 2

    def fbp(self, sino):
        return self.from_sino(self._filter(sino * self._cell_weight()), "backproject_weighted") * self._step()

    def fbp_t(self, image):
        return self._filter(self.from_image(image * self._step(), "backproject_weighted_t")) * self._cell_weight()


def _cost(c):
    return c["batch"] * c["V"] * max(c["W"], c["H"]) * c["Nu"] * (max(1, c["D"]) + max(1, c["Nv"])) * \
        (2 if "gradient" in c["what"] or c["what"] == "project_backproject" else 1)


def _exact_one(c, image, sino):
    what, e = c["what"], _Exact(c)
    image = None if image is None else image.detach().double().reshape(c["batch"], e.D, c["H"], c["W"])
    sino = None if sino is None else sino.detach().double().reshape(c["batch"], c["V"], e.Nv, c["Nu"])
    as_image = lambda x: x[:, None] if c["D"] else x.reshape(c["batch"], 1, c["H"], c["W"])  # noqa: E731
    as_sino = lambda x: x[:, None] if c["Nv"] else x.reshape(c["batch"], 1, c["V"], c["Nu"])  # noqa: E731
    if what in FROM_IMAGE:
        return as_sino(e.from_image(image, what))
    if what in FROM_SINO:
        return as_image(e.from_sino(sino, what))
    if what == "project_backproject":
        y = e.from_image(image, "project")
        return as_sino(y), as_image(e.from_sino(y, "backproject"))
    if what == "fbp":
        return as_image(e.fbp(sino))
    if what == "gradient":
        y = e.from_image(image, "project")
        return as_sino(y), as_image(e.from_sino(y - sino, "project_t"))
    x = e.fbp(sino)
    return as_image(x), as_sino(e.fbp_t(x - image))


def exact(case, seed):
    c = case
    if c["what"] == "ragged":
        sinos, recons = [], []
        for i, p in enumerate(_ragged_instances(c)):
            image = _volume(p, 1000 * seed + i)
            y = _Exact(p).from_image(image.double(), "project")
            sinos.append(y.reshape(1, 1, p["V"], p["Nu"]))
            recons.append(_exact_one(p, None, y))
        return sinos, recons
    # Helical FBP weights its views by float32 window decisions, which have no value in 64 bits.
    if c["scan"] == "helical" and (c["what"].startswith("fbp") or "weighted" in c["what"]):
        return None
    if _cost(c) > 2.5e10:  # over about 20 seconds
        return None
    image = _volume(c, 1000 * seed) if c["what"] not in FROM_SINO + ("fbp",) else None
    sino = _sinogram(c, 1000 * seed + 500) if c["what"] in FROM_SINO + ("fbp", "gradient", "fbp_gradient") else None
    return _exact_one(c, image, sino)
