"""The workloads this framework is measured on, through its public Python entry points.

A case is a dict of plain values.  ``op`` names the call:

* ``project`` / ``backproject``  ``Plan.project`` / ``Plan.backproject`` (distance-driven
  ``dd`` or separable-footprint ``tf``), all views or one ordered subset;
* ``fdk``    ``FDK.__call__``: weighting, row filter and backprojection of a whole scan;
* ``pwls``   ``reconPwlsSeSqs``: a whole OS-SQS call (surrogate set-up and one iteration);
* ``fan``    the 2-D fan-beam pair (``FanPlan.project`` and ``FanPlan.backproject``).

The scan is given by the volume (``nx ny nz``, in-plane spacing ``d``, slice spacing ``dz``,
mm), the detector (``nu nv du dv``, ``flat`` 1 or curved 0), the number of ``views`` over
2 pi and, for ordered subsets, their number ``subsets`` (views 1, 1 + subsets, ...).
SAD is 1000 mm and SDD 1500 mm throughout, as in the benchmark configurations.
``offset`` shifts volume and detector by fractions of a cell, ``couch`` moves the table
by that many mm over the scan, ``fov`` switches off the columns outside the inscribed
circle.  ``dtype`` is the storage type of the call's input.
"""
from __future__ import annotations

import math

import numpy as np
import torch

SAD, SDD = 1000.0, 1500.0
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
CONFIG1 = dict(nx=128, ny=128, nz=64, d=1.0, dz=1.0, nu=256, nv=96, du=1.6, dv=1.6, views=360, subsets=1)
CONFIG2 = dict(nx=512, ny=512, nz=256, d=0.5, dz=0.5, nu=1024, nv=384, du=0.8, dv=0.8, views=720, subsets=1)


def _case(op, base, **kw):
    c = dict(base, op=op, method="dd", flat=1, offset=0.0, couch=0.0, fov=False, dtype="f32")
    c.update(kw)
    return c


def listed():
    return [
        # the headline step of a large scan: the forward projection and its matched adjoint
        _case("project", CONFIG2, name="proj_dd_512"),
        _case("backproject", CONFIG2, name="back_dd_512"),
        # the analytic reconstruction of the same scan
        _case("fdk", CONFIG2, name="fdk_512"),
        # one ordered-subset step of iterative reconstruction on it (24 subsets of 30 views)
        _case("project", CONFIG2, name="proj_tf_512_subset", method="tf", subsets=24),
        _case("backproject", CONFIG2, name="back_tf_512_subset", method="tf", subsets=24),
        # a small scan, as served many at a time; 16-bit storage on the measured data
        _case("project", CONFIG1, name="proj_dd_128"),
        _case("backproject", CONFIG1, name="back_dd_128_bf16", dtype="bf16"),
        _case("fdk", CONFIG1, name="fdk_128_bf16", dtype="bf16"),
        # sizes that fit no tile: a curved detector with quarter-pixel offsets, FP16 volume
        _case("project", dict(nx=211, ny=187, nz=93, d=0.9, dz=0.8, nu=391, nv=157, du=0.95, dv=0.9, views=241,
                              subsets=1), name="proj_tf_ragged_f16", method="tf", flat=0, offset=0.25, dtype="f16"),
        # a moving couch and a circular field of view on an odd detector
        _case("backproject", dict(nx=190, ny=203, nz=77, d=1.0, dz=1.1, nu=413, nv=130, du=0.9, dv=1.3, views=300,
                                  subsets=1), name="back_dd_couch_fov", offset=0.3, couch=24.0, fov=True),
        # a whole iterative call on the small scan: set-up and one iteration of 12 subsets
        _case("pwls", CONFIG1, name="pwls_128", method="tf", subsets=12),
        # the 2-D pair on one slice, the smallest call
        _case("fan", dict(nx=256, ny=256, nz=1, d=1.0, dz=1.0, nu=360, nv=1, du=1.2, dv=1.0, views=180, subsets=1),
              name="fan_256"),
    ]


def draw(rng):
    """Another case of the same calls and ranges: in-plane 96 to 512, 32 to 256 slices, 90 to
    720 views, detectors that cover the volume with pixels 0.6 to 1.4 voxels wide at the axis."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["project", "project", "project", "backproject", "backproject", "backproject", "fdk", "fdk",
                     "pwls", "fan"])
    nx = logint(96, 512)
    ny = max(90, min(512, int(round(nx * rng.uniform(0.85, 1.15)))))
    nz = 1 if op == "fan" else logint(32, 256)
    if op == "pwls":
        nx, ny, nz = min(nx, 224), min(ny, 224), min(nz, 96)
    size = 256.0 * rng.uniform(0.6, 1.0)  # mm across
    d = round(size / max(nx, ny), 3)
    dz = 1.0 if op == "fan" else round(d * rng.uniform(0.8, 1.3), 3)
    mag = SDD / SAD
    du = round(d * mag * rng.uniform(0.6, 1.4), 3)
    dv = 1.0 if op == "fan" else round(dz * mag * rng.uniform(0.75, 1.35), 3)
    nu = int(math.ceil(max(nx, ny) * d * mag * 1.25 / du)) + rng.randrange(0, 9)
    nv = 1 if op == "fan" else int(math.ceil(nz * dz * mag * rng.uniform(0.9, 1.25) / dv)) + rng.randrange(0, 5)
    views = logint(90, 720)
    subsets = 1
    if op == "pwls":
        views, subsets = min(views, 360), rng.choice([6, 10, 12])
    elif op in ("project", "backproject") and rng.random() < 0.3:
        subsets = rng.choice([5, 12, 24])
    curved = op != "fan" and rng.random() < 0.25
    return _case(op, dict(nx=nx, ny=ny, nz=nz, d=d, dz=dz, nu=nu, nv=nv, du=du, dv=dv, views=views, subsets=subsets),
                 method="tf" if op == "pwls" else rng.choice(["dd", "tf"]),
                 flat=0 if curved else 1, offset=rng.choice([0.0, 0.0, 0.25]),
                 couch=0.0 if op in ("fdk", "fan", "pwls") else rng.choice([0.0, 0.0, 12.0]),
                 fov=op in ("project", "backproject") and rng.random() < 0.3,
                 dtype="f32" if op in ("pwls", "fan") else rng.choice(["f32", "f32", "bf16", "f16"]))


# ---------------------------------------------------------------------------
# The scan and the inputs
# ---------------------------------------------------------------------------
class _Scan:
    """The numbers of a case: view angles, couch, centre offsets and the field-of-view mask."""

    def __init__(self, c):
        f = lambda v: float(np.float32(v))
        self.d, self.dz, self.du, self.dv = f(c["d"]), f(c["dz"]), f(c["du"]), f(c["dv"])
        self.off = f(c["offset"])
        n = c["views"]
        self.betas = np.arange(n, dtype=np.float64) * (2 * np.pi / n)
        self.couch = (np.linspace(-0.5, 0.5, n) * c["couch"]).astype(np.float32)
        self.sel = slice(1 % c["subsets"], None, c["subsets"]) if c["op"] != "pwls" else slice(None)
        self.wx, self.wy = -(c["nx"] - 1) / 2 + self.off, -(c["ny"] - 1) / 2 + self.off
        self.wu, self.wv = -(c["nu"] - 1) / 2 + self.off, -(c["nv"] - 1) / 2 + self.off
        self.wz = -(c["nz"] - 1) / 2 + self.off
        self.mask = None
        if c["fov"]:
            x, y = np.arange(c["nx"]) - (c["nx"] - 1) / 2, np.arange(c["ny"]) - (c["ny"] - 1) / 2
            self.mask = x[None, :] ** 2 + y[:, None] ** 2 < (min(c["nx"], c["ny"]) / 2) ** 2

    def geometry(self, c):
        from ctsim_b200 import CTGeometry
        o = self.off
        return CTGeometry((c["nx"], c["ny"], c["nz"]), (self.d, self.d, self.dz), (o, o, o), (c["nu"], c["nv"]),
                          (self.du, self.dv), (o, o), SAD, SDD - SAD, SDD, self.betas, couchZ=self.couch,
                          flatPanel=c["flat"], map=self.mask)


def _spheres(c, s, seed):
    """A water cylinder's radius and 8 seeded spheres: centre (x, y, z), radius, attenuation (1/cm)."""
    rng = np.random.default_rng([seed, c["nx"], c["nz"]])
    r = 0.45 * min(c["nx"], c["ny"]) * s.d
    h = max(0.5 * c["nz"] * s.dz, 1.0)
    a, q = rng.uniform(0, 2 * np.pi, 8), r * 0.8 * np.sqrt(rng.random(8))
    z = rng.uniform(-0.8, 0.8, 8) * h if c["nz"] > 1 else np.zeros(8)
    return r, [(q[i] * np.cos(a[i]), q[i] * np.sin(a[i]), z[i], r * rng.uniform(0.05, 0.3), rng.uniform(-0.1, 0.3))
               for i in range(8)]


def _image(c, s, seed):
    """The phantom with a little seeded texture: [nz, ny, nx], 1/cm."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    ax = lambda n, w, d: (torch.arange(n, device="cuda", dtype=torch.float32) + w) * d
    x, y, z = ax(c["nx"], s.wx, s.d), ax(c["ny"], s.wy, s.d), ax(c["nz"], s.wz, s.dz)
    r, balls = _spheres(c, s, seed)
    img = torch.rand((c["nz"], c["ny"], c["nx"]), generator=g, device="cuda").mul_(0.01)
    img += 0.2 * ((x[None, :] ** 2 + y[:, None] ** 2) < r * r)
    for bx, by, bz, br, mu in balls:
        img += mu * (((x - bx) ** 2)[None, None, :] + ((y - by) ** 2)[None, :, None] +
                     ((z - bz) ** 2)[:, None, None] < br * br)
    return img.clamp_(min=0.0)


def _sinogram(c, s, seed):
    """Line integrals of the phantom's analytic shapes with log-Poisson-like noise:
    [selected views, nu, nv]."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    betas = s.betas[s.sel]
    r, balls = _spheres(c, s, seed)
    u = ((torch.arange(c["nu"], device="cuda", dtype=torch.float32) + s.wu) * s.du)[:, None]
    v = ((torch.arange(c["nv"], device="cuda", dtype=torch.float32) + s.wv) * s.dv)[None, :]
    st, ct = (u / torch.sqrt(u * u + SDD * SDD), SDD / torch.sqrt(u * u + SDD * SDD)) if c["flat"] else \
        (torch.sin(u / SDD), torch.cos(u / SDD))
    tan = v / (torch.sqrt(u * u + SDD * SDD) if c["flat"] else SDD)
    norm = torch.sqrt(1.0 + tan * tan)
    dt, ds, dz = st / norm, ct / norm, tan / norm  # ray directions: across, along, up
    chord = 2.0 * torch.sqrt((r * r - (SAD * st) ** 2).clamp_(min=0.0)) * norm
    out = torch.randn((len(betas), c["nu"], c["nv"]), generator=g, device="cuda")
    for k, b in enumerate(betas):
        line = 0.02 * chord
        for bx, by, bz, br, mu in balls:
            t, q = bx * math.cos(b) - by * math.sin(b), SAD + bx * math.sin(b) + by * math.cos(b)
            along = t * dt + q * ds + bz * dz
            line = line + (0.2 * mu) * torch.sqrt((br * br - (t * t + q * q + bz * bz) + along * along).clamp_(min=0.0))
        out[k] = line + out[k] * (0.003 * torch.exp(0.5 * line))
    return out.clamp_(min=0.0)


class _State:
    pass


def prepare(case, seed):
    c, s, st = case, _Scan(case), _State()
    torch.cuda.set_device(0)
    st.case, dt = c, DTYPES[c["dtype"]]
    if c["op"] == "fan":
        from ctsim_b200.fan import FanPlan
        from ctsim_b200.geometry import FanGeometry
        st.plan = FanPlan(FanGeometry((c["nx"], c["ny"]), (s.d, s.d), (s.off, s.off), c["nu"], s.du, s.off, SAD,
                                      SDD - SAD, SDD, s.betas, c["flat"]))
        st.image, st.sino = _image(c, s, seed)[0].contiguous(), _sinogram(c, s, seed)[:, :, 0].contiguous()
        return st
    st.geom = s.geometry(c)
    if c["op"] == "pwls":
        st.y = _sinogram(c, s, seed)
        st.w = 1e5 * torch.exp(-st.y)
        st.x0 = torch.full(st.geom.image_shape, 0.15, device="cuda")
        return st
    from ctsim_b200.projector import Plan
    st.plan = Plan(st.geom)
    st.views = (s.sel.start, c["subsets"], len(s.betas[s.sel]))
    if c["op"] == "project":
        st.image = _image(c, s, seed).to(dt)
    else:
        st.sino = _sinogram(c, s, seed).to(dt)
    if c["op"] == "fdk":
        from ctsim_b200.fdk import FDK
        st.fdk = FDK(st.geom, "hann", plan=st.plan)
    return st


def run(state):
    c = state.case
    if c["op"] == "project":
        return state.plan.project(state.image, c["method"], *state.views)
    if c["op"] == "backproject":
        return state.plan.backproject(state.sino, c["method"], *state.views, out_dtype=torch.float32)
    if c["op"] == "fdk":
        return state.fdk(state.sino)
    if c["op"] == "pwls":
        from ctsim_b200.pwls import reconPwlsSeSqs
        return reconPwlsSeSqs(state.y, state.w, state.geom, 1e3, "huber", 1, 0.01, c["subsets"], state.x0)[0]
    return {"sino": state.plan.project(state.image, c["method"]),
            "image": state.plan.backproject(state.sino, c["method"])}


def work(case):
    """Bytes: the volume and the sinogram once each (FP32 data terms and updates in the
    iterative call).  Operations: per voxel and view an axial overlap of two or three cells
    and the weighted sum into (from) the detector columns, 2 flops per weight: 10 for the
    footprint projectors, 16 for the bilinear FDK sample with its weights; the row filter's
    two FFTs."""
    c, s = case, _Scan(case)
    nviews = len(s.betas[s.sel])
    vox, pix = c["nx"] * c["ny"] * c["nz"], nviews * c["nu"] * c["nv"]
    size = 4 if c["dtype"] == "f32" else 2
    vv = vox * nviews
    if c["op"] == "project":
        return {"bytes": size * (vox + pix), "flops": 10 * vv}
    if c["op"] == "backproject":
        return {"bytes": size * pix + 4 * vox, "flops": 10 * vv}
    if c["op"] == "fdk":
        n = max(64, 1 << (2 * c["nu"] - 2).bit_length())
        return {"bytes": size * pix + 4 * vox, "flops": 16 * vv + 5 * n * (n.bit_length() - 1) * nviews * c["nv"]}
    if c["op"] == "pwls":  # A and A^T for the surrogate and again for the iteration
        return {"bytes": 4 * (4 * pix + 4 * vox * c["subsets"]), "flops": 4 * 10 * vv}
    return {"bytes": 8 * (vox + pix), "flops": 2 * 8 * vv}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
class _Exact:
    """The footprint projectors, FDK and OS-SQS in float64 tensors, one view at a time."""

    def __init__(self, c, s):
        self.c, self.s = c, s
        ar = lambda n: torch.arange(n, device="cuda", dtype=torch.float64)
        x, y = (ar(c["nx"]) + s.wx) * s.d, (ar(c["ny"]) + s.wy) * s.d
        self.x, self.y = x.repeat(c["ny"]), y.repeat_interleave(c["nx"])
        self.on = None if s.mask is None else torch.from_numpy(s.mask.reshape(-1)).cuda()
        u, v = ((ar(c["nu"]) + s.wu) * s.du)[:, None], ((ar(c["nv"]) + s.wv) * s.dv)[None, :]
        self.ampv = torch.sqrt(1 + v * v / (SDD * SDD + u * u)) if c["flat"] else \
            torch.sqrt(1 + v * v / (SDD * SDD)).expand(c["nu"], c["nv"])

    def _u(self, t, q):
        s = self.s
        return (SDD / s.du) * (t / q if self.c["flat"] else torch.atan(t / q)) - s.wu

    def footprint(self, k, lo, hi):
        """Of columns lo .. hi in view k: amplitude, first detector column, the weights of the
        columns from there (a list), voxel height in rows, bottom edge of voxel 0."""
        c, s = self.c, self.s
        sn, cs = math.sin(s.betas[k]), math.cos(s.betas[k])
        x, y = self.x[lo:hi], self.y[lo:hi]
        t, q = x * cs - y * sn, SAD + x * sn + y * cs
        r = torch.sqrt(t * t + q * q)
        cp, sp = torch.abs((cs * q - sn * t) / r), torch.abs((sn * q + cs * t) / r)
        hx, hy = (s.d * cs / 2, s.d * sn / 2), (s.d * sn / 2, -s.d * cs / 2)  # half steps in x, in y
        amp = s.d / torch.maximum(cp, sp) / 10
        if self.on is not None:
            amp = amp * self.on[lo:hi]
        if c["method"] == "dd":
            a = torch.where(cp > sp, self._u(t + hx[0], q + hx[1]), self._u(t + hy[0], q + hy[1]))
            b = torch.where(cp > sp, self._u(t - hx[0], q - hx[1]), self._u(t - hy[0], q - hy[1]))
            p = [torch.minimum(a, b) + 0.5, torch.maximum(a, b) + 0.5]
            mass = lambda e: torch.minimum(torch.maximum(e, p[0]), p[1])
        else:
            p = torch.sort(torch.stack([self._u(t + i * hx[0] + j * hy[0], q + i * hx[1] + j * hy[1])
                                        for i in (1, -1) for j in (1, -1)]), dim=0).values + 0.5
            ramp = lambda e, a, b: torch.minimum(torch.maximum(e, a), b) - a
            up, dn = (p[1] - p[0]).clamp(min=1e-30), (p[3] - p[2]).clamp(min=1e-30)
            mass = lambda e: ramp(e, p[0], p[1]) ** 2 / (2 * up) + ramp(e, p[1], p[2]) + \
                (dn - ramp(e, p[2], p[3]) / 2) * ramp(e, p[2], p[3]) / dn
        iu = torch.floor(p[0])
        n = int((torch.floor(p[-1]) - iu).max()) + 1
        edges = [mass(iu + b) for b in range(n + 1)]
        iu = iu.long()
        w = [torch.where((iu + b >= 0) & (iu + b < c["nu"]), (edges[b + 1] - edges[b]) * amp, 0.0) for b in range(n)]
        zinc = s.dz / s.dv * SDD / q
        return iu, w, zinc, (s.wz + float(s.couch[k]) / s.dz - 0.5) * zinc - s.wv + 0.5

    def _chunks(self):
        n = self.x.numel()
        step = max(1024, (1 << 25) // max(self.c["nz"], self.c["nv"]))
        return [(a, min(n, a + step)) for a in range(0, n, step)]

    @staticmethod
    def _at(table, row, e):
        """Piecewise-linear table[row] at positions e [n, m]."""
        n = table.shape[1] - 1
        k = torch.floor(e).clamp_(0, n - 1)
        i = k.long() + row[:, None] * (n + 1)
        a = table.reshape(-1)[i]
        return a + (e - k) * (table.reshape(-1)[i + 1] - a)

    def project(self, img, views):
        c = self.c
        cols = img.double().reshape(c["nz"], -1).t()
        sums = torch.cat([torch.zeros_like(cols[:, :1]), torch.cumsum(cols, 1)], 1)
        iv = torch.arange(c["nv"] + 1, device="cuda", dtype=torch.float64)
        out = torch.zeros((len(views), c["nu"], c["nv"]), device="cuda", dtype=torch.float64)
        for k, view in enumerate(views):
            for a, b in self._chunks():
                iu, w, zinc, v0 = self.footprint(view, a, b)
                e = ((iv[None, :] - v0[:, None]) / zinc[:, None]).clamp_(0, c["nz"])
                rows = self._at(sums[a:b], torch.arange(b - a, device="cuda"), e).diff(dim=1) * zinc[:, None]
                for j, wj in enumerate(w):
                    out[k].index_add_(0, (iu + j).clamp(0, c["nu"] - 1), rows * wj[:, None])
        return out * self.ampv

    def backproject(self, sino, views, scale=1.0):
        c = self.c
        iz = torch.arange(c["nz"] + 1, device="cuda", dtype=torch.float64)
        img = torch.zeros((self.x.numel(), c["nz"]), device="cuda", dtype=torch.float64)
        for k, view in enumerate(views):
            p = sino[k].double() * self.ampv
            sums = torch.cat([torch.zeros_like(p[:, :1]), torch.cumsum(p, 1)], 1)
            for a, b in self._chunks():
                iu, w, zinc, v0 = self.footprint(view, a, b)
                e = (v0[:, None] + iz[None, :] * zinc[:, None]).clamp_(0, c["nv"])
                acc = 0.0
                for j, wj in enumerate(w):
                    acc = acc + self._at(sums, (iu + j).clamp(0, c["nu"] - 1), e) * wj[:, None]
                img[a:b] += acc.diff(dim=1)
        return (img * scale).t().reshape(c["nz"], c["ny"], c["nx"])

    def fdk(self, sino):
        c, s = self.c, self.s
        n = max(64, 1 << (2 * c["nu"] - 2).bit_length())
        i = np.arange(-n // 2 + 1, n // 2)
        h = np.zeros(n)
        odd = i % 2 == 1
        d = i * np.pi * s.du if c["flat"] else SDD * np.pi * np.sin(i * s.du / SDD)
        h[:-1][odd] = -1.0 / d[odd] ** 2
        h[:-1][i == 0] = 1.0 / (4 * s.du ** 2)
        H = np.abs(np.fft.fft(h))
        f = np.minimum(np.arange(n), n - np.arange(n)) * (2 * np.pi / n)
        H = torch.from_numpy(H * (1 + np.cos(f)) / 2 * s.du).cuda()[None, :, None]
        u = (torch.arange(c["nu"], device="cuda", dtype=torch.float64) + s.wu)[:, None] * s.du
        v = (torch.arange(c["nv"], device="cuda", dtype=torch.float64) + s.wv)[None, :] * s.dv
        wt = SAD * torch.sqrt(1 + u * u / SDD ** 2) / torch.sqrt(u * u + v * v + SDD ** 2) if c["flat"] else \
            SAD / SDD * torch.cos(u / torch.sqrt(SDD ** 2 + v * v))
        z = (torch.arange(c["nz"], device="cuda", dtype=torch.float64) + s.wz) * s.dz
        img = torch.zeros((c["nz"], self.x.numel()), device="cuda", dtype=torch.float64)
        for k, beta in enumerate(s.betas):
            q = torch.fft.ifft(torch.fft.fft(sino[k:k + 1].double() * wt, n=n, dim=1) * H, dim=1).real[0, :c["nu"]]
            q = q.reshape(-1)
            xr, yr = self.x * math.cos(beta) - self.y * math.sin(beta), self.x * math.sin(beta) + self.y * math.cos(beta)
            den = SAD + yr
            w2 = SDD / den
            if c["flat"]:
                pu, w2s = xr * w2 / s.du - s.wu, w2 * w2
            else:
                xo = xr - s.off * s.du * SAD / SDD
                pu, w2s = torch.atan(xo / den) * SDD / s.du - s.wu, SDD ** 2 / (den * den + xo * xo)
            w2s = torch.where((pu >= 1e-6) & (pu <= c["nu"] - 1 - 1e-6), w2s, 0.0)
            iu = torch.floor(pu).clamp(0, c["nu"] - 2)
            fu = pu - iu
            pv = (z[:, None] * w2[None, :] / s.dv - s.wv).clamp_(0.5, c["nv"] - 1.5)
            iv = torch.floor(pv).clamp_(0, c["nv"] - 2)
            fv = pv - iv
            at = (iu * c["nv"])[None, :] + iv
            at = at.long()
            s0 = (1 - fv) * q[at] + fv * q[at + 1]
            s1 = (1 - fv) * q[at + c["nv"]] + fv * q[at + c["nv"] + 1]
            img += w2s * ((1 - fu) * s0 + fu * s1)
        step = abs(s.betas[-1] - s.betas[0]) / (len(s.betas) - 1) / 2
        return (img * (step * 10)).reshape(c["nz"], c["ny"], c["nx"])

    @staticmethod
    def _huber(x, delta):
        """Gradient and curvature of the Huber penalty over the five neighbour directions."""
        S, T = torch.zeros_like(x), torch.zeros_like(x)
        cut = lambda o: (slice(max(0, -o), None if o <= 0 else -o), slice(max(0, o), None if o >= 0 else o))
        for oz, oy, ox, w in ((0, 0, 1, 1.0), (0, 1, 0, 1.0), (0, 1, 1, 2 ** -0.5), (0, 1, -1, 2 ** -0.5),
                              (1, 0, 0, 0.5)):
            (z0, z1), (y0, y1), (x0, x1) = cut(oz), cut(oy), cut(ox)
            d = x[z0, y0, x0] - x[z1, y1, x1]
            g, k = d.clamp(-delta, delta) * w, (d.abs() <= delta).double() * w
            S[z0, y0, x0] += g
            S[z1, y1, x1] -= g
            T[z0, y0, x0] += k
            T[z1, y1, x1] += k
        return S, T

    def pwls(self, y, w, x, beta, delta):
        n, m = len(self.s.betas), self.c["subsets"]
        y, w, x, every = y.double(), w.double(), x.double(), range(n)
        pre = self.backproject(w * self.project(torch.ones_like(x), every), every)
        for i in range(1, m + 1):
            views = list(range(i % m, n, m))
            num = self.backproject(w[i % m::m] * (self.project(x, views) - y[i % m::m]), views, float(m))
            S, T = self._huber(x, delta)
            x = x - (num + beta * S) / (pre + beta * T)
            x = torch.where(torch.isfinite(x) & (x > 0), x, 0.0)
        return x

    def fan(self, image, sino):
        c, n = self.c, self.x.numel()
        x, out, img = image.double().reshape(-1), [], torch.zeros(n, device="cuda", dtype=torch.float64)
        for k in range(len(self.s.betas)):
            iu, w, _, _ = self.footprint(k, 0, n)
            row = torch.zeros(c["nu"], device="cuda", dtype=torch.float64)
            for j, wj in enumerate(w):
                at = (iu + j).clamp(0, c["nu"] - 1)
                row.index_add_(0, at, x * wj)
                img += sino[k].double()[at] * wj
            out.append(row)
        return {"sino": torch.stack(out), "image": img.reshape(c["ny"], c["nx"])}


def exact(case, seed):
    c, s = case, _Scan(case)
    views = range(len(s.betas))[s.sel]
    passes = 4 if c["op"] == "pwls" else 1
    if passes * c["nx"] * c["ny"] * c["nz"] * len(views) > 6e9:  # over about 20 seconds
        return None
    e = _Exact(c, s)
    dt = DTYPES[c["dtype"]]
    if c["op"] == "project":
        return e.project(_image(c, s, seed).to(dt), views)
    sino = _sinogram(c, s, seed)
    if c["op"] == "backproject":
        return e.backproject(sino.to(dt), views)
    if c["op"] == "fdk":
        return e.fdk(sino.to(dt))
    if c["op"] == "pwls":
        x0 = torch.full((c["nz"], c["ny"], c["nx"]), float(np.float32(0.15)), device="cuda")
        return e.pwls(sino, 1e5 * torch.exp(-sino), x0, 1e3, float(np.float32(0.01)))
    return e.fan(_image(c, s, seed)[0], sino[:, :, 0])
