"""Measured cases: the calls a user of this library makes, over the sizes they are made at.

A case is a dict of plain values.  ``prepare`` builds what a program holds before the call
(seeded synthetic surveys: diffractions plus noise, generated here with torch), ``run`` is
one call through the public Python entry points, ``work`` the bytes and operations the
call cannot do without, ``exact`` the same result in 64 bits with plain torch.

Kinds
  dropin     ktmMigrationCPU on host arrays, the reference's own call (synchronous)
  reference  the same arithmetic on device arrays (mode "reference")
  fast       migration of a packed trace set that the program keeps
  raw        migration straight from raw device traces: filter, pack and migrate
  batch      many small target jobs in one launch
  prep       trace preparation: rho filter, weight fold, scale, packing
  demigrate  the adjoint: image to data
  gradient   dI/dv of a packed trace set
  lsm        least-squares migration (CGLS)
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "seismic-migration_b200"))
import ktm  # noqa: E402
from ktm import inverse  # noqa: E402

DEV = "cuda"
RHO = {"none": 0, "2d": 1, "2.5d": 2, "3d": 3}


def listed():
    return [
        # a quick look at a short line through the reference's own C call: launch and copy
        # latency count as much as the kernel
        dict(name="dropin_small", kind="dropin", geom="line", nx=64, noff=8, nt=251, nz=251,
             dt=0.004),
        # the reference's call on a whole 2-D line (256 CMPs x 64 offsets, 1001 samples),
        # data resident on the device
        dict(name="reference_line", kind="reference", geom="line", nx=256, noff=64, nt=1001,
             nz=1001, dt=0.004),
        # bit-exact migration of an odd-sized 3-D target (quality control of the fast modes)
        dict(name="reference_areal", kind="reference", geom="areal", nx=23, ny=19, ntr=3001,
             nt=451, nz=401, dt=0.004),
        # the 2-D line in the mixed-precision mode, packed once, migrated for a velocity
        dict(name="line_f16", kind="fast", geom="line", nx=256, noff=64, nt=1001, nz=1001,
             dt=0.004, fmt="f16", weight="prefold", pick="linear", aperture=2000.0),
        # one call from raw traces of a shorter line, default weight and FP32 storage
        dict(name="line_raw", kind="raw", geom="line", nx=128, noff=48, nt=751, nz=751, dt=0.004,
             fmt="f32", weight="table", pick="linear", aperture=1500.0, rho="2.5d"),
        # a slice of the 3-D survey into the full 200 x 200 x 1501 image with a Vrms cube
        dict(name="areal_f16", kind="fast", geom="areal", nx=200, ny=200, ntr=2500, nt=1501,
             nz=1501, dt=0.002, fmt="f16", weight="prefold", pick="linear", aperture=3000.0),
        # target-oriented jobs of mixed sizes in one launch
        dict(name="batch_targets", kind="batch", geom="areal", jobs=12, nx=16, ny=12, ntr=4000,
             nt=751, nz=501, dt=0.004, fmt="bf16", weight="table", pick="linear",
             aperture=1500.0),
        # preparation of one block of the 3-D survey
        dict(name="prep_areal", kind="prep", ntr=62500, nt=1501, dt=0.002, fmt="f16", rho="3d",
             prefold=True, ibm=False),
        # preparation of a line as it comes from tape: IBM words, odd counts
        dict(name="prep_ibm_line", kind="prep", ntr=4097, nt=1001, dt=0.004, fmt="f32",
             rho="2.5d", prefold=False, ibm=True),
        # the adjoint on the least-squares line (512 CMPs x 64 offsets)
        dict(name="demigrate_line", kind="demigrate", geom="line", nx=512, noff=64, nt=1001,
             nz=1001, dt=0.004, weight="prefold", aperture=2000.0),
        # velocity gradient on the 2-D line
        dict(name="gradient_line", kind="gradient", geom="line", nx=256, noff=64, nt=1001,
             nz=1001, dt=0.004, fmt="f16", weight="table", aperture=2000.0),
        # a least-squares run of a few iterations on a small line
        dict(name="lsm_line", kind="lsm", geom="line", nx=96, noff=24, nt=501, nz=501, dt=0.004,
             weight="prefold", aperture=1500.0, iterations=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "reference", "fast", "fast", "raw", "batch", "prep", "prep",
                       "demigrate", "gradient", "lsm"])
    dt = rng.choice([0.001, 0.002, 0.004])
    if kind == "prep":
        nt = _log(rng, 150, 6001)
        return dict(kind=kind, ntr=max(1, min(_log(rng, 17, 62500), 90_000_000 // nt)), nt=nt,
                    dt=dt, fmt=rng.choice(["f16", "bf16", "f32"]),
                    rho=rng.choice(["none", "2d", "2.5d", "3d"]),
                    prefold=rng.random() < 0.5, ibm=rng.random() < 0.3)
    nt = _log(rng, 200, 2201)
    step = rng.choice([1, 1, 2])                     # tau step in half sample intervals
    case = dict(kind=kind, nt=nt, nz=max(33, nt // step - rng.randrange(8)), dt=dt, step=step)
    most = {"dropin": 2e9, "reference": 8e9, "fast": 8e10, "raw": 3e10, "batch": 2e10,
            "demigrate": 1.2e10, "gradient": 3e10, "lsm": 2e8}[kind]
    if kind == "batch" or (kind in ("dropin", "reference", "fast", "raw") and rng.random() < 0.5):
        case.update(geom="areal", nx=_log(rng, 8, 150), ny=_log(rng, 8, 150))
        jobs = 1
        if kind == "batch":
            jobs = rng.randrange(3, 25)
            case.update(jobs=jobs, nx=rng.randrange(5, 40), ny=rng.randrange(5, 40))
        cap = most / (jobs * case["nx"] * case["ny"] * case["nz"])
        case.update(ntr=int(max(50, min(_log(rng, 500, 60000), cap))))
    else:
        nx = _log(rng, 24, 256 if kind == "lsm" else 700)
        cap = most / (nx * nx * case["nz"])
        case.update(geom="line", nx=nx, noff=int(max(2, min(_log(rng, 8, 96), cap))))
    if kind in ("fast", "raw", "batch"):
        pick = "truncate" if rng.random() < 0.2 else "linear"
        weights = ["table", "sqrt"] + (["prefold", "prefold"] if pick == "linear" else [])
        case.update(fmt=rng.choice(["f16", "bf16", "f32"]), weight=rng.choice(weights), pick=pick,
                    aperture=rng.choice([0.0, 1000.0, 2000.0, 3000.0]))
    if kind == "raw":
        case.update(rho=rng.choice(["none", "2d", "2.5d", "3d"]))
    if kind in ("demigrate", "lsm"):
        case.update(weight=rng.choice(["prefold", "table", "sqrt"]),
                    aperture=rng.choice([0.0, 1500.0, 2500.0]))
    if kind == "gradient":
        case.update(fmt=rng.choice(["f16", "f32"]), weight=rng.choice(["table", "prefold"]),
                    aperture=rng.choice([1500.0, 2500.0]))
    if kind == "lsm":
        case.update(iterations=rng.randrange(2, 7))
    return case


# ------------------------------------------------------------------------------ surveys ---
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _uniform(n, lo, hi, g):
    return lo + (hi - lo) * torch.rand(n, device=DEV, dtype=torch.float64, generator=g)


def _survey(case, seed, part=0):
    """Grids, FP32 device coordinates, velocity and raw traces [ntr, nt] of one survey."""
    g = _gen(seed * 1009 + part)
    dt, nt, nz = float(case["dt"]), int(case["nt"]), int(case["nz"])
    dtau = dt / 2.0 * case.get("step", 1)
    tmax = dt * (nt - 1)
    tau = dtau * torch.arange(nz, device=DEV, dtype=torch.float64)
    if case["geom"] == "line":
        # CMPs every 12.5 m, constant-offset bins every 50 m, offset-major order
        nx, noff = int(case["nx"]), int(case["noff"])
        cmp_x = 12.5 * torch.arange(nx, device=DEV, dtype=torch.float64)
        half = 25.0 * torch.arange(noff, device=DEV, dtype=torch.float64)
        mx, ox = cmp_x.repeat(noff), half.repeat_interleave(nx)
        my, oy = torch.zeros_like(mx), torch.zeros_like(mx)
        gx, gy = (nx, 12.5, 0.0), (1, 1.0, 0.0)
        vel = 1500.0 + 0.5 * 2000.0 * tau
        # a survey's traveltimes vary with the seed: the velocity trend by a few per cent
        vel = vel * (1.0 + 0.02 * float(torch.rand(1, device=DEV, generator=g)))
        wide, deep, freq, nsc = float(cmp_x[-1]), 0.0, 25.0, 20
    else:
        # sources uniform over the area around the image, offsets up to 4 km, any azimuth
        nx, ny, ntr = int(case["nx"]), int(case["ny"]), int(case["ntr"])
        if case["kind"] == "batch":                  # jobs of mixed sizes
            nx, ny = max(2, nx - part % 5), max(2, ny + part % 3)
            ntr = max(20, int(ntr * (1.0 + (part % 4)) / 4.0))
        wide, deep = max(25.0 * nx, 2000.0), max(25.0 * ny, 2000.0)
        sx, sy = _uniform(ntr, 0.0, wide, g), _uniform(ntr, 0.0, deep, g)
        off = _uniform(ntr, 0.0, min(4000.0, 0.8 * max(wide, deep)), g)
        az = _uniform(ntr, 0.0, 2.0 * math.pi, g)
        rx = (sx + off * torch.cos(az)).clamp(0.0, wide)
        ry = (sy + off * torch.sin(az)).clamp(0.0, deep)
        mx, my, ox, oy = (sx + rx) / 2, (sy + ry) / 2, (rx - sx) / 2, (ry - sy) / 2
        gx, gy = (nx, 25.0, 12.5), (ny, 25.0, 12.5)
        vel = 1500.0 + 2500.0 * 2.0 * tau / max(tmax, 1e-9)
        if case["kind"] == "fast":                   # Vrms cube, +-5 % smooth lateral field
            ax = torch.arange(nx, device=DEV, dtype=torch.float64) * 25.0
            ay = torch.arange(ny, device=DEV, dtype=torch.float64) * 25.0
            ph = _uniform(2, 0.0, 2.0 * math.pi, g)
            field = (torch.sin(ax / 400.0 + ph[0])[:, None] * torch.cos(ay / 500.0 + ph[1])[None])
            vel = vel[None, None, :] * (1.0 + 0.05 * field[:, :, None])
        freq, nsc = 30.0, 32
    mx, my, ox, oy, vel = (a.float().contiguous() for a in (mx, my, ox, oy, vel))
    traces = _traces(g, (mx, my, ox, oy), nt, dt, wide, deep, freq, nsc)
    return dict(gx=gx, gy=gy, gz=(nz, dtau, 0.0), dt=dt, nt=nt, mx=mx, my=my, ox=ox, oy=oy,
                vel=vel, traces=traces)


def _traces(g, coords, nt, dt, wide, deep, freq, nsc):
    """Ricker diffractions of nsc scatterers plus noise, FP32 [ntr, nt]."""
    mx, my, ox, oy = coords
    ntr, tmax = mx.numel(), dt * (nt - 1)
    freq = min(freq, 0.12 / dt)
    out = torch.randn((ntr, nt), device=DEV, generator=g) * 0.05
    px, py = _uniform(nsc, 0.0, max(wide, 1.0), g), _uniform(nsc, 0.0, deep, g)
    pt, pa = _uniform(nsc, 0.03 * tmax, 0.45 * tmax, g), _uniform(nsc, -1.0, 1.0, g)
    j = torch.arange(nt, device=DEV, dtype=torch.float32) * dt
    rows = max(1, 40_000_000 // nt)
    for x, y, t0, a in torch.stack([px, py, pt, pa], 1).tolist():
        v2 = (1500.0 + 1000.0 * t0) ** 2
        ts = torch.sqrt(t0 * t0 + ((mx - ox - x) ** 2 + (my - oy - y) ** 2) / v2)
        ts = ts + torch.sqrt(t0 * t0 + ((mx + ox - x) ** 2 + (my + oy - y) ** 2) / v2)
        for k in range(0, ntr, rows):
            b = ((j[None] - ts[k:k + rows, None]) * (math.pi * freq)) ** 2
            out[k:k + rows].addcmul_(1.0 - 2.0 * b, torch.exp(-b), value=a)
    return out


def _ibm_words(x):
    """FP32 -> IBM System/360 words (int32 bits), fraction rounded to nearest."""
    a = x.double().abs()
    nz = a > 0
    e = torch.where(nz, torch.floor(torch.log2(a.clamp_min(1e-300)) / 4.0) + 1.0, 0.0)
    f = a / torch.pow(torch.tensor(16.0, device=x.device, dtype=torch.float64), e)
    frac = torch.round(f * float(1 << 24)).long()
    over = frac >= (1 << 24)
    frac = torch.where(over, torch.full_like(frac, 1 << 20), frac)
    e = (e.long() + over.long() + 64).clamp(0, 127)
    w = ((x < 0).long() << 31) | (e << 24) | frac
    w = torch.where(nz, w, torch.zeros_like(w))
    return torch.where(w >= (1 << 31), w - (1 << 32), w).to(torch.int32)


def _prep_input(case, seed):
    g = _gen(seed * 1009 + 7)
    ntr = int(case["ntr"])
    coords = [_uniform(ntr, 0.0, hi, g).float() for hi in (3000.0, 3000.0, 1200.0, 1200.0)]
    x = _traces(g, coords, int(case["nt"]), float(case["dt"]), 3000.0, 3000.0, 30.0, 6)
    if not case["ibm"]:
        return x
    w = torch.empty(x.shape, device=DEV, dtype=torch.int32)
    rows = max(1, 8_000_000 // x.shape[1])
    for k in range(0, ntr, rows):
        w[k:k + rows] = _ibm_words(x[k:k + rows])
    return w


def _model(case, seed):
    """A sparse reflectivity image [nx, 1, nz]."""
    g = _gen(seed * 1009 + 13)
    shape = (int(case["nx"]), 1, int(case["nz"]))
    m = torch.randn(shape, device=DEV, generator=g)
    return m * (torch.rand(shape, device=DEV, generator=g) < 0.2)


# ------------------------------------------------------------------------------ prepare ---
def _job(sv, **more):
    return dict(imageX=sv["gx"], imageY=sv["gy"], imageZ=sv["gz"], dt=sv["dt"], midX=sv["mx"],
                midY=sv["my"], offX=sv["ox"], offY=sv["oy"], velocity=sv["vel"], **more)


def _image(sv):
    return torch.empty((sv["gx"][0], sv["gy"][0], sv["gz"][0]), device=DEV)


def _packed_job(case, sv):
    packed = ktm.prepare(sv["traces"], sv["dt"], fmt=case["fmt"], rho=0,
                         prefold=case["weight"] == "prefold")
    return _job(sv, traces=packed, image=_image(sv), pick=case["pick"], weight=case["weight"],
                aperture=case["aperture"])


def _operator(case, sv):
    return inverse.MigrationOperator(
        imageX=sv["gx"], imageY=sv["gy"], imageZ=sv["gz"], dt=sv["dt"], nt=sv["nt"],
        midX=sv["mx"], midY=sv["my"], offX=sv["ox"], offY=sv["oy"], velocity=sv["vel"],
        aperture=case["aperture"], weight=case["weight"])


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "prep":
        st["in"] = _prep_input(case, seed)
        st["args"] = dict(fmt=case["fmt"], rho=case["rho"], prefold=case["prefold"])
        dtype = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[case["fmt"]]
        st["dt"] = case["dt"]
        st["out"] = torch.empty((case["ntr"], ktm.packed_pitch(case["nt"], case["fmt"])),
                                device=DEV, dtype=dtype)
        st["scale"] = torch.empty(case["ntr"], device=DEV)
    elif kind == "batch":
        st["jobs"] = [_packed_job(case, _survey(case, seed, p)) for p in range(case["jobs"])]
    else:
        sv = _survey(case, seed)
        if kind == "dropin":
            host = {k: sv[k].cpu().numpy() for k in ("mx", "my", "ox", "oy", "traces", "vel")}
            st["args"] = (ktm.grid(*sv["gx"]), ktm.grid(*sv["gy"]), ktm.grid(*sv["gz"]),
                          ktm.JobParams(host["mx"].size, sv["nt"], sv["dt"]), host["mx"],
                          host["my"], host["ox"], host["oy"], host["traces"], host["vel"],
                          np.empty((sv["gx"][0], sv["gy"][0], sv["gz"][0]), np.float32))
        elif kind == "reference":
            st["job"] = _job(sv, traces=sv["traces"], image=_image(sv), mode="reference",
                             pick="truncate")
        elif kind == "fast":
            st["job"] = _packed_job(case, sv)
        elif kind == "raw":
            st["job"] = _job(sv, traces=sv["traces"], image=_image(sv), pick=case["pick"],
                             weight=case["weight"], aperture=case["aperture"], rho=case["rho"],
                             pack_format=case["fmt"])
        elif kind == "demigrate":
            st["op"] = _operator(case, sv)
            st["image"] = _model(case, seed)
            st["data"] = torch.empty((sv["mx"].numel(), st["op"].pitch), device=DEV)
        elif kind == "gradient":
            st["op"] = _operator(case, sv)
            st["packed"] = ktm.prepare(sv["traces"], sv["dt"], fmt=case["fmt"], rho=0,
                                       prefold=case["weight"] == "prefold")
            st["grad"] = _image(sv)
        elif kind == "lsm":
            st["op"] = _operator(case, sv)
            st["data"] = st["op"].pack(sv["traces"])
            st["iterations"] = case["iterations"]
        else:
            raise ValueError("unknown kind %r" % kind)
    return st


def run(st):
    kind = st["kind"]
    if kind == "dropin":
        return ktm.ktmMigrationCPU(*st["args"])
    if kind in ("reference", "fast", "raw"):
        return ktm.migrate(**st["job"])
    if kind == "batch":
        return ktm.migrate_batch(st["jobs"])
    if kind == "prep":
        p = ktm.prepare(st["in"], st["dt"], out=st["out"], out_scale=st["scale"], **st["args"])
        return p.data, p.scale
    if kind == "demigrate":
        return st["op"].demigrate(st["image"], st["data"])
    if kind == "gradient":
        return st["op"].vrms_gradient(st["packed"], st["grad"])
    model, residuals, gradients = st["op"].least_squares(st["data"], st["iterations"])
    return model, residuals, gradients


# --------------------------------------------------------------------------------- work ---
def _in_aperture(case, nx, ny):
    """Share of (image column, trace) pairs within the aperture."""
    ap = float(case.get("aperture", 0.0))
    if ap <= 0.0:
        return 1.0
    if case["geom"] == "line":
        x = 12.5 * np.arange(nx)
        return float(np.mean(np.abs(x[:, None] - x[None]) <= ap))
    r = np.random.default_rng(0)
    n, wx, wy = 20000, 25.0 * nx, 25.0 * ny
    dx = r.uniform(0, wx, n) - r.uniform(0, max(wx, 2000.0), n)
    dy = r.uniform(0, wy, n) - r.uniform(0, max(wy, 2000.0), n)
    return float(np.mean(dx * dx + dy * dy <= ap * ap))


def work(case):
    kind, nt = case["kind"], case["nt"]
    if kind == "prep":
        out = case["ntr"] * nt * (4 if case["fmt"] == "f32" else 2)
        m = 1 << max(1, math.ceil(math.log2(max(2, nt))))
        # two real transforms a trace (2.5 M log2 M each), the filter, fold and scaling
        fft = 0 if case["rho"] == "none" else 2 * 2.5 * m * math.log2(m) + 3 * m
        return {"bytes": case["ntr"] * (nt * 4 + 4) + out, "flops": case["ntr"] * (fft + 4 * nt)}
    esize = 2 if case.get("fmt") in ("f16", "bf16") and kind in ("fast", "batch", "gradient") else 4
    total = {"bytes": 0.0, "flops": 0.0}
    for part in range(case.get("jobs", 1)):
        if case["geom"] == "line":
            nx, ny, ntr = case["nx"], 1, case["nx"] * case["noff"]
        else:
            nx, ny, ntr = case["nx"], case["ny"], case["ntr"]
            if kind == "batch":
                nx, ny = max(2, nx - part % 5), max(2, ny + part % 3)
                ntr = max(20, int(ntr * (1.0 + (part % 4)) / 4.0))
        image, traces = nx * ny * case["nz"], ntr * nt
        pairs = image * ntr * _in_aperture(case, nx, ny)
        cube = case["geom"] == "areal" and kind == "fast"
        nbytes = traces * esize + 16 * ntr + image * 4 * (2 if cube else 1)
        # a pair: two DSR square roots, the sample index and fraction, the interpolation,
        # the weight and the sum; bit-exact mode adds its divisions and third square root
        flops = pairs * (24 if kind in ("dropin", "reference") else 20)
        if kind == "gradient":
            flops = pairs * 30
        if kind == "lsm":                            # L and L^T per iteration, and once before
            flops *= 2 * (case["iterations"] + 1)
        total["bytes"] += nbytes
        total["flops"] += flops
    return total


# -------------------------------------------------------------------------------- exact ---
def _rho64(x, dt, opt):
    """The rho filter of the reference's script, 64 bits: real part of the filtered trace."""
    if opt == 0:
        return x
    n = x.shape[1]
    m = 1
    while m < n:
        m *= 2
    k = torch.arange(m, device=x.device, dtype=torch.float64)
    k = torch.where(k < m // 2, k, k - m)
    w = 2.0 * math.pi * k / dt
    if opt == 1:
        h = torch.complex(w.abs(), torch.zeros_like(w))
    elif opt == 2:
        h = torch.polar(w.abs().sqrt(), math.pi / 4.0 * torch.sign(w))
    else:
        h = torch.complex(torch.zeros_like(w), w)
    return torch.fft.ifft(torch.fft.fft(x, n=m, dim=1) * h[None], dim=1).real[:, :n]


def _f32(x):
    return float(np.float32(x))


def _kin(sv, cols, aperture):
    """Per image column block: t/dt [C, ntr, nz] and the in-aperture mask [C, ntr], 64 bits."""
    ny, nz = sv["gy"][0], sv["gz"][0]
    ci, cj = cols // ny, cols % ny
    x = _f32(sv["gx"][2]) + ci.double() * _f32(sv["gx"][1])
    y = _f32(sv["gy"][2]) + cj.double() * _f32(sv["gy"][1])
    tau = _f32(sv["gz"][2]) + torch.arange(nz, device=DEV).double() * _f32(sv["gz"][1])
    mx, my, ox, oy = (sv[k].double() for k in ("mx", "my", "ox", "oy"))
    dx, dy = mx[None] - x[:, None], my[None] - y[:, None]
    ok = dx * dx + dy * dy <= aperture * aperture if aperture > 0 else torch.ones_like(dx).bool()
    ds = (dx - ox) ** 2 + (dy - oy) ** 2
    dr = (dx + ox) ** 2 + (dy + oy) ** 2
    v = sv["vel"].double()
    v = v.reshape(-1, nz)[cols] if v.dim() == 3 else v[None].expand(cols.numel(), nz)
    s, dt = 1.0 / (v * v), _f32(sv["dt"])
    t2 = (tau * tau)[None, None]
    u = torch.addcmul(t2, ds[:, :, None], s[:, None, :]).sqrt_()
    u += torch.addcmul(t2, dr[:, :, None], s[:, None, :]).sqrt_()
    u /= dt
    return u, ok, tau, dt, ds, dr, s


def _migrate64(sv, data, pick, weight, aperture):
    """data: 64-bit [ntr, nt], without the sqrt(t) weight.  weight: "prefold" interpolates
    the folded samples, anything else multiplies the pick by sqrt(t)."""
    ncol, nz, nt = sv["gx"][0] * sv["gy"][0], sv["gz"][0], sv["nt"]
    ntr = data.shape[0]
    dt = _f32(sv["dt"])
    j = torch.arange(nt, device=DEV).double()
    q = data.clone()
    q[:, 0] = 0.0
    if weight == "prefold":
        q = q * torch.sqrt(j * dt)[None]
    q = torch.nn.functional.pad(q, (0, 2)).reshape(-1)
    out = torch.empty((ncol, nz), device=DEV, dtype=torch.float64)
    rows = min(ntr, max(1, 120_000_000 // nz))
    step = max(1, 120_000_000 // (rows * nz))
    base = (torch.arange(ntr, device=DEV) * (nt + 2))
    for c0 in range(0, ncol, step):
        cols = torch.arange(c0, min(ncol, c0 + step), device=DEV)
        out[cols] = 0.0
        for k0 in range(0, ntr, rows):
            part = dict(sv, **{k: sv[k][k0:k0 + rows] for k in ("mx", "my", "ox", "oy")})
            u, ok, tau, _, _, _, _ = _kin(part, cols, aperture)
            u.clamp_(max=float(nt))
            i0 = u.floor()
            at = i0.long()
            at += base[k0:k0 + rows][None, :, None]
            if pick == "linear":
                a = q[at]
                a += (u - i0) * (q[at + 1] - a)
            else:
                a = q[at]
            if weight != "prefold":
                a *= torch.sqrt(u * dt)
            a *= ok[:, :, None]
            out[cols] += a.sum(1)
    tau = _f32(sv["gz"][2]) + torch.arange(nz, device=DEV).double() * _f32(sv["gz"][1])
    out *= tau.abs()[None]
    return out.reshape(sv["gx"][0], sv["gy"][0], nz)


def _demigrate64(sv, image, weight, aperture, pitch):
    """64-bit [ntr, pitch]: the transpose of _migrate64 with the linear pick."""
    ncol, nz, nt = sv["gx"][0] * sv["gy"][0], sv["gz"][0], sv["nt"]
    ntr, dt = sv["mx"].numel(), _f32(sv["dt"])
    out = torch.zeros(ntr * pitch, device=DEV, dtype=torch.float64)
    img = image.double().reshape(ncol, nz)
    rows = max(1, 120_000_000 // nz)
    for k0 in range(0, ntr, rows):
        part = dict(sv, **{k: sv[k][k0:k0 + rows] for k in ("mx", "my", "ox", "oy")})
        for c in range(ncol):
            pick = torch.arange(c, c + 1, device=DEV)
            u, ok, tau, _, _, _, _ = _kin(part, pick, aperture)
            keep = ok[0].nonzero()[:, 0]
            if keep.numel() == 0:
                continue
            u = u[0][keep]
            u.clamp_(max=float(nt))
            i0 = u.floor()
            f = u - i0
            val = (tau.abs() * img[c])[None].expand_as(u)
            if weight != "prefold":
                val = val * torch.sqrt(u * dt)
            at = i0.long() + ((keep + k0) * pitch)[:, None]
            right = val * f
            out.index_add_(0, at.reshape(-1), (val - right).reshape(-1))
            out.index_add_(0, (at + 1).reshape(-1), right.reshape(-1))
    out = out.reshape(ntr, pitch)
    out[:, 0] = 0.0
    out[:, nt:] = 0.0
    if weight == "prefold":
        out *= torch.sqrt(torch.arange(pitch, device=DEV).double() * dt)[None]
    return out


def _gradient64(sv, data, weight, aperture):
    """dI/dv: d/dv of |tau| sum_k W(u) V(u), W the linearly interpolated sqrt(j dt)."""
    ncol, nz, nt = sv["gx"][0] * sv["gy"][0], sv["gz"][0], sv["nt"]
    ntr, dt = data.shape[0], _f32(sv["dt"])
    j = torch.arange(nt + 2, device=DEV).double()
    root = torch.sqrt(j * dt)
    q = data.clone()
    q[:, 0] = 0.0
    if weight == "prefold":
        q = q * root[None, :nt]
    q = torch.nn.functional.pad(q, (0, 2)).reshape(-1)
    out = torch.zeros((ncol, nz), device=DEV, dtype=torch.float64)
    rows = min(ntr, max(1, 60_000_000 // nz))
    base = torch.arange(ntr, device=DEV) * (nt + 2)
    for c in range(ncol):
        col = torch.arange(c, c + 1, device=DEV)
        for k0 in range(0, ntr, rows):
            part = dict(sv, **{k: sv[k][k0:k0 + rows] for k in ("mx", "my", "ox", "oy")})
            u, ok, tau, _, ds, dr, s = _kin(part, col, aperture)
            # u = sqrt(T2 + Ds S) + sqrt(T2 + Dr S) over dt: du/dv = -(Ds/ls + Dr/lr) S / v / dt
            t2 = (tau * tau)[None, None]
            ls = torch.addcmul(t2, ds[:, :, None], s[:, None]).sqrt_()
            lr = torch.addcmul(t2, dr[:, :, None], s[:, None]).sqrt_()
            dudv = torch.where(ls > 0, ds[:, :, None] / ls, 0.0)
            dudv += torch.where(lr > 0, dr[:, :, None] / lr, 0.0)
            dudv *= (-s * s.sqrt())[:, None] / dt
            u.clamp_(max=float(nt))
            i0 = u.floor()
            f = u - i0
            i0 = i0.long()
            at = i0 + base[k0:k0 + rows][None, :, None]
            a = q[at]
            dv = q[at + 1] - a
            if weight == "prefold":
                term = dv
            else:
                w0 = root[i0]
                dw = root[i0 + 1] - w0
                term = dw * (a + f * dv) + (w0 + f * dw) * dv
            out[c] += ((term * dudv) * ok[:, :, None]).sum(1)[0] * tau.abs()
    return out.reshape(sv["gx"][0], sv["gy"][0], nz)


def _cgls64(sv, case):
    op = dict(weight=case["weight"], aperture=case["aperture"])
    nt = sv["nt"]
    d = sv["traces"].double().clone()
    d[:, 0] = 0.0

    def fwd(m):
        return _demigrate64(sv, m, op["weight"], op["aperture"], nt + 2)[:, :nt]

    def adj(r):
        return _migrate64(sv, r, "linear", op["weight"], op["aperture"])

    m = torch.zeros((sv["gx"][0], 1, sv["gz"][0]), device=DEV, dtype=torch.float64)
    r = d.clone()
    s = adj(r)
    p, gamma = s.clone(), float((s * s).sum())
    rn, gn = [float(r.norm())], [math.sqrt(gamma)]
    for _ in range(case["iterations"]):
        q = fwd(p)
        alpha = gamma / float((q * q).sum())
        m, r = m + alpha * p, r - alpha * q
        s = adj(r)
        new = float((s * s).sum())
        p, gamma = s + (new / gamma) * p, new
        rn.append(float(r.norm()))
        gn.append(math.sqrt(gamma))
    return m, np.array(rn), np.array(gn)


def exact(case, seed):
    kind = case["kind"]
    if kind == "prep":
        x = _prep_input(case, seed)
        nt, dt, fmt = int(case["nt"]), _f32(case["dt"]), case["fmt"]
        pitch = ktm_pitch(nt, fmt)
        out = torch.zeros((x.shape[0], pitch), device=DEV, dtype=torch.float64)
        rows = max(1, 60_000_000 // nt)
        for k in range(0, x.shape[0], rows):
            y = x[k:k + rows]
            if case["ibm"]:
                w = y.long() & 0xFFFFFFFF
                y = (w & 0xFFFFFF).double() / 16777215.0
                y = y * torch.pow(16.0, ((w >> 24) & 127).double() - 64.0)
                y = torch.where(w >> 31 > 0, -y, y)
            y = _rho64(y.double(), dt, RHO[case["rho"]])
            if case["prefold"]:
                y = y * torch.sqrt(torch.arange(nt, device=DEV).double() * dt)[None]
            out[k:k + rows, 1:nt] = y[:, 1:]
        top = out.abs().amax(1)
        scale = torch.where(top > 0, top / (32768.0 if fmt == "f16" else 1.0), 1.0)
        if fmt == "f32":
            scale = torch.ones_like(scale)
        return out / scale[:, None], scale
    if kind == "batch":
        return [_migrate64(sv, sv["traces"].double(), case["pick"], case["weight"],
                           case["aperture"])
                for sv in (_survey(case, seed, p) for p in range(case["jobs"]))]
    sv = _survey(case, seed)
    if kind in ("dropin", "reference"):
        return _migrate64(sv, sv["traces"].double(), "truncate", "table", 0.0)
    if kind == "fast":
        return _migrate64(sv, sv["traces"].double(), case["pick"], case["weight"],
                          case["aperture"])
    if kind == "raw":
        y = _rho64(sv["traces"].double(), _f32(sv["dt"]), RHO[case["rho"]])
        return _migrate64(sv, y, case["pick"], case["weight"], case["aperture"])
    if kind == "demigrate":
        return _demigrate64(sv, _model(case, seed), case["weight"], case["aperture"],
                            ktm_pitch(sv["nt"], "f32"))
    if kind == "gradient":
        return _gradient64(sv, sv["traces"].double(), case["weight"], case["aperture"])
    return _cgls64(sv, case)


def ktm_pitch(nt, fmt):
    """Samples between packed traces: tracePts + 2 rounded up to 16 bytes."""
    per = 4 if fmt == "f32" else 8
    return (nt + 2 + per - 1) // per * per
