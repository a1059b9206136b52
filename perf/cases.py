"""Performance cases of the wavefront-sensor engine: the calls a user's
program makes each frame, from an 8x8 SCAO sensor to the 74x74 ELT sensors,
through the public entry points, with their inputs (made from a seed), their
algorithmic work and, where the outputs are computed numbers, the same result
in 64 bits by plain torch.

Families (``kind``):

* ``frame``  one readout through ``centcmod.run`` with host numpy arrays, the
  reference's own calling pattern.
* ``batch``  independent frames of one sensor through ``run_batch``, device
  tensors.
* ``lgs``    one readout of a sensor with a spot PSF per subaperture (laser
  guide stars), device tensors.
* ``multi``  several sensors of uneven size per step (``WfsBatch``).
* ``slope``  a detector image to centroids (``runSlope``), host arrays: the
  real-camera path.
* ``corr``   correlation centroiding of a detector image, device tensors.
* ``screen`` one frame of a wind-blown layer: new lines extruded on the
  device, the pupil's window cut out.
* ``pupil``  the pupil phase of a star from several moving layers.
* ``recon``  the reconstructor step on the slope vector.

Frames with shot and read noise run the FP16 tensor-core form, as a closed
loop does; the FP32 and split-product forms run without noise, as interaction
matrices, calibration ramps and reference frames are recorded, so that their
images are computed numbers.
"""
import functools
import math

import numpy as np
import torch

from dasp_gb300.batch import WfsBatch
from dasp_gb300.centcmod import centcmod
from dasp_gb300.correlation import transform_psf
from dasp_gb300.infscreen import DeviceScreen, extrusion_matrices, phase_covariance, pupil_phase
from dasp_gb300.recon import Reconstructor
from dasp_gb300.tel import Pupil

OBS = 0.28  # central obstruction of every pupil here
SKY, FLOOR = 10.0, 6.0
SIG = 500.0  # photons per subaperture and frame


def listed():
    return [
        # the smallest call: one frame of an 8x8 SCAO sensor, the class's
        # default form; launches and host work are what it costs
        dict(name="frame_scao_8x8", kind="frame", form="fp32", nsubx=8, p=8, N=16, m=8, psf=False, noise=False),
        # the ELT sensor, one closed-loop frame at a time from host arrays
        dict(name="frame_elt_74x74", kind="frame", form="fp16", nsubx=74, p=10, N=20, m=10, psf=True, noise=True),
        # 64 independent closed-loop frames of the ELT sensor (Monte Carlo)
        dict(name="batch_elt_fp16", kind="batch", form="fp16", frames=64, nsubx=74, p=10, N=20, m=10, psf=True,
             noise=True),
        # the 2 x 8 tilt ramps of a centroid calibration, reference precision
        dict(name="batch_elt_fp32", kind="batch", form="fp32", frames=16, nsubx=74, p=10, N=20, m=10, psf=True,
             noise=False),
        # a poke sequence of a 40x40 sensor at split-product precision
        dict(name="batch_40x40_bf16x3", kind="batch", form="bf16x3", frames=50, nsubx=40, p=8, N=16, m=8, psf=True,
             noise=False),
        # one laser-guide-star sensor: an elongated spot per subaperture
        dict(name="lgs_74x74", kind="lgs", nsubx=74, p=10, N=32, m=16),
        # a tomographic step: laser and natural sensors in one graph
        dict(name="multi_3lgs_3ngs", kind="multi", lgs=3, nsubx=74, p=10, N=32, m=16),
        # a 740x740 camera frame to centroids, host in and out
        dict(name="slope_elt", kind="slope", nsubx=74, m=10, brightest=0),
        # extended-source tracking: correlation with a 20x20 reference
        dict(name="corr_elt", kind="corr", nsubx=74, m=10, cs=20, mode=1),
        # one fast layer of the ELT atmosphere, two new columns a frame
        dict(name="screen_elt", kind="screen", npup=740, lines=2, axis=0),
        # the ELT pupil through four layers
        dict(name="pupil_elt", kind="pupil", npup=740, layers=4),
        # 5316 actuators from the slopes of the 3972 lit subapertures
        dict(name="recon_elt", kind="recon", nacts=5316, ncents=7944, vectors=False),
    ]


KINDS = ("frame", "batch", "lgs", "multi", "slope", "corr", "screen", "pupil", "recon")
#: (fftsize, phasesizes) of the drawn sensors
FFTS = ((8, (4,)), (12, (6, 5)), (15, (7,)), (16, (8, 7)), (20, (10, 9)), (24, (12,)), (25, (12,)), (32, (16, 10)),
        (40, (20,)), (64, (32,)))
#: the largest listed work (flops): drawn cases stay below
MOST_FLOPS = 1e10


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(KINDS)
    if kind in ("frame", "batch"):
        form = rng.choice(("fp32", "fp32", "fp16", "fp16", "bf16x3", "tf32"))
        N, ps = rng.choice([f for f in FFTS if form == "fp32" or f[0] <= 24])
        c = dict(kind=kind, form=form, nsubx=_log(rng, 5, 74), p=rng.choice(ps), N=N,
                 m=rng.choice([m for m in (N // 2, N // 2, N // 4, N // 2 - 1, N) if 3 <= m <= 32]),
                 psf=rng.random() < 0.6, noise=form == "fp16")
        while _sensor_flops(c) > MOST_FLOPS / 16:
            c["nsubx"] = c["nsubx"] * 2 // 3
        if kind == "batch":
            c["frames"] = max(1, min(_log(rng, 1, 64), int(MOST_FLOPS / _sensor_flops(c))))
        return c
    if kind == "lgs":
        N, ps = rng.choice([f for f in FFTS if 16 <= f[0] <= 40 and f[0] % 2 == 0])
        return dict(kind=kind, nsubx=_log(rng, 8, 74 if N <= 32 else 40), p=rng.choice(ps), N=N,
                    m=rng.choice((N // 2, N // 4)))
    if kind == "multi":
        return dict(kind=kind, lgs=rng.randint(1, 4), nsubx=_log(rng, 16, 60), p=10, N=rng.choice((20, 32)), m=10)
    if kind == "slope":
        m = rng.randint(4, 20)
        return dict(kind=kind, nsubx=_log(rng, 8, 80), m=m, brightest=rng.choice((0, 0, m, 2 * m)))
    if kind == "corr":
        m = 2 * rng.randint(3, 8)
        return dict(kind=kind, nsubx=_log(rng, 8, 74), m=m, cs=m + 2 * rng.randint(0, m // 2),
                    mode=rng.choice((1, 1, 5)))
    if kind == "screen":
        return dict(kind=kind, npup=_log(rng, 32, 760), lines=rng.randint(1, 4), axis=rng.randint(0, 3))
    if kind == "pupil":
        return dict(kind=kind, npup=_log(rng, 40, 800), layers=rng.randint(1, 9))
    return dict(kind=kind, nacts=_log(rng, 400, 6000), ncents=_log(rng, 800, 8000), vectors=rng.random() < 0.5)


# ---------------------------------------------------------------- inputs

def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _annulus(npup):
    """The 0/1 pupil on the grid whose origin lies between its two central pixels."""
    x = torch.arange(npup, dtype=torch.float64, device="cuda") - npup / 2.0 + 0.5
    r = torch.sqrt(x[:, None] ** 2 + x[None, :] ** 2)
    return (r <= npup / 2.0) & (r >= npup / 2.0 * OBS)


def _phase(frames, npup, nsubx, seed, salt=0, wavelength=589.0):
    """Von Karman phase (radians) over a pupil of 0.53 m subapertures: r0
    0.157 m at 500 nm, L0 25 m; frames are rolls of a few screens."""
    d = 0.527 * nsubx
    n = 2 * npup
    f = torch.fft.fftfreq(n, d=d / npup, dtype=torch.float64, device="cuda")
    amp = (f[:, None] ** 2 + f[None, :] ** 2 + (1 / 25.0) ** 2) ** (-11.0 / 12.0)
    amp *= math.sqrt(0.0229) * 0.157 ** (-5.0 / 6.0) * n / (2 * d) * n / n
    g = _gen(seed, 17 + salt)
    out = torch.empty((frames, npup, npup), dtype=torch.float32, device="cuda")
    base = None
    for k in range(frames):
        if k % 8 == 0:
            w = torch.fft.fft2(torch.randn((n, n), generator=g, dtype=torch.float64, device="cuda"))
            base = torch.fft.ifft2(w * amp).real * (500.0 / wavelength)
        out[k] = torch.roll(base, (k * 37, k * 91), (0, 1))[:npup, :npup]
    return out


def _spot(n, fwhm):
    """A Gaussian spot of peak 1 centred between the middle pixels."""
    x = np.arange(n) - n // 2 + 0.5
    return np.exp(-4 * math.log(2) * (x[:, None] ** 2 + x[None, :] ** 2) / fwhm ** 2).astype(np.float32)


def _lgs_spots(nsubx, n, theta):
    """Spots elongated away from a launch point at the pupil's edge, unit sum."""
    pos = torch.arange(nsubx, dtype=torch.float64, device="cuda") - nsubx / 2.0 + 0.5
    xs = pos[:, None] + nsubx / 2.0 * math.cos(theta)
    ys = pos[None, :] + nsubx / 2.0 * math.sin(theta)
    r = torch.sqrt(xs ** 2 + ys ** 2)
    phi = torch.atan2(xs.expand_as(r), ys.expand_as(r))
    a, b = 1.2 / 2.3548, torch.sqrt((6.0 * r / r.max()) ** 2 + 1.2 ** 2) / 2.3548
    x = torch.arange(n, dtype=torch.float64, device="cuda") - n // 2 + 0.5
    u = x[None, None, None, :] * phi.cos()[..., None, None] + x[:, None] * phi.sin()[..., None, None]
    v = x[:, None] * phi.cos()[..., None, None] - x[None, None, None, :] * phi.sin()[..., None, None]
    s = torch.exp(-0.5 * ((u / b[..., None, None]) ** 2 + (v / a) ** 2))
    return (s / s.sum((-2, -1), keepdim=True)).to(torch.float32)


def _images(nsubx, m, seed, fwhm=2.5):
    """A detector image: one noisy spot per subaperture, tiled."""
    g = _gen(seed, 5)
    off = torch.randn((nsubx, nsubx, 2), generator=g, device="cuda") * 0.6
    x = torch.arange(m, device="cuda") - (m - 1) / 2.0
    ey = torch.exp(-4 * math.log(2) * (x[None, None] - off[..., :1]) ** 2 / fwhm ** 2)
    ex = torch.exp(-4 * math.log(2) * (x[None, None] - off[..., 1:]) ** 2 / fwhm ** 2)
    im = ey[..., :, None] * ex[..., None, :]
    im = im * (SIG / im.sum((-2, -1), keepdim=True)) + SKY
    im = im + im.sqrt() * torch.randn(im.shape, generator=g, device="cuda")
    return im.permute(0, 2, 1, 3).reshape(nsubx * m, nsubx * m).contiguous()


def _engine(c, phs, cents, bimg, psf=None, floor=FLOOR, noise=False, brightest=0, mode=0, pattern=None, corrimg=None,
            image=None, seed=0):
    p, N = c.get("p", 10), c.get("N", 20)
    npup = c["nsubx"] * p
    return centcmod(8, c["nsubx"], c["m"], N, N, c["m"], p, 3.0 if noise else 0.0, 0.0, 1 if noise else 0, floor, SIG,
                    SKY, 0, 1.0, 1, 0, 1000 + seed, phs, Pupil(npup, npup / 2.0, npup / 2.0 * OBS), psf, cents, bimg,
                    0.5, 0, None, mode, 0.0, pattern, corrimg, 0, 0, brightest, 1, 0, None, image, None)


def _spot_psf(c):
    return _spot(c["N"], 1.5) if c.get("psf") else None


#: the multi-sensor step's natural guide stars: (nsubx, phasesize, fftsize, nimg)
NGS = ((8, 8, 16, 8), (16, 16, 32, 16), (24, 32, 64, 16))


def _sensors(c):
    """The (sensor, launch angle or None) list of an ``lgs`` or ``multi`` case."""
    one = {k: c[k] for k in ("nsubx", "p", "N", "m")}
    if c["kind"] == "lgs":
        return [(one, 0.4)]
    return [(one, 0.4 + 2 * math.pi * k / c["lgs"]) for k in range(c["lgs"])] + \
        [(dict(zip(("nsubx", "p", "N", "m"), n), psf=True), None) for n in NGS]


_stream = None


def stream():
    """The one stream that a program of ours queues its work on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


@functools.lru_cache(maxsize=8)
def _matrices(n, scale):
    return extrusion_matrices(n, phase_covariance(n, 25.0, scale))


def _screen_shape(c):
    return (c["npup"] + 1, c["npup"] + 2) if c["axis"] in (0, 2) else (c["npup"] + 2, c["npup"] + 1)


def _screen_init(shape, seed, salt):
    n = max(shape)
    return _phase(1, n, max(1, n // 10), seed, salt, 500.0)[0, :shape[0], :shape[1]].contiguous()


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(kind=kind, case=c)
    if kind in ("frame", "batch"):
        W, ns = c["nsubx"] * c["p"], c["nsubx"] ** 2
        F = c.get("frames", 1)
        phs = _phase(F, W, c["nsubx"], seed)
        if kind == "frame":
            s.update(phs=phs[0].cpu().numpy(), cents=np.zeros(2 * ns, np.float32),
                     bimg=np.zeros((c["nsubx"], c["nsubx"], c["m"], c["m"]), np.float32))
            s["eng"] = _engine(c, s["phs"], s["cents"], s["bimg"], _spot_psf(c), noise=c["noise"], seed=seed)
        else:
            s.update(phs=phs, cents=torch.zeros((F, 2 * ns), device="cuda"),
                     bimg=torch.zeros((F, ns, c["m"], c["m"]), device="cuda"))
            s["eng"] = _engine(c, phs[0], s["cents"][0], s["bimg"][0], _spot_psf(c), noise=c["noise"], seed=seed)
        s["eng"].set_form(c["form"])
    elif kind in ("lgs", "multi"):
        s["engines"], s["out"] = [], []
        for k, (g, theta) in enumerate(_sensors(c)):
            ns = g["nsubx"] ** 2
            phs = _phase(1, g["nsubx"] * g["p"], g["nsubx"], seed, k)[0]
            cents = torch.zeros(2 * ns, device="cuda")
            bimg = torch.zeros((g["nsubx"], g["nsubx"], g["m"], g["m"]), device="cuda")
            psf = _spot_psf(g) if theta is None else _lgs_spots(g["nsubx"], g["N"], theta).cpu().numpy()
            e = _engine(g, phs, cents, bimg, psf, seed=seed)
            if theta is None:
                e.set_form("bf16x3")
            s["engines"].append(e)
            s["out"].append({"cents": cents, "bimg": bimg})
        if kind == "multi":
            s["batch"] = WfsBatch(s["engines"])
    elif kind in ("slope", "corr"):
        ns, m = c["nsubx"] ** 2, c["m"]
        image = _images(c["nsubx"], m, seed)
        if kind == "slope":
            s.update(image=image.cpu().numpy(), cents=np.zeros(2 * ns, np.float32),
                     bimg=np.zeros((c["nsubx"], c["nsubx"], m, m), np.float32))
            s["eng"] = _engine(c, None, s["cents"], s["bimg"], floor=12.0, brightest=c["brightest"], image=s["image"])
        else:
            cs = c["cs"]
            spots = np.ascontiguousarray(np.broadcast_to(_spot(cs, 2.5), (c["nsubx"], c["nsubx"], cs, cs)))
            s.update(image=image, cents=torch.zeros(2 * ns, device="cuda"),
                     bimg=torch.zeros((c["nsubx"], c["nsubx"], m, m), device="cuda"),
                     corrimg=torch.zeros((c["nsubx"], c["nsubx"], cs, cs), device="cuda"))
            s["eng"] = _engine(c, None, s["cents"], s["bimg"], floor=12.0, mode=c["mode"],
                               pattern=transform_psf(spots) if c["mode"] == 1 else spots, corrimg=s["corrimg"],
                               image=s["image"])
    elif kind == "screen":
        shape = _screen_shape(c)
        a, b = _matrices(c["npup"] + 1, 0.0527)
        mats = dict(ay=a, by=b) if c["axis"] in (0, 2) else dict(ax=a, bx=b)
        init = _screen_init(shape, seed, 3)
        s["screen"] = DeviceScreen(init.cpu().numpy(), 25.0, seed=seed, **mats)
        s["add"] = (s["screen"].add_columns, s["screen"].add_rows, s["screen"].add_columns_start,
                    s["screen"].add_rows_start)[c["axis"]]
        # the window holds the new lines: the far end of the screen, or the near one
        end = c["axis"] < 2
        s["at"] = (shape[0] - c["npup"], shape[1] - c["npup"]) if end else (0, 0)
        s["out"] = torch.zeros((c["npup"], c["npup"]), device="cuda")
    elif kind == "pupil":
        n = c["npup"]
        s["layers"] = [(scr, *_window(n, k)) for k, (scr, _) in enumerate(_layers(c, seed))]
        s["pupil"] = _annulus(n).to(torch.float32)
        s["area"] = float(s["pupil"].double().sum())
        s["out"] = torch.zeros((n, n), device="cuda")
    else:
        g = _gen(seed, 9)
        R = torch.randn((c["nacts"], c["ncents"]), generator=g, device="cuda") * 1e-3
        gain, decay = (0.5, 0.99) if not c["vectors"] else _vectors(c, seed)
        s["recon"] = Reconstructor(R, gain, decay)
        s["recon"].act.copy_(torch.randn(c["nacts"], generator=g, device="cuda"))
        s["slopes"] = torch.randn(c["ncents"], generator=g, device="cuda")
    torch.cuda.synchronize()
    return s


def _vectors(c, seed):
    r = np.random.default_rng([seed, 4])
    return (r.uniform(0.3, 0.6, c["nacts"]).astype(np.float32), r.uniform(0.98, 1.0, c["nacts"]).astype(np.float32))


#: lines that the layers of a ``pupil`` case have moved by
MOVED = 37


def _layers(c, seed):
    """Moving layers: (screen, its present content).  Even ones have moved
    along columns, odd ones along rows, by lines that repeat the last one."""
    n = c["npup"] + 3
    eye = np.hstack([np.zeros((n, n)), np.eye(n)])
    for k in range(c["layers"]):
        init = _screen_init((n, n), seed, 20 + k)
        mats = dict(ay=eye, by=np.zeros((n, n))) if k % 2 == 0 else dict(ax=eye, bx=np.zeros((n, n)))
        scr = DeviceScreen(init.cpu().numpy(), 25.0, seed=k, **mats)
        (scr.add_columns if k % 2 == 0 else scr.add_rows)(MOVED, 0.157)
        yield scr, init


def _window(n, k):
    """(y0, x0, yshift, xshift) of layer k"""
    return k % 3, (k + 1) % 3, (0.13 + 0.31 * k) % 1.0, (0.77 + 0.17 * k) % 1.0


# ---------------------------------------------------------------- one pass

def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["eng"].run(0)
    elif kind == "batch":
        s["eng"].run_batch(s["phs"], s["cents"], s["bimg"], stream=stream())
    elif kind == "lgs":
        s["engines"][0].run_async(stream())
        return s["out"]
    elif kind == "multi":
        s["batch"].run(stream())
        return s["out"]
    elif kind in ("slope", "corr"):
        s["eng"].runSlope(0)
        if kind == "corr":
            return {"cents": s["cents"], "bimg": s["bimg"], "corrimg": s["corrimg"]}
    elif kind == "screen":
        s["add"](s["case"]["lines"], 0.157, stream=stream())
        s["screen"].window(*s["at"], s["out"], stream=stream())
        return s["out"]
    elif kind == "pupil":
        return pupil_phase(s["layers"], s["pupil"], s["out"], pupil_area=s["area"], wavelength=589.0, stream=stream())
    else:
        return s["recon"].step(s["slopes"], stream=stream())
    return {"cents": s["cents"], "bimg": s["bimg"]}


# ---------------------------------------------------------------- work

def _lit(nsubx):
    """Lit subapertures of an annular pupil, at half-area threshold."""
    return max(1.0, math.pi / 4 * (1 - OBS ** 2) * nsubx ** 2)


def _sensor_flops(c):
    p, N, m = c["p"], c["N"], c["m"]
    f = 6 * p * p + 10 * N * N * math.log2(N) + 4 * N * N + 3 * m * m
    if c.get("psf") or c["kind"] in ("lgs", "multi"):
        f += 10 * N * N * math.log2(N) + 6 * N * (N // 2 + 1)
    return f * _lit(c["nsubx"])


def work(case):
    c, kind = case, case["kind"]
    if kind in ("frame", "batch"):
        F = c.get("frames", 1)
        return {"bytes": F * _lit(c["nsubx"]) * (4 * c["p"] ** 2 + 4 * c["m"] ** 2 + 8), "flops": F * _sensor_flops(c)}
    if kind in ("lgs", "multi"):
        b = f = 0.0
        for g, theta in _sensors(c):
            n = _lit(g["nsubx"])
            b += n * (4 * g["p"] ** 2 + 4 * g["m"] ** 2 + 8 + (8 * g["N"] * (g["N"] // 2 + 1) if theta is not None else 0))
            f += _sensor_flops(dict(g, kind=kind))
        return {"bytes": b, "flops": f}
    if kind in ("slope", "corr"):
        n, m, cs = _lit(c["nsubx"]), c["m"], c.get("cs", 0)
        f = 5 * m * m
        if kind == "corr":
            f += 10 * cs * cs * math.log2(cs) + 6 * cs * cs if c["mode"] == 1 else 1.5 * m ** 4
        return {"bytes": n * (8 * m * m + 8 + 8 * cs * cs), "flops": n * f}
    if kind == "screen":
        n = c["npup"] + 1
        return {"bytes": 24 * n * n + 8 * c["npup"] ** 2, "flops": 6 * n * n * c["lines"]}
    if kind == "pupil":
        n = c["npup"] ** 2
        return {"bytes": 4 * n * (c["layers"] + 2), "flops": n * (8 * c["layers"] + 5)}
    n = c["nacts"] * c["ncents"]
    return {"bytes": 4 * (n + c["ncents"] + 2 * c["nacts"]), "flops": 2 * n}


# ---------------------------------------------------------------- 64 bits

def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("frame", "batch"):
        if c["noise"]:
            return None
        psf = _spot_psf(c)
        phs = _phase(c.get("frames", 1), c["nsubx"] * c["p"], c["nsubx"], seed)
        got = [_exact_frame(c, ph, None if psf is None else torch.from_numpy(psf).cuda()) for ph in phs]
        if kind == "batch":
            return {"cents": torch.stack([g[0] for g in got]), "bimg": torch.stack([g[1] for g in got])}
        return {"cents": got[0][0], "bimg": got[0][1]}
    if kind in ("lgs", "multi"):
        out = []
        for k, (g, theta) in enumerate(_sensors(c)):
            ph = _phase(1, g["nsubx"] * g["p"], g["nsubx"], seed, k)[0]
            psf = torch.from_numpy(_spot_psf(g)).cuda() if theta is None else \
                _lgs_spots(g["nsubx"], g["N"], theta).reshape(-1, g["N"], g["N"])
            cents, bimg = _exact_frame(g, ph, psf)
            out.append({"cents": cents, "bimg": bimg})
        return out
    if kind in ("slope", "corr"):
        return _exact_image(c, seed)
    if kind == "screen":
        return _exact_screen(c, seed)
    if kind == "pupil":
        n = c["npup"]
        total = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        for k in range(c["layers"]):
            scr = _screen_init((n + 3, n + 3), seed, 20 + k).double()
            dim = 1 - k % 2
            last = scr.narrow(dim, n + 2, 1)
            scr = torch.cat([scr.narrow(dim, MOVED, n + 3 - MOVED)] + [last] * MOVED, dim) if n + 3 > MOVED else \
                last.expand_as(scr)
            y0, x0, ys, xs = _window(n, k)
            w = scr[y0:y0 + n + 1, x0:x0 + n + 1]
            total += (1 - xs) * ((1 - ys) * w[:n, :n] + ys * w[1:, :n]) + xs * ((1 - ys) * w[:n, 1:] + ys * w[1:, 1:])
        pup = _annulus(n).double()
        return (total - (total * pup).sum() / pup.sum()) * pup * (500.0 / 589.0)
    g = _gen(seed, 9)
    R = torch.randn((c["nacts"], c["ncents"]), generator=g, device="cuda") * 1e-3
    act = torch.randn(c["nacts"], generator=g, device="cuda").double()
    x = torch.randn(c["ncents"], generator=g, device="cuda").double()
    gain, decay = (0.5, float(np.float32(0.99)))
    if c["vectors"]:
        gain, decay = (torch.from_numpy(v).cuda().double() for v in _vectors(c, seed))
    return decay * act - gain * torch.cat([r.double() @ x for r in R.split(512)])


def _subaps(a, nsubx):
    """(nsubx * p, nsubx * p) -> (nsubx^2, p, p)"""
    p = a.shape[0] // nsubx
    return a.reshape(nsubx, p, nsubx, p).permute(0, 2, 1, 3).reshape(-1, p, p)


def _bin_matrix(C, m):
    """Binning of C points to m: each point's share to its own output and the
    rest to the next, the rest taken from the next point's value."""
    R = torch.zeros((m, C), dtype=torch.float64)
    if C == m:
        return torch.eye(C, dtype=torch.float64).cuda()
    cnt = o = 0
    for i in range(C):
        cnt += m
        over = max(0, cnt - C)
        R[o, i] += (m - over) / m
        if over and i < C - 1 and o + 1 < m:
            R[o + 1, i + 1] += over / m
        if cnt >= C:
            cnt = over
            o = min(o + 1, m - 1) if i < C - 1 else o
    return R.cuda()


def _cog(img):
    m = img.shape[-1]
    x = torch.arange(m, dtype=torch.float64, device="cuda")
    s = img.sum((-2, -1))
    ok = s > 0
    d = torch.where(ok, s, torch.ones_like(s))
    cx = (img.sum(-2) * x).sum(-1) / d - (m - 1) / 2.0
    cy = (img.sum(-1) * x).sum(-1) / d - (m - 1) / 2.0
    return torch.stack([torch.where(ok, cx, 0.0 * cx), torch.where(ok, cy, 0.0 * cy)], -1)


def _exact_frame(c, ph, psf):
    """One noise-free readout: (centroids, images), unlit subapertures 0."""
    nsubx, p, N, m = c["nsubx"], c["p"], c["N"], c["m"]
    pup = _subaps(_annulus(nsubx * p).double(), nsubx)
    area = pup.sum((-2, -1))
    lit = torch.nonzero(area >= 0.5 * p * p)[:, 0]
    k = torch.arange(p, dtype=torch.float64, device="cuda")
    tilt = math.pi * (N + 1.0) / N * (k[:, None] + k[None, :] + 1 - p)
    ph = _subaps(ph.double(), nsubx)
    R = _bin_matrix(N, m)
    cents = torch.zeros((nsubx * nsubx, 2), dtype=torch.float64, device="cuda")
    bimg = torch.zeros((nsubx * nsubx, m, m), dtype=torch.float64, device="cuda")
    for i in lit.split(2048):
        t = ph[i] - tilt
        e = torch.complex(pup[i] * t.cos(), pup[i] * t.sin())
        img = torch.fft.fft2(e, s=(N, N)).abs().square().flip((-2, -1))
        scale = SIG * (area[i] / (p * p)) / (area[i] * N * N)
        if psf is not None:
            q = psf.double() if psf.dim() == 2 else psf[i].double()
            spec = torch.fft.rfft2(torch.roll(q, (-(N // 2), -(N // 2)), (-2, -1)))
            img = torch.fft.irfft2(torch.fft.rfft2(img) * spec, s=(N, N))
            scale = scale / q.sum((-2, -1))
        img = R @ img @ R.T * scale[:, None, None] + (SKY * area[i] / (p * p))[:, None, None]
        img = torch.clamp(img - FLOOR, min=0.0)
        bimg[i] = img
        cents[i] = _cog(img)
    return cents.reshape(-1), bimg


def _exact_image(c, seed):
    nsubx, m = c["nsubx"], c["m"]
    lit = _subaps(_annulus(nsubx * 10).double(), nsubx).sum((-2, -1)) >= 50
    img = torch.clamp(_subaps(_images(nsubx, m, seed), nsubx).double() - 12.0, min=0.0) * lit[:, None, None]
    if c["kind"] == "slope":
        if 0 < c["brightest"] < m * m:
            f = img.reshape(-1, m * m)
            thr = f.sort(-1).values[:, m * m - c["brightest"]]
            img = torch.where(f < thr[:, None], 0.0 * f, f).reshape(-1, m, m)
        return {"cents": _cog(img).reshape(-1), "bimg": img}
    cs = c["cs"]
    o = (cs - m) // 2
    pad = torch.zeros((img.shape[0], cs, cs), dtype=torch.float64, device="cuda")
    pad[:, o:o + m, o:o + m] = img
    spot = torch.from_numpy(_spot(cs, 2.5)).cuda().double()
    if c["mode"] == 1:  # circular, unnormalised
        spec = torch.fft.fft2(torch.fft.fftshift(spot)).conj()
        corr = torch.fft.ifft2(torch.fft.fft2(pad) * spec).real * (cs * cs)
        corr = torch.clamp(corr, min=0.0)
    else:  # overlap sums for offsets within the image
        corr = torch.zeros_like(pad)
        d0 = (cs - m) // 2

        def overlap(i):
            off = i - m // 2
            ref, at, n = max(0, -off + d0), max(0, off - d0), m
            n = min(n, m - at)
            return ref, at, min(n, cs - ref)
        for i in range(m):
            ry, iy, ny = overlap(i)
            for j in range(m):
                rx, ix, nx = overlap(j)
                corr[:, i + d0, j + d0] = (spot[ry:ry + ny, rx:rx + nx] * img[:, iy:iy + ny, ix:ix + nx]).sum((-2, -1))
    corr = corr * lit[:, None, None]
    n = cs
    x = torch.arange(n, dtype=torch.float64, device="cuda")
    f = corr.reshape(-1, n * n)
    # centre of gravity in the ncen x ncen window about the brightest pixel
    pos = f.argmax(-1)
    sx = torch.clamp((pos % n - m / 2.0 + 0.5).trunc(), 0, n - m)
    sy = torch.clamp((pos // n - m / 2.0 + 0.5).trunc(), 0, n - m)
    wx = (x >= sx[:, None]) & (x < sx[:, None] + m)
    wy = (x >= sy[:, None]) & (x < sy[:, None] + m)
    w = corr * wy[:, :, None] * wx[:, None, :]
    s = w.sum((-2, -1))
    ok = s > 0
    d = torch.where(ok, s, torch.ones_like(s))
    cx = (w.sum(-2) * x).sum(-1) / d + sx - (n - 1) / 2.0
    cy = (w.sum(-1) * x).sum(-1) / d + sy - (n - 1) / 2.0
    cents = torch.stack([torch.where(ok, cx, 0.0 * cx), torch.where(ok, cy, 0.0 * cy)], -1)
    return {"cents": cents.reshape(-1), "bimg": img, "corrimg": corr}


def _philox(key, ctr):
    """Philox4x32-10 (Salmon et al., SC'11) on arrays of four counter words."""
    m32 = np.uint64(0xFFFFFFFF)
    x, y, z, w = (np.asarray(v, np.uint64) for v in ctr)
    k0, k1 = np.uint64(key & 0xFFFFFFFF), np.uint64((key >> 32) & 0xFFFFFFFF)
    for _ in range(10):
        p, q = x * np.uint64(0xD2511F53), z * np.uint64(0xCD9E8D57)
        x, y, z, w = (q >> np.uint64(32)) ^ y ^ k0, q & m32, (p >> np.uint64(32)) ^ w ^ k1, p & m32
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m32, (k1 + np.uint64(0xBB67AE85)) & m32
    return x, y, z, w


def _normals(seed, line, n):
    """The screen's normals of one extruded line: Box-Muller on the first two
    words of element j's block (counter 0, purpose 3, j, line)."""
    zero = np.zeros(n, np.uint64)
    w = _philox(seed, (zero, zero + np.uint64(3 << 24), np.arange(n, dtype=np.uint64), zero + np.uint64(line)))
    u1, u2 = (((v >> np.uint64(8)).astype(np.float64) + 0.5) / 16777216.0 for v in w[:2])
    return -np.sqrt(-2.0 * np.log(u1)) * np.cos(2 * math.pi * u2 - math.pi)


def _exact_screen(c, seed):
    a, b = (torch.from_numpy(v).cuda() for v in _matrices(c["npup"] + 1, 0.0527))
    rows, start = c["axis"] in (1, 3), c["axis"] >= 2
    scr = _screen_init(_screen_shape(c), seed, 3).double()
    if rows:
        scr = scr.T
    for k in range(c["lines"]):
        z = torch.cat([scr[:, 1], scr[:, 0]] if start else [scr[:, -2], scr[:, -1]])
        g = torch.from_numpy(_normals(seed, k, c["npup"] + 1)).cuda()
        new = (a @ z + (b @ g) * (25.0 / 0.157) ** (5.0 / 6.0))[:, None]
        scr = torch.cat([new, scr[:, :-1]], 1) if start else torch.cat([scr[:, 1:], new], 1)
    if rows:
        scr = scr.T
    n = c["npup"]
    y, x = (0, 0) if start else (scr.shape[0] - n, scr.shape[1] - n)
    return scr[y:y + n, x:x + n].contiguous()
