"""The work a program gives this framework, as cases that can be timed.

Every case is a reconstruction (or a batch of them) that a program already
holds: the handles exist, the measured intensity, the support and a starting
estimate are on the device.  One pass is what such a program then does over and
over: iterate a number of times, perhaps tighten the support, and read the
estimate and the error metric back.

Two kinds of start are used.  The FP64 form is reproducible to the last bit, so
its cases start as a reconstruction does, from a random phase with Poisson noise
in the data.  In the FP32 form an early HIO run multiplies any rounding
difference until no two arithmetics agree on the estimate, so its cases are the
late part of a reconstruction: a tight support, an estimate half a per cent away
from the solution, and noise-free data except under ER, which is stable on noisy
data too.  The work per iteration is the same.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "nadia-coecxs_b200"))
import pynadia  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
BETA = 0.9
LINES = 10           # spectrum lines of a PolyCDI case
FP32_SIZES = (256, 512, 768, 1024, 1536, 2048)
# grids whose padded transform is 256, 512 or 1080 points (the FP32 PolyCDI form)
POLY32_GRIDS = ((240, 8), (480, 16), (1024, 28), (496, 8), (1040, 20), (1008, 36))

# FresnelCDI: 8 keV, focus to sample 1 mm, focus to detector 1 m
FRESNEL = dict(wavelength=1.23984198e-9 / 8.0, focal_detector_length=1.0,
               focal_sample_length=1e-3, pixel_size=13.5e-6)
# FresnelCDI_WF: the reference example's zone plate
WF = dict(wavelength=4.892e-10, zone_focal_length=16.353e-3,
          focal_detector_length=0.909513 - 16.353e-3, pixel_size=13.5e-6)


def case(kind, fp, nx, ny, count=1, algorithm="HIO", iterations=32, shrink=0, step=0, stop=0,
         pad=0, mixed=0, name=None):
    """kind: planar, fresnel, poly, fresnel_wf; fp: 64 or 32; count: reconstructions
    stepped together; shrink: a shrinkwrap after every so many iterations; step: 1
    where the program calls iterate() once at a time and reads the error each time;
    stop: side of the central beam stop; mixed: 1 where the batch's sizes run over
    the FP32 sizes up to nx."""
    c = dict(kind=kind, fp=fp, nx=nx, ny=ny, count=count, algorithm=algorithm,
             iterations=iterations, shrink=shrink, step=step, stop=stop, pad=pad, mixed=mixed)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a test pattern, stepped one iteration at a time with the error printed
        # each time, as the reference's examples do: launches and latency count
        case("planar", 64, 128, 128, iterations=16, step=1, name="planar64_128_stepwise"),
        # the plain workload: 256^2 HIO with a shrinkwrap every 20 iterations
        case("planar", 64, 256, 256, iterations=40, shrink=20, name="planar64_256_shrinkwrap"),
        # a detector crop with odd sides
        case("planar", 64, 645, 475, iterations=16, name="planar64_645x475"),
        # the ER stretch of the 1024^2 workload
        case("planar", 64, 1024, 1024, algorithm="ER", iterations=50, name="planar64_1024_er"),
        # 2048^2 in the reference's double precision, with a beam stop
        case("planar", 64, 2048, 2048, iterations=32, stop=8, name="planar64_2048"),
        # curved-beam data on a detector that is not a power of two
        case("fresnel", 64, 1000, 1200, iterations=32, name="fresnel64_1000x1200"),
        # polychromatic data, double precision (padded to 640^2)
        case("poly", 64, 600, 600, pad=20, iterations=24, name="poly64_600"),
        # the short ER stretch that ends an FP32 reconstruction
        case("planar", 32, 512, 512, algorithm="ER", iterations=50, shrink=50, name="planar32_512_shrinkwrap"),
        # random restarts of the 2048^2 workload stepped together
        case("planar", 32, 2048, 2048, count=4, iterations=100, stop=8, name="planar32_2048_x4"),
        # curved-beam data of several detector crops in one call
        case("fresnel", 32, 2048, 2048, count=5, mixed=1, iterations=50,
             name="fresnel32_mixed_x5"),
        # the polychromatic requests of a server: 1024^2, padded to 1080^2
        case("poly", 32, 1024, 1024, count=4, pad=28, iterations=32, name="poly32_1024_x4"),
        # white-field recovery at the example's size
        case("fresnel_wf", 32, 2048, 2048, iterations=26, name="wf32_2048"),
    ]


def largest_prime(n):
    p, f = 1, 2
    while n > 1:
        while n % f == 0:
            n //= f
            p = f
        f += 1
    return p


def draw(rng):
    def side(lo, hi, even):
        while True:
            n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
            n += n & 1 if even else 0
            if largest_prime(n) <= 131:
                return n

    def steps(pixels, lo=8, hi=36):
        # so that no drawn case iterates over more pixels than the largest listed one
        return max(lo, min(hi, int(2e8 / pixels), int(rng.uniform(lo, hi))))

    family = rng.choice(["planar64", "planar64", "fresnel64", "poly64", "planar32", "planar32",
                         "fresnel32", "poly32", "wf32", "wf64"])
    alg = rng.choice(["HIO", "HIO", "ER", "RAAR"])
    if family == "planar64":
        square = rng.random() < 0.5
        nx = side(64, 2048, False)
        ny = nx if square else side(64, 2048, False)
        n = steps(nx * ny)
        shrink = rng.choice([0, max(4, n // 2)]) if square and nx % 2 == 0 else 0
        return case("planar", 64, nx, ny, algorithm=alg, iterations=n, shrink=shrink,
                    step=0 if shrink else int(rng.random() < 0.25),
                    stop=rng.choice([0, 6]))
    if family == "fresnel64":
        nx, ny = side(64, 2048, True), side(64, 2048, True)
        return case("fresnel", 64, nx, ny, algorithm=alg, iterations=steps(nx * ny))
    if family == "poly64":
        while True:
            n, pad = side(64, 1100, True), rng.randrange(4, 29)
            if largest_prime(n + 2 * pad) <= 131:
                break
        return case("poly", 64, n, n, pad=pad, algorithm=alg, iterations=steps(n * n))
    if family == "wf64":
        n = side(64, 1600, True)
        return case("fresnel_wf", 64, n, n, iterations=steps(n * n, 8, 30))
    if family == "wf32":
        nx, ny = rng.choice(FP32_SIZES), rng.choice(FP32_SIZES)
        return case("fresnel_wf", 32, nx, ny, iterations=steps(nx * ny, 8, 30))
    if family == "poly32":
        n, pad = rng.choice(POLY32_GRIDS)
        return case("poly", 32, n, n, pad=pad, count=rng.randrange(1, 5), algorithm=alg,
                    iterations=rng.randrange(8, 40))
    nx, ny = rng.choice(FP32_SIZES), rng.choice(FP32_SIZES)
    count = rng.randrange(1, 6) if nx * ny > 1 << 20 else rng.randrange(1, 9)
    kind = family[:-2]
    return case(kind, 32, nx, ny, algorithm=alg, count=count, iterations=rng.randrange(8, 60 if kind == "fresnel" else 100),
                stop=rng.choice([0, 8]) if kind == "planar" else 0)


# ------------------------------------------------------------------- inputs

def sizes(c):
    """(nx, ny) of each reconstruction of a case."""
    if not c["mixed"]:
        return [(c["nx"], c["ny"])] * c["count"]
    pick = [s for s in FP32_SIZES if 512 <= s <= c["nx"]]
    return [(pick[k % len(pick)],) * 2 for k in range(c["count"])]


def rand(g, nx, ny):
    return torch.rand(nx, ny, generator=g, device=DEV, dtype=torch.float64)


def gauss(g, nx, ny):
    return torch.complex(torch.randn(nx, ny, generator=g, device=DEV, dtype=torch.float64),
                         torch.randn(nx, ny, generator=g, device=DEV, dtype=torch.float64))


def disk(nx, ny, radius):
    i = torch.arange(nx, device=DEV, dtype=torch.float64)[:, None] - nx / 2.0
    j = torch.arange(ny, device=DEV, dtype=torch.float64)[None, :] - ny / 2.0
    return i * i + j * j <= radius * radius


def smooth(a, sigma):
    """Periodic Gaussian blur of a real array."""
    kx = torch.fft.fftfreq(a.shape[0], device=DEV, dtype=torch.float64)[:, None]
    ky = torch.fft.fftfreq(a.shape[1], device=DEV, dtype=torch.float64)[None, :]
    h = torch.exp(-2 * (math.pi * sigma) ** 2 * (kx * kx + ky * ky))
    return torch.fft.ifft2(torch.fft.fft2(a.to(torch.complex128)) * h).real


def disk_object(g, nx, ny, radius, sigma):
    """Transmission inside a centred disk: amplitude in [0.5, 1], smoothed phase."""
    amp = 0.5 + 0.5 * rand(g, nx, ny)
    ph = smooth((rand(g, nx, ny) - 0.5) * math.pi, sigma)
    return torch.where(disk(nx, ny, radius), torch.polar(amp, ph), torch.zeros((), dtype=torch.complex128, device=DEV))


def folded(m):
    """Distance of each index from the middle as multiply_factors folds it."""
    mid = (m - 1) / 2.0
    k = torch.arange(m, device=DEV, dtype=torch.float64)
    return mid - torch.trunc(mid - (mid - k).abs())


def fresnel_coef(nx, ny):
    zfd, zsd = FRESNEL["focal_detector_length"], FRESNEL["focal_detector_length"] - FRESNEL["focal_sample_length"]
    f = FRESNEL["pixel_size"] ** 2 * math.pi / FRESNEL["wavelength"] * (1 / zfd - 1 / zsd)
    a, b = folded(nx)[:, None], folded(ny)[None, :]
    phi = f * (a * a + b * b)
    return torch.complex(torch.cos(phi), torch.sin(phi))


def wf_coef(nx, ny):
    sx = WF["wavelength"] * WF["focal_detector_length"] / (WF["pixel_size"] * nx)
    sy = WF["wavelength"] * WF["focal_detector_length"] / (WF["pixel_size"] * ny)
    rho2 = (sx * folded(nx))[:, None] ** 2 + (sy * folded(ny))[None, :] ** 2
    phi = (rho2 / WF["zone_focal_length"] + rho2 / WF["focal_detector_length"]) * math.pi / WF["wavelength"]
    return torch.complex(torch.sin(phi), -torch.cos(phi)) / math.sqrt(nx * ny)


def swap(a):
    """The quadrant swap with 1/sqrt(N); on odd grids the pairwise swap visits
    some elements twice and others never."""
    nx, ny = a.shape
    s = 1.0 / math.sqrt(nx * ny)
    if nx % 2 == 0 and ny % 2 == 0:
        return torch.fft.fftshift(a) * s
    a, mx, my = a.clone(), nx // 2, ny // 2
    for i in range(nx):
        o = i + mx - (2 * mx if i >= mx else 0)
        t = a[o, my:2 * my].clone()
        a[o, my:2 * my] = a[i, :my] * s
        a[i, :my] = t * s
    return a


def to_detector(kind, x, coef):
    if kind == "fresnel":
        return torch.fft.fft2(swap(x)) * coef.conj()
    if kind == "fresnel_wf":
        return torch.fft.fft2(swap(torch.fft.fft2(x) * coef.conj()))
    return swap(torch.fft.fft2(x))


def from_detector(kind, f, coef):
    n = f.numel()
    if kind == "fresnel":
        return swap(torch.fft.ifft2(f * coef) * n)
    if kind == "fresnel_wf":
        return torch.fft.ifft2(swap(torch.fft.ifft2(f) * n) * coef) * n
    return torch.fft.ifft2(swap(f)) * n


def spectrum(c):
    """Ten Gaussian lines, longest wavelength first, spaced so that the padding
    derived from the first line is c["pad"]."""
    r = (2 * c["pad"] + 1) / c["nx"]
    span = 9 * r / (8 - r)
    k = np.arange(LINES)
    d = span * (9 - 2 * k) / 9
    w = np.exp(-(9 - 2.0 * k) ** 2 / 30.0)
    return np.stack([1e-10 * (1 + d), w], axis=1)


def expanded(c, psi):
    """sqrt of the polychromatic intensity on the unpadded window."""
    n, p = c["nx"], c["pad"]
    sp = spectrum(c)
    w = sp[:, 1] / sp[:, 1].sum()
    lc = sp[int(np.argmax(sp[:, 1])), 0]
    m2 = psi.real ** 2 + psi.imag ** 2
    i = torch.arange(n, device=DEV, dtype=torch.float64) + p
    acc = torch.zeros(n, n, device=DEV, dtype=torch.float64)
    for wl, wt in zip(sp[:, 0], w):
        v = (wl / lc) * (i - n / 2.0) + n / 2.0
        ok = (v >= 0) & (v < n + 2 * p)
        at = v.clamp(0, n + 2 * p - 1).long()
        acc += wt * m2[at][:, at] * (ok[:, None] & ok[None, :])
    return acc.sqrt()


def padded(c, x):
    p = c["pad"]
    return torch.nn.functional.pad(x, (p, p, p, p))


def inputs(c, nx, ny, seed):
    """Intensity, support, start estimate (and beam stop, white field) of one
    reconstruction, as float64 or complex128 tensors."""
    kind, late = c["kind"], c["fp"] == 32 or c["kind"] == "fresnel_wf"
    g = torch.Generator(device=DEV).manual_seed(seed)
    noisy = not late or c["algorithm"] == "ER"
    m = min(nx, ny)
    d = dict(stop=None, white=None)
    if c["stop"]:
        s, d["stop"] = c["stop"], torch.ones(nx, ny, device=DEV, dtype=torch.float64)
        d["stop"][nx // 2 - s // 2:nx // 2 + s // 2, ny // 2 - s // 2:ny // 2 + s // 2] = 0
    if kind == "fresnel_wf":
        r = 0.3 * m
        i = torch.arange(nx, device=DEV, dtype=torch.float64)[:, None] - nx / 2.0
        j = torch.arange(ny, device=DEV, dtype=torch.float64)[None, :] - ny / 2.0
        ph = smooth((rand(g, nx, ny) - 0.5) * 2 * math.pi, 3.0) + 0.5 * ((i * i + j * j) / (r * r)) ** 2
        zone = disk(nx, ny, 0.95 * r) * torch.polar(torch.ones_like(ph), ph)
        truth = to_detector(kind, zone, wf_coef(nx, ny))
        rms = truth.abs().square().mean().sqrt()
        return dict(d, intensity=truth.abs().square(), support=disk(nx, ny, r).double(),
                    start=truth + 0.005 * rms * gauss(g, nx, ny))
    if kind == "fresnel":
        i = torch.arange(nx, device=DEV, dtype=torch.float64)[:, None] - nx / 2.0
        j = torch.arange(ny, device=DEV, dtype=torch.float64)[None, :] - ny / 2.0
        r2, rf = i * i + j * j, 0.42 * m
        amp = smooth((r2 <= rf * rf).double(), 2.0).clamp(min=0)
        d["white"] = torch.polar(100.0 * amp, (math.pi / 8) / (2 * rf) * r2)
        coef = fresnel_coef(nx, ny)
        ill = from_detector(kind, d["white"], coef)
        t = torch.polar(0.8 + 0.2 * rand(g, nx, ny), smooth((rand(g, nx, ny) - 0.5) * math.pi / 2, 2.0))
        t = torch.where(disk(nx, ny, 0.3 * m), t, torch.ones((), dtype=torch.complex128, device=DEV))
        truth = (t - 1) * ill
        inten = (to_detector(kind, truth, coef) + d["white"]).abs().square()
        inten = torch.poisson(inten, generator=g) if noisy else inten
        d["support"] = disk(nx, ny, 0.3 * m if late else 0.33 * m).double()
        if late:
            rms = truth.abs().square().mean().sqrt()
            return dict(d, intensity=inten, start=truth + 0.005 * rms * gauss(g, nx, ny))
        start = -0.2 * rand(g, nx, ny) * ill * d["support"]   # as initialise_estimate draws it
        return dict(d, intensity=inten, start=start)
    radius = 0.16 * m
    obj = disk_object(g, nx, ny, radius, 2.0)
    if kind == "poly":
        inten = expanded(c, to_detector(kind, padded(c, obj), None)).square()
    else:
        inten = torch.fft.fftshift(torch.fft.fft2(obj)).abs().square() / (nx * ny)
    scale = 1e8 / inten.sum()
    inten, obj = inten * scale, obj * scale.sqrt()
    total = inten.sum()
    inten = torch.poisson(inten, generator=g) if noisy else inten
    if late:
        inside = disk(nx, ny, radius)
        rms = obj.abs().square().sum().div(inside.sum()).sqrt()
        return dict(d, intensity=inten, support=inside.double(),
                    start=obj + 0.005 * rms * gauss(g, nx, ny))
    side = int(2.5 * radius)
    sup = torch.zeros(nx, ny, device=DEV, dtype=torch.float64)
    sup[nx // 2 - side // 2:nx // 2 + side // 2, ny // 2 - side // 2:ny // 2 + side // 2] = 1
    amp = (total / sup.sum()).sqrt()
    start = sup * amp * torch.polar(torch.ones_like(sup), 2 * math.pi * rand(g, nx, ny))
    return dict(d, intensity=inten, support=sup, start=start)


# --------------------------------------------------------------------- runs

def prepare(case, seed):
    c, fp = case, case["fp"]
    precision = pynadia.FP64 if fp == 64 else pynadia.FP32
    solvers, starts, supports = [], [], []
    for k, (nx, ny) in enumerate(sizes(c)):
        d = inputs(c, nx, ny, seed * 64 + k)
        kw = {}
        if c["kind"] == "fresnel":
            kw = dict(FRESNEL, white_field=d["white"].cpu().numpy())
        elif c["kind"] == "fresnel_wf":
            kw = WF
        s = pynadia.Solver(c["kind"], nx, ny, precision=precision, **kw)
        if c["kind"] == "poly":
            s.set_spectrum(spectrum(c))
        support = d["support"].cpu().numpy()
        s.set_support(support)
        s.set_intensity(d["intensity"].cpu().numpy())
        if d["stop"] is not None:
            s.set_beam_stop(d["stop"].cpu().numpy())
        start = d["start"].cpu().numpy()
        if fp == 64:
            s.set_exit_surface_wave(start)
        else:
            start = start.astype(np.complex64)
            s.set_exit_surface_wave_f32(start)
        if c["kind"] != "fresnel_wf":
            s.set_relaxation_parameter(BETA)
            s.set_algorithm(c["algorithm"])
        solvers.append(s)
        starts.append(start)
        supports.append(support)
    return dict(case=c, solvers=solvers, starts=starts, supports=supports)


def tells(c):
    """Whether the error metric of an FP32 case says anything: on noise-free data
    near the solution it is the sum of squared rounding errors."""
    return c["algorithm"] == "ER" and c["kind"] != "fresnel_wf"


def run(state):
    c, solvers = state["case"], state["solvers"]
    f64, errors = c["fp"] == 64, []
    first = solvers[0]
    if c["shrink"]:
        # a new run of the schedule: the estimate and the support go back to the start
        first.set_support(state["supports"][0])
        (first.set_exit_surface_wave if f64 else first.set_exit_surface_wave_f32)(state["starts"][0])
    if c["step"]:
        for _ in range(c["iterations"]):
            first.iterate()
            errors.append(first.get_error())
    else:
        left = c["iterations"]
        while left:
            n = min(left, c["shrink"] or left)
            if len(solvers) > 1:
                pynadia.iterate_many(solvers, n)
            else:
                first.iterate(n)
            left -= n
            if c["shrink"]:
                first.apply_shrinkwrap(1.5, 0.1)
        errors = [s.get_error() for s in solvers]
    if f64:
        out = dict(estimate=[first.get_exit_surface_wave()], error=np.array(errors))
        if c["shrink"]:
            out["support"] = first.get_support()
        return out
    out = dict(estimate=[s.get_exit_surface_wave_f32() for s in solvers])
    if tells(c):
        # the FP32 form's error metric is good to its own precision
        out["error"] = np.array(errors, dtype=np.float32)
    return out


# --------------------------------------------------------------- 64 bits

def exact_one(c, nx, ny, seed):
    """(estimate, errors, support) of one reconstruction after one pass."""
    d = inputs(c, nx, ny, seed)
    kind, alg = c["kind"], c["algorithm"]
    x = d["start"] if c["fp"] == 64 else d["start"].to(torch.complex64).to(torch.complex128)
    sup, b = d["support"], BETA
    mag = d["intensity"].sqrt()
    seen = torch.ones_like(mag, dtype=torch.bool) if d["stop"] is None else d["stop"] > 0
    norm = (mag * mag)[seen].sum()
    coef = {"fresnel": fresnel_coef, "fresnel_wf": wf_coef}.get(kind, lambda *_: None)(nx, ny)
    errors = []

    def modulus(f, value):
        a = f.abs()
        return torch.where(a == 0, value + 0j, f * (value / torch.where(a == 0, 1.0, a)))

    def project(x):
        if kind == "poly":
            p = c["pad"]
            psi = to_detector(kind, padded(c, x), None)
            calc = expanded(c, psi)
            errors.append(((mag - calc)[seen] ** 2).sum() / norm)
            ratio = torch.where(seen, torch.where(calc == 0, 0.0, mag / torch.where(calc == 0, 1.0, calc)), 1.0)
            psi[p:p + nx, p:p + ny] *= ratio
            return from_detector(kind, psi, None)[p:p + nx, p:p + ny]
        f = to_detector(kind, x, coef)
        if kind == "fresnel":
            f = f + d["white"]
        errors.append(((f.abs() - mag)[seen] ** 2).sum() / norm)
        f = torch.where(seen, modulus(f, mag), f)
        if kind == "fresnel":
            f = f - d["white"]
        return from_detector(kind, f, coef)

    for it in range(c["iterations"]):
        if kind == "fresnel_wf":
            f = to_detector(kind, from_detector(kind, x, coef) * sup, coef)
            errors.append(((f.abs() - mag) ** 2).sum() / norm)
            x = modulus(f, mag)
        else:
            y = project(x)
            if alg == "ER":
                x = sup * y
            elif alg == "HIO":
                x = x - b * y - sup * x + (1 + b) * sup * y
            else:  # RAAR with this library's weights
                x = b * x - b * y - b * sup * x + (1 + b) * sup * y
        if c["shrink"] and ((it + 1) % c["shrink"] == 0 or it + 1 == c["iterations"]):
            t = torch.arange(-4, 5, device=DEV, dtype=torch.float64)
            w = torch.exp(-(t[:, None] ** 2 + t[None, :] ** 2) / (2 * 1.5 * 1.5))
            v = torch.nn.functional.conv2d(x.abs()[None, None], w[None, None], padding=4)[0, 0]
            sup = (v >= 0.1 * v.max()).double()
    return x.cpu().numpy(), [float(e) for e in errors], sup.cpu().numpy()


def exact(case, seed):
    c, fp = case, case["fp"]
    done = [exact_one(c, nx, ny, seed * 64 + k) for k, (nx, ny) in enumerate(sizes(c))]
    errors = np.array(done[0][1] if c["step"] else [d[1][-1] for d in done])
    out = dict(estimate=[d[0] for d in done])
    if fp == 64 or tells(c):
        out["error"] = errors
    if c["shrink"] and fp == 64:
        out["support"] = done[0][2]
    return out


def work(case):
    """Per iteration the estimate, the magnitudes and the support are read and the
    estimate is written; a projection is two 2-D transforms.  At the end the
    estimate goes to the host."""
    c = case
    z = 16 if c["fp"] == 64 else 8
    total_b = total_f = 0.0
    for nx, ny in sizes(c):
        n = nx * ny
        fields = 1 if c["kind"] in ("planar", "fresnel_wf", "poly") else 2   # the white field
        mx, my = nx + 2 * c["pad"], ny + 2 * c["pad"]
        transforms = 4 if c["kind"] == "fresnel_wf" else 2
        per_b = n * (2 * z + 2 * (z // 2) + (fields - 1) * z)
        per_f = transforms * 5.0 * mx * my * math.log2(mx * my) + 30.0 * n
        if c["kind"] == "poly":
            per_f += n * LINES * 6.0
        total_b += c["iterations"] * per_b + n * z
        total_f += c["iterations"] * per_f
    return {"bytes": total_b, "flops": total_f}
