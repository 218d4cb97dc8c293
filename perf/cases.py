"""Performance cases: the work a user has this framework do, with its inputs.

Every case goes through the public Python binding of the C API
(``libspimage_b200``): a phaser with its amplitudes, start and support in
hand advances by some iteration slots and hands back its model and Fourier
error; a host image is transformed; a set of reconstructions is turned into a
PRTF.  ``listed`` holds the fixed cases, ``draw`` one more of the same ranges,
``prepare``/``run`` the set-up and the measured call, ``work`` the bytes and
operations a pass cannot do without, ``exact`` the same results in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

import libspimage_b200 as L
from libspimage_b200 import prtf as prtf_api

ALGORITHMS = {"hio": L.SpHIO, "raar": L.SpRAAR, "dm": L.SpDiffMap, "er": L.SpER}
RULES = {"area": L.SpSupportArea, "threshold": L.SpSupportThreshold}


def _phase(name, shape, alg, slots, beta=0.9, starts=1, period=20, rule="area", value=0.05, constraints=2):
    nz, ny, nx = (1,) * (3 - len(shape)) + tuple(shape)
    return {"name": name, "kind": "phase", "nz": nz, "ny": ny, "nx": nx, "alg": alg, "beta": beta, "starts": starts,
            "slots": slots, "period": period, "rule": rule, "value": value, "constraints": constraints}


def listed():
    return [
        # one support period of a small crop: launches and latency count
        _phase("hio 64x64", (64, 64), "hio", 20),
        # a binned detector frame, the plain single reconstruction of the benchmark
        _phase("hio 256x256", (256, 256), "hio", 200),
        # the benchmark's headline: one full detector frame with RAAR
        _phase("raar 1024x1024", (1024, 1024), "raar", 200, beta=0.87, period=50),
        # a frame cropped to a round, non-power-of-two size (the mixed batches' largest)
        _phase("hio 1000x1000", (1000, 1000), "hio", 100),
        # a 1300 x 1340 CCD frame binned by two: axes with prime factors 13 and 67
        _phase("raar 650x670", (650, 670), "raar", 20, beta=0.87, rule="threshold", value=0.2),
        # the difference map (two transform pairs an iteration), real object
        _phase("dm 512x512", (512, 512), "dm", 200, beta=0.8, constraints=1),
        # an assembled 3-D intensity, the volume of the mixed and serving workloads
        _phase("hio 128x128x128", (128, 128, 128), "hio", 100),
        # a larger volume on a size that is not a power of two, refined with ER
        _phase("er 192x192x192", (192, 192, 192), "er", 20, period=10),
        # one job of the serving mix: eight random starts of a binned frame
        _phase("hio 8 starts 256x256", (256, 256), "hio", 200, starts=8),
        # a batch of random starts that exceeds the L2 cache (throughput)
        _phase("hio 32 starts 512x512", (512, 512), "hio", 400, starts=32),
        # a transform of one host image, as sp_image_fft gives it
        {"name": "fft 900x1200", "kind": "fft", "nz": 1, "ny": 900, "nx": 1200, "sign": -1},
        # the transfer function over a few finished reconstructions
        {"name": "prtf 8 of 256x256", "kind": "prtf", "nz": 1, "ny": 256, "nx": 256, "images": 8},
    ]


def _largest_prime(n):
    p, big = 2, 1
    while n > 1:
        if n % p == 0:
            big, n = p, n // p
        else:
            p += 1 if p * p <= n else n - p
    return big


def _axis(rng, lo, hi):
    """An axis length, spread over its logarithm: powers of two, 2^a 3^b 5^c
    and ragged lengths (no prime factor above 67: users crop away from those)."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    style = rng.random()
    if style < 0.3:
        return min(hi, max(lo, 1 << int(round(math.log2(n)))))
    top = 5 if style < 0.65 else 67
    while _largest_prime(n) > top:
        n -= 1
    return n


def draw(rng):
    kind = rng.choices(["single", "volume", "batch", "fft", "prtf"], [45, 20, 20, 8, 7])[0]
    dims = 3 if kind == "volume" or (kind == "fft" and rng.random() < 0.3) else 2
    lo, hi = {"single": (48, 1400), "volume": (24, 192), "batch": (32, 512), "fft": (48, 2048), "prtf": (64, 512)}[kind]
    if dims == 3:
        lo, hi = 24, 192
    n = _axis(rng, lo, hi)
    shape = [n] * dims if rng.random() < 0.6 else [_axis(rng, max(lo, n // 2), n) for _ in range(dims)]
    nz, ny, nx = [1] * (3 - dims) + shape
    if kind == "fft":
        return {"kind": "fft", "nz": nz, "ny": ny, "nx": nx, "sign": rng.choice([-1, 1])}
    if kind == "prtf":
        return {"kind": "prtf", "nz": nz, "ny": ny, "nx": nx, "images": rng.randint(3, 8)}
    starts = int(round(math.exp(rng.uniform(math.log(2), math.log(48))))) if kind == "batch" else 1
    # the pass stays below the largest listed one; ragged axes get fewer slots
    room = 8e6 if max(_largest_prime(s) for s in shape) > 5 else 2.4e8
    most = max(4, min(200, int(room / (nz * ny * nx * starts))))
    slots = rng.randint(max(2, most // 4), most)
    rule = rng.choice(["area", "area", "threshold"])
    c = _phase("", (nz, ny, nx), rng.choice(["hio", "hio", "raar", "raar", "er", "dm"]), slots,
               beta=round(rng.uniform(0.7, 0.95), 3), starts=starts, period=rng.choice([10, 20, 50]), rule=rule,
               value=0.05 if rule == "area" else 0.2, constraints=rng.choice([0, 1, 2, 2, 4]))
    del c["name"]
    return c


# ------------------------------------------------------------------- inputs
def _shape(case):
    return (case["ny"], case["nx"]) if case["nz"] == 1 else (case["nz"], case["ny"], case["nx"])


def _distance(shape):
    """Distance of every pixel from the zero frequency at index 0, in pixels."""
    r2 = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for ax, n in enumerate(shape):
        i = torch.arange(n, dtype=torch.float64, device="cuda")
        r2 += (torch.minimum(i, n - i) ** 2).reshape([-1 if a == ax else 1 for a in range(len(shape))])
    return r2.sqrt()


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _object(shape, g):
    """A smoothed random block of a quarter of the frame, centred on index 0."""
    obj = torch.zeros(shape, dtype=torch.float64, device="cuda")
    blob = max(2, min(shape) // 4)
    obj[tuple(slice(0, blob) for _ in shape)] = torch.rand([blob] * len(shape), dtype=torch.float64, device="cuda",
                                                         generator=g)
    for ax, n in enumerate(shape):  # Gaussian of sigma 2 pixels
        f = torch.fft.fftfreq(n, dtype=torch.float64, device="cuda")
        w = torch.exp(-2.0 * (math.pi * 2.0 * f) ** 2).reshape([-1 if a == ax else 1 for a in range(len(shape))])
        obj = torch.fft.ifft(torch.fft.fft(obj, dim=ax) * w, dim=ax).real
    return torch.roll(obj, [-(blob // 2)] * len(shape), list(range(len(shape)))), blob


def _pattern(case, seed):
    """(amplitudes with photon noise and a beamstop, mask, initial support, random-phase start)."""
    shape = _shape(case)
    g = _generator(seed)
    obj, blob = _object(shape, g)
    inten = torch.fft.fftn(obj).abs() ** 2
    inten *= 50.0 * inten.numel() / inten.sum()  # fifty photons a pixel, most of them near the centre
    amp = torch.poisson(inten, generator=g).sqrt()
    r = _distance(shape)
    mask = r >= max(1.0, min(shape) / 64.0)
    amp = torch.where(mask, amp, torch.zeros_like(amp)).float()
    phase = 2.0 * math.pi * torch.rand(shape, dtype=torch.float64, device="cuda", generator=g)
    start = torch.fft.ifftn(torch.polar(amp.double(), phase)).to(torch.complex64)
    return amp, mask, r < 0.75 * blob, start


def _images(case, seed):
    """Reconstructions of one object as a run of random starts leaves them:
    shifted by a few pixels, turned by a global phase, slightly different."""
    shape, n = _shape(case), case["images"]
    g = _generator(seed)
    obj, blob = _object(shape, g)
    dims = list(range(len(shape)))
    sup = _distance(shape) < 0.75 * blob
    shifts = torch.randint(-3, 4, (n, len(shape)), generator=torch.Generator().manual_seed(seed)).tolist()
    ims, sups = [], []
    for k in range(n):
        phi = 2.0 * math.pi * torch.rand((), dtype=torch.float64, device="cuda", generator=g)
        noise = torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)
        im = obj * torch.polar(torch.ones_like(phi), phi) + 0.02 * obj.abs().max() * noise * sup
        ims.append(torch.roll(im, shifts[k], dims))
        sups.append(torch.roll(sup, shifts[k], dims))
    return torch.stack(ims).to(torch.complex64).cpu().numpy(), torch.stack(sups).int().cpu().numpy()


def _host_image(case, seed):
    shape = _shape(case)
    return torch.randn(shape, dtype=torch.complex64, device="cuda", generator=_generator(seed))


def prepare(case, seed):
    if case["kind"] == "fft":
        return {"case": case, "x": _host_image(case, seed).cpu().numpy()}
    if case["kind"] == "prtf":
        ims, sups = _images(case, seed)
        return {"case": case, "images": ims, "supports": sups}
    shape = _shape(case)
    amp, mask, support, start = _pattern(case, seed)
    ph = L.Phaser(shape)
    ph.set_algorithm(ALGORITHMS[case["alg"]], beta=case["beta"], constraints=case["constraints"])
    ph.add_support_update(RULES[case["rule"]], case["period"], 2.0, case["value"])
    ph.start()
    if case["starts"] > 1:
        ph.set_starts(case["starts"])
    ph.set_amplitudes(amp.cpu().numpy(), mask.int().cpu().numpy())
    if case["starts"] > 1:
        rc = ph.init_models_device(L.SpModelRandomPhases, [seed * 1000 + b for b in range(case["starts"])])
    else:
        rc = ph.init_model(0, model=start.cpu().numpy())
    if rc:
        raise RuntimeError("starting model failed (%d)" % rc)
    ph.set_support(support.cpu().numpy())
    # the images a program reads its starts into, once for the run
    out = [_Image(shape) for _ in range(case["starts"])] if case["starts"] > 1 else []
    return {"case": case, "ph": ph, "out": out}


class _Image:
    """A library image that lives as long as somebody looks at it."""

    def __init__(self, shape):
        self.img = L.new_image(shape=shape)

    def __del__(self):
        L.free_image(self.img)


def _pixels(img, shape, owner):
    """The pixels of a library image where they are; the view keeps `owner` alive."""
    buf = (ctypes.c_float * (2 * math.prod(shape))).from_address(img.contents.image.contents.data)
    buf.owner = owner
    return np.frombuffer(buf, np.complex64).reshape(shape)


def run(state):
    case = state["case"]
    shape = _shape(case)
    if case["kind"] == "fft":
        return L.fft(state["x"], case["sign"])
    if case["kind"] == "prtf":
        return prtf_api.prtf(state["images"], state["supports"])
    ph = state["ph"]
    rc = ph.iterate(case["slots"])
    if rc:
        raise RuntimeError("sp_phaser_iterate returned %d" % rc)
    if case["starts"] == 1:
        return {"model": _pixels(ph.lib.sp_phaser_model(ph.ph), shape, ph), "efourier": ph.efourier()[0]}
    for b, out in enumerate(state["out"]):
        if ph.lib.sp_phaser_start_model(ph.ph, b, out.img):
            raise RuntimeError("sp_phaser_start_model failed")
    return {"models": [_pixels(out.img, shape, out) for out in state["out"]], "efourier": ph.starts_efourier()[0]}


def work(case):
    """Bytes and operations of one pass.  A transform of N points costs
    5 N log2 N operations.  An iteration of a multi-dimensional iterate that
    lives in device memory reads and writes the iterate (8 + 8 bytes a pixel),
    reads the amplitudes (4) and the two masks (bits), and passes the spectrum
    between the axes once each way (16 + 16); the difference map has a second
    spectrum.  The images that go to or come from the host are counted once."""
    n = case["nz"] * case["ny"] * case["nx"]
    fft = 5.0 * n * math.log2(n)
    if case["kind"] == "fft":
        return {"bytes": 16.0 * n, "flops": fft}
    if case["kind"] == "prtf":
        k = case["images"]
        return {"bytes": 12.0 * n * k + 12.0 * n, "flops": k * (5 * fft + 60.0 * n)}
    pairs = 2 if case["alg"] == "dm" else 1
    slots = case["slots"] * case["starts"]
    per = 4.25 + 32.0 * pairs + (8.0 if case["alg"] == "er" else 16.0)
    return {"bytes": slots * n * per + 8.0 * n * case["starts"], "flops": slots * pairs * (2 * fft + 40.0 * n)}


# ------------------------------------------------------- the same in 64 bits
def _constrain(g, inside, c):
    re, im = g.real.clone(), g.imag.clone()
    if c & 3:
        im[inside] = 0
    if c & 6:
        re[inside & (re < 0)] = 0
    if c & 4:
        im[inside & (im < 0)] = 0
    return torch.complex(re, im)


def _exact_phase(case, seed):
    amp, mask, inside, g = _pattern(case, seed)
    amp, g = amp.double(), g.to(torch.complex128)
    n, alg = g.numel(), case["alg"]
    beta = float(np.float32(case["beta"]))
    blur = torch.exp(-2.0 * math.pi ** 2 * (_distance(g.shape) / g.shape[-1]) ** 2 * 4.0)
    s = 0.1
    gamma1 = float(np.float32(-(4 + (2 + beta) * s + beta * s * s) / (beta * (4 - s + s * s))))
    gamma2 = float(np.float32((3 - beta) / (2 * beta)))

    def modulus(x):  # onto the measured amplitudes
        X = torch.fft.fftn(x)
        m = amp / X.abs()
        P = torch.where(torch.isfinite(m), X * m, amp.to(X.dtype))
        return torch.fft.ifftn(torch.where(mask, P, X))

    it = 0
    while it < case["slots"]:
        if it % case["period"] == case["period"] - 1:  # a support update takes a slot
            b = torch.fft.ifftn(torch.fft.fftn(g.abs()) * blur).abs()
            value = float(np.float32(case["value"]))
            if case["rule"] == "area":
                rank = int(np.float32(n) * np.float32(value))
                t = torch.sort(b.flatten(), descending=True).values[min(rank, n - 1)]
            else:
                t = b.max() * value
            inside = b > t
        elif alg == "dm":
            rho = modulus(g)
            f1 = modulus(torch.where(inside, g, -gamma1 * g))
            g = torch.where(inside, g + beta * ((1 + gamma2) * rho - gamma2 * g), g)
            g = _constrain(g - beta * f1, inside, case["constraints"])
        else:
            p = modulus(g)
            out = {"hio": g - beta * p, "raar": (1 - 2 * beta) * p + beta * g, "er": torch.zeros_like(p)}[alg]
            g = _constrain(torch.where(inside, p, out), inside, case["constraints"])
        it += 1
    F = torch.fft.fftn(g).abs()
    nom = ((F - amp) ** 2)[mask].sum()
    den = (amp ** 2)[mask].sum() + (F ** 2)[~mask].sum()
    return {"model": g.cpu().numpy(), "efourier": float((nom / den).sqrt())}


def _exact_prtf(case, seed):
    """The alignment of the reference's prtf in 64 bits: each image is moved
    to the peak of its moduli's correlation with the running sum (or, where the
    convolution's peak is higher, turned round first), then phased to it."""
    ims, _ = _images(case, seed)
    ims = torch.from_numpy(ims).cuda().to(torch.complex128)
    dims = list(range(ims.dim() - 1))
    total = ims[0].clone()
    phasors = torch.zeros_like(total)
    dead = torch.zeros(total.shape, dtype=torch.bool, device="cuda")

    def add(im):
        F = torch.fft.fftn(im)
        a = F.abs()
        dead.logical_or_(a == 0)
        phasors.add_(torch.where(a > 0, F / a, torch.zeros_like(F)))

    add(total)
    for im in ims[1:]:
        A, B = torch.fft.fftn(total.abs()), torch.fft.fftn(im.abs())
        corr = torch.fft.ifftn(A * B.conj()).real
        conv = torch.fft.ifftn(A * B).real
        turned = bool(conv.max() > corr.max())
        at = np.unravel_index(int((conv if turned else corr).argmax()), tuple(total.shape))
        if turned:
            im = torch.flip(im, dims).conj()
            at = [p + 1 for p in at]
        im = torch.roll(im, [int(p) for p in at], dims)
        z = (total * im.conj()).sum()
        im = im * (z / z.abs())
        total = total + im
        add(im)
    out = torch.where(dead, torch.zeros_like(phasors.real), phasors.abs() / len(ims))
    return {"prtf": torch.fft.fftshift(out).cpu().numpy(), "super_image": total.cpu().numpy()}


def exact(case, seed):
    """What run gives on a new state, in 64 bits; None where rounding alone
    decides the result: a reconstruction amplifies it from slot to slot, and
    device-drawn starts have no value here."""
    if case["kind"] == "fft":
        x = _host_image(case, seed).to(torch.complex128)
        return (torch.fft.fftn(x) if case["sign"] < 0 else torch.fft.ifftn(x, norm="forward")).cpu().numpy()
    if case["kind"] == "prtf":
        return _exact_prtf(case, seed)
    if case["starts"] > 1 or case["slots"] > 20:
        return None
    return _exact_phase(case, seed)
