"""The work a user of this framework has it do, as measurable cases.

Each case goes through the Python entry points of the package on inputs that
its seed fixes: `prepare` makes what a program has in hand before the call
(patterns, start iterates, a context, a trained network's weights), `run` is
one pass, `exact` the same results in 64-bit arithmetic from plain torch, and
`work` the bytes and operations a pass cannot do without.  The sizes are
those of the repository's configurations and benchmark; `draw` spreads over
the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cdixx_gb300 import native as cdx
from cdixx_gb300 import ptycho as pty
from cdixx_gb300 import unet

BETA = 0.9            # HIO / RAAR feedback of the configurations
SHRINK = 0.1          # shrinkwrap threshold
OPTICS = dict(lam=0.6328, d=125e3, dpupil=6800.0, pixelsize=13.0, exposure=0.01)   # the benchmark's ptychography
LENGTHS = [96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048]


# --------------------------------------------------------------------- the cases
def listed():
    return [
        # one measured frame of the plain configuration, new data each time: a few CTAs' worth of work,
        # so launches and latency count
        dict(name="job_256", kind="job", rows=256, cols=256, photons=1e6, algo="15*HIO+1*shrinkWrap+25*ER"),
        # the large single pattern: a complex phase object, RAAR, a shrinkwrap, then error reduction
        dict(name="job_2048", kind="job", rows=2048, cols=2048, photons=1e9, algo="15*RAAR+1*shrinkWrap+35*ER"),
        # a host program's one call (pinned buffers in and out, the context kept between calls)
        dict(name="host_1024", kind="host", rows=1024, cols=1024, photons=1e8, algo="15*RAAR+1*shrinkWrap+85*ER"),
        # detector-model projection with a beamstop on an oblong detector, positivity steps
        dict(name="ccd_768x1536", kind="ccd", rows=768, cols=1536, photons=1e7, algo="3*POSHIO+1*shrinkWrap+37*ER"),
        # fresh random starts on a batch of equal patterns kept on the device: the throughput path
        dict(name="starts_192", kind="starts", rows=192, cols=192, batch=96, photons=1e6, algo="10*HIO+110*ER"),
        dict(name="starts_512", kind="starts", rows=512, cols=512, batch=48, photons=1e7, algo="10*HIO+110*ER"),
        # the uneven batch: five sizes in one group run
        dict(name="group_uneven", kind="group", sizes="128x20,192x22,256x21,384x20,512x20", photons=1e7,
             algo="10*HIO+110*ER"),
        # the transform by itself, forward and back: many small oblong fields, and one of the largest length
        dict(name="fft_96x192", kind="fft", rows=96, cols=192, batch=9),
        dict(name="fft_4096", kind="fft", rows=4096, cols=4096, batch=1),
        # the learned start: a handful of patterns through the network to Psi0 and support
        dict(name="unet_infer", kind="infer", n=256, batch=8, levels=4, base=32),
        # one training step: forward, loss, backward, Adam
        dict(name="unet_train", kind="train", n=256, batch=32, levels=4, base=32),
        # sweeps of the benchmark's ptychography (object phase with the TV step, momentum)
        dict(name="ptycho_512", kind="ptycho", probe=512, obj=1280, step=250.0, sweeps=40, first=0, zernike=1200),
    ]


def draw(rng):
    kind = rng.choice(["job", "job", "host", "ccd", "starts", "starts", "group", "fft", "fft", "infer", "train", "ptycho"])
    photons = 10.0 ** rng.uniform(5, 8)
    if kind in ("job", "host", "ccd"):
        rows = rng.choice(LENGTHS)
        cols = rows if kind == "job" and rng.random() < 0.6 else rng.choice(LENGTHS)
        a, b = rng.randint(2, 4 if kind == "ccd" else 12), rng.randint(8, 30)
        first = {"job": rng.choice(["HIO", "RAAR", "FHIO"]), "host": "RAAR", "ccd": "POSHIO"}[kind]
        return dict(kind=kind, rows=rows, cols=cols, photons=max(photons, rows * cols * 4.0),
                    algo="%d*%s+1*shrinkWrap+%d*ER" % (a, first, b))
    if kind == "starts":
        rows, cols = rng.choice(LENGTHS[:7]), rng.choice(LENGTHS[:7])
        if rng.random() < 0.6:
            cols = rows
        most = max(1, 12_000_000 // (rows * cols))
        return dict(kind=kind, rows=rows, cols=cols, batch=max(1, int(most ** rng.uniform(0.3, 1.0))), photons=photons,
                    algo="%d*HIO+%d*ER" % (rng.randint(2, 10), rng.randint(10, 100)))
    if kind == "group":
        sizes = rng.sample(LENGTHS[:6], rng.randint(2, 5))
        return dict(kind=kind, sizes=",".join("%dx%d" % (s, rng.randint(1, 20)) for s in sorted(sizes)),
                    photons=photons, algo="%d*RAAR+%d*ER" % (rng.randint(2, 10), rng.randint(10, 60)))
    if kind == "fft":
        n = [16, 32, 48, 64] + LENGTHS + [3072, 4096]
        rows, cols = rng.choice(n), rng.choice(n)
        most = max(1, (1 << 24) // (rows * cols))
        return dict(kind=kind, rows=rows, cols=cols, batch=max(1, min(512, int(most ** rng.random()))))
    if kind in ("infer", "train"):
        n = rng.choice([64, 128, 192, 256, 384, 512])
        most = max(1, 32 * 256 * 256 // (n * n) // (1 if kind == "train" else 2))
        return dict(kind=kind, n=n, batch=max(1, min(64, int(most ** rng.uniform(0.2, 1.0)))),
                    levels=rng.choice([3, 4]), base=rng.choice([16, 32]))
    probe = rng.choice([128, 192, 256, 384, 512])
    phase = rng.choice([dict(first=0, zernike=1200), dict(first=0, zernike=0), dict(first=400, zernike=0)])
    return dict(kind="ptycho", probe=probe, obj=int(probe * rng.uniform(2.2, 2.6)) // 2 * 2,
                step=float(round(probe * rng.uniform(0.3, 0.5))), sweeps=rng.randint(5, 20), **phase)


# --------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _grid(rows, cols):
    y = torch.arange(rows, device="cuda", dtype=torch.float32)[:, None] - rows / 2
    x = torch.arange(cols, device="cuda", dtype=torch.float32)[None, :] - cols / 2
    return y, x


def _blobs(rows, cols, batch, g):
    """Sums of 8 Gaussian blobs in a centred disk a quarter of the field wide (real, positive)."""
    y, x = _grid(rows, cols)
    r = min(rows, cols) / 8
    u = torch.rand(4, batch, 8, 1, 1, device="cuda", generator=g)
    rad, ang = r * u[0].sqrt(), 2 * math.pi * u[1]
    sig, amp = 2 + 4 * u[2], 0.3 + 0.7 * u[3]
    o = torch.zeros(batch, rows, cols, device="cuda")
    for k in range(8):
        d2 = (y - (rad * ang.sin())[:, k]) ** 2 + (x - (rad * ang.cos())[:, k]) ** 2
        o += amp[:, k] * torch.exp(-d2 / (2 * sig[:, k] ** 2))
    return o * (y * y + x * x <= r * r)


def _smooth(rows, cols, sigma, g):
    """Gaussian-smoothed white noise scaled to [0, 1]."""
    f = torch.fft.fftfreq(rows, device="cuda")[:, None] ** 2 + torch.fft.fftfreq(cols, device="cuda")[None, :] ** 2
    v = torch.fft.ifft2(torch.fft.fft2(torch.randn(rows, cols, device="cuda", generator=g)) *
                        torch.exp(-2 * (math.pi * sigma) ** 2 * f)).real
    return (v - v.min()) / (v.max() - v.min())


def _phase_object(rows, cols, g):
    """Amplitude in [0.5, 1] and phase in [0, pi], smooth, in a support with a wavy boundary."""
    y, x = _grid(rows, cols)
    th, r0 = torch.atan2(y, x), min(rows, cols) / 8
    rb = torch.full_like(th, r0)
    ab = torch.randn(5, 2, device="cuda", generator=g) * 0.03 * r0
    for k in range(1, 6):
        rb += (ab[k - 1, 0] * torch.cos(k * th) + ab[k - 1, 1] * torch.sin(k * th)) / k
    o = torch.polar(0.5 + 0.5 * _smooth(rows, cols, 4.0, g), math.pi * _smooth(rows, cols, 4.0, g))
    return o * (y * y + x * x <= rb * rb)


def _patterns(case, rows, cols, batch, g):
    """Poisson-sampled |FFT(object)|^2 at the case's photon count, FFT order, [batch, rows, cols]."""
    o = _phase_object(rows, cols, g)[None] if min(rows, cols) >= 1024 else _blobs(rows, cols, batch, g)
    i = torch.fft.fft2(o.to(torch.complex64)).abs() ** 2
    i *= case["photons"] / i.sum((1, 2), keepdim=True)
    return torch.poisson(i, generator=g)


def _random_phase(i, g):
    return torch.where(torch.rand(i.shape, device="cuda", generator=g) > 0.5, -1.0, 1.0) * i.sqrt() + 0j


def _beamstop(rows, cols):
    """A disk over the low frequencies, FFT order."""
    y, x = _grid(rows, cols)
    return torch.fft.ifftshift((y * y + x * x < 9.0).float()).contiguous()


def _params(case, rows, cols, batch=1):
    more = dict(sim_ccd_bit=1, noise_level=4, exposure=2e-4) if case["kind"] == "ccd" else {}
    return cdx.default_params(rows, cols, batch=batch, beta=BETA, shrink_threshold=SHRINK, oversampling_spt=4.0, **more)


def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]


def _job_inputs(case, seed):
    g = _gen(seed)
    i = _patterns(case, case["rows"], case["cols"], 1, g)[0]
    psi0 = _random_phase(i, g)
    if case["kind"] == "ccd":   # a detector's frame: counts of a 16-bit sensor, its full well at 1/exposure
        i = torch.clamp(i, max=65535.0) / 65535.0 / 2e-4
        psi0 = _random_phase(i, g)
    return i, psi0.contiguous()


def _batch_inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "group":
        return [_patterns(case, n, n, b, g) for n, b in _sizes(case)]
    return [_patterns(case, case["rows"], case["cols"], case["batch"], g)]


def _net_inputs(case, seed):
    """Weights as He-normal draws (GroupNorm and bias near 1 and 0), patterns and targets."""
    g, n, b = _gen(seed), case["n"], case["batch"]
    parts = []
    for d in _net_layers(n, case["levels"], case["base"]):
        fan = d["cin"] if d["kind"] == "convt" else d["k"] ** 2 * d["cin"]
        parts.append(torch.randn(math.prod(d["shape"]), device="cuda", generator=g) *
                     math.sqrt((1.0 if d["kind"] == "head" else 2.0) / fan))
        if d["kind"] == "head":
            parts.append(0.1 * torch.randn(4, device="cuda", generator=g))
        else:
            parts.append(1 + 0.1 * torch.randn(d["cout"], device="cuda", generator=g))
            parts.append(0.1 * torch.randn(d["cout"], device="cuda", generator=g))
    amp = _blobs(n, n, b, g)
    i = torch.fft.fft2(amp).abs() ** 2
    i = torch.poisson(i * (1e6 / i.sum((1, 2), keepdim=True)), generator=g)
    y, x = _grid(n, n)
    ph = (0.5 * torch.cos(y / 9 + x / 13) * (amp > 1e-3)).contiguous()
    return torch.cat(parts).float(), i, amp.contiguous(), ph, (amp > 1e-3).float()


def _pty_inputs(case, seed):
    """Scan, probe, patterns of a smooth object and a random-phase start object."""
    g, r, ro = _gen(seed), case["probe"], case["obj"]
    sx, sy = pty.scan_triangle(ro, ro, r, r, case["step"])
    y, x = _grid(r, r)
    pd = 0.65 * r
    res = OPTICS["lam"] * OPTICS["d"] / OPTICS["pixelsize"] / r
    probe = _spectrum64((y * y + x * x <= pd * pd / 4).to(torch.complex128), OPTICS["dpupil"], res).to(torch.complex64)
    truth = torch.polar(0.5 + 0.5 * _smooth(ro, ro, 6.0, g), math.pi * _smooth(ro, ro, 6.0, g))
    pats = []
    for px, py in zip(sx, sy):
        w, at, to = _window(truth, px, py, r)
        f = torch.fft.fft2(probe * w)
        pats.append((f.real ** 2 + f.imag ** 2) / (r * r))
    start = torch.polar(torch.ones(ro, ro, device="cuda"), 2 * math.pi * torch.rand(ro, ro, device="cuda", generator=g))
    order = torch.rand(case["sweeps"], len(sx), device="cuda", generator=g).argsort(1).int().cpu().numpy()
    return sx, sy, pd, probe, torch.stack(pats), start, order


# --------------------------------------------------------------------- prepare and run
def _pinned(t):
    return t.cpu().pin_memory()


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    if kind in ("job", "ccd"):
        s["i"], s["psi0"] = _job_inputs(case, seed)
        shape = tuple(s["i"].shape)
        s["ctx"] = cdx.Context(_params(case, *shape))
        if kind == "ccd":
            s["bs"] = _beamstop(*shape)
        s["rho"] = torch.empty(shape, dtype=torch.complex64, device="cuda")
        s["spt"] = torch.empty(shape, device="cuda")
    elif kind == "host":
        i, psi0 = _job_inputs(case, seed)
        s["keep"] = [_pinned(i), _pinned(psi0), _pinned(psi0), _pinned(psi0), _pinned(i)]
        s["i"], s["psi0"], *s["out"] = [t.numpy() for t in s["keep"]]
        s["params"] = _params(case, *i.shape)
    elif kind in ("starts", "group"):
        s["seed"], s["ctx"], s["rho"] = int(seed) % 100003, [], []
        for i in _batch_inputs(case, seed):
            b, r, c = (case["batch"], case["rows"], case["cols"]) if kind == "starts" else i.shape
            ctx = cdx.Context(_params(case, r, c, b))
            for k in range(b):
                ctx.set_pattern(k, i[k])
            s["ctx"].append(ctx)
            s["rho"].append(torch.empty((b, r, c), dtype=torch.complex64, device="cuda"))
        if kind == "group":
            s["group"] = cdx.Group(s["ctx"])
    elif kind == "fft":
        s["x"] = torch.randn(case["batch"], case["rows"], case["cols"], dtype=torch.complex64, device="cuda",
                             generator=_gen(seed))
        s["f"], s["b"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    elif kind in ("infer", "train"):
        p, *s["data"] = _net_inputs(case, seed)
        s["net"] = unet.UNet(n=case["n"], levels=case["levels"], base=case["base"], batch=case["batch"])
        s["net"].set_params(p.cpu().numpy())
    else:
        sx, sy, pd, probe, pats, start, s["order"] = _pty_inputs(case, seed)
        t = pty.Ptycho(case["probe"], case["probe"], case["obj"], case["obj"], sx, sy, pupil_size=pd,
                       zernike_iter=case["zernike"], **OPTICS)
        t.probe, t.patterns, t.objectWave = probe.cpu().numpy(), pats.cpu().numpy(), start.cpu().numpy()
        s["t"] = t
    torch.cuda.synchronize()   # the library's contexts run on streams of their own
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("job", "ccd"):
        ctx = s["ctx"]
        ctx.set_pattern(0, s["i"])
        if kind == "ccd":
            ctx.set_beamstop(0, s["bs"])
        ctx.set_initial(0, s["psi0"])
        stats = ctx.run(case["algo"])
        return dict(rho=ctx.get_object(0, s["rho"]), spt=ctx.get_support(0, s["spt"]), rfactor=stats["rfactor"])
    if kind == "host":
        rho, psi, spt, _ = cdx.phase_retrieve_host(s["params"], case["algo"], s["i"], s["psi0"], out=s["out"])
        return dict(rho=rho, psi=psi, spt=spt)
    if kind in ("starts", "group"):
        for ctx in s["ctx"]:
            ctx.random_start(s["seed"])
        if kind == "group":
            s["group"].run(case["algo"])
        else:
            s["ctx"][0].run(case["algo"])
        for ctx, rho in zip(s["ctx"], s["rho"]):
            for k in range(rho.shape[0]):
                ctx.get_object(k, rho[k])
        return s["rho"]
    if kind == "fft":
        st = torch.cuda.current_stream().cuda_stream
        cdx.fft2(s["x"], s["f"], stream=st)
        cdx.fft2(s["f"], s["b"], inverse=True, stream=st)
        return [s["f"], s["b"]]
    if kind == "infer":
        out = s["net"].forward(s["data"][0])
        psi0, spt = s["net"].warm_start(s["data"][0], out)
        return dict(out=out, psi0=psi0, spt=spt)
    if kind == "train":
        loss = s["net"].train_step(*s["data"], lr=1e-3)
        return dict(loss=loss, grads=s["net"].grads())
    t = s["t"]
    t.iterate(case["sweeps"], first_iter=case["first"], orders=s["order"])
    return dict(object=t.objectWave, probe=t.probe)


# --------------------------------------------------------------------- what a pass cannot do without
def _steps(algo):
    """The algorithm string as (count, name) pairs (the cases use no groups)."""
    return [(int(n), a) for n, a in (t.split("*") for t in algo.split("+"))]


def work(case):
    kind = case["kind"]
    if kind in ("infer", "train"):
        # activations: each layer's output written once and read once by the next (BF16), the
        # backward the same again for the gradients with the activations read once more
        b, fl, act = case["batch"], 0, 0
        for d in _net_layers(case["n"], case["levels"], case["base"]):
            px = d["h"] ** 2 if d["kind"] == "convt" else d["oh"] ** 2
            fl += 2 * b * px * d["cin"] * d["cout"] * d["k"] ** 2
            act += b * d["oh"] ** 2 * d["cout"]
        npx = b * case["n"] ** 2
        return dict(bytes=act * (4 if kind == "infer" else 10) + npx * (32 if kind == "infer" else 16),
                    flops=fl * (1 if kind == "infer" else 3))
    if kind == "ptycho":
        # per position 28 bytes a pixel: pattern, probe and window read, the window written
        n = case["sweeps"] * 8 * case["probe"] ** 2
        return dict(bytes=28 * n + 16 * case["obj"] ** 2 * case["sweeps"], flops=n * 10 * math.log2(case["probe"] ** 2))
    if kind == "fft":
        n = case["batch"] * case["rows"] * case["cols"]
        return dict(bytes=2 * 16 * n, flops=2 * 5 * n * math.log2(case["rows"] * case["cols"]))
    if kind == "group":
        shapes = [(n, n, b) for n, b in _sizes(case)]
    else:
        shapes = [(case["rows"], case["cols"], case.get("batch", 1))]
    its = sum(n for n, a in _steps(case["algo"]) if a != "shrinkWrap")
    by = fl = 0
    for r, c, b in shapes:
        # an iteration: rho read and written, I and the support read; a pass: Psi0 or the start in, rho out
        by += r * c * b * (21 * its + 24)
        fl += its * r * c * b * 10 * math.log2(r * c)
    return dict(bytes=by, flops=fl)


# --------------------------------------------------------------------- 64-bit results
def _algo_update(name, inside, x, p):
    b = float(np.float32(BETA))
    relax = x + 1.9 * (p - x)
    if name == "HIO":
        return torch.where(inside, p, x - b * p)
    if name == "RAAR":
        return torch.where(inside, p, b * x + (1 - 2 * b) * p)
    if name == "ER":
        return torch.where(inside, relax, 0)
    if name == "POSHIO":
        re = torch.where(inside & (p.real > 0), relax.real, x.real - b * p.real)
        return torch.complex(re, x.imag - b * p.imag)
    return torch.where(inside, relax, x - 1.2 * p)   # FHIO


def _project(case, psi, i, bs):
    if case["kind"] != "ccd":
        m = psi.abs()
        return torch.where(m == 0, i.sqrt() + 0j, psi * (i.sqrt() / torch.where(m == 0, 1.0, m)))
    scale, src = float(np.float32(1) / np.float32(2e-4)), psi.real ** 2 + psi.imag ** 2
    m2 = torch.where(i >= scale * float(np.float32(0.95)), torch.maximum(i, src), i)
    tol = torch.sqrt(4 + m2 * 65535.0 / scale) * scale / 65535.0
    val = torch.where(m2 - src > tol, m2 - tol, torch.where(m2 - src < -tol, m2 + tol, m2))
    out = torch.where(src == 0, val + 0j, psi * torch.sqrt(val.clamp(min=0) / torch.where(src == 0, 1.0, src)))
    return torch.where(bs > 0.5, psi, out)


def _retrieve64(case, i, psi, bs=None):
    """The iteration on [batch, rows, cols] patterns: (rho, Psi, support, R-factor)."""
    i, psi = i.double(), psi.to(torch.complex128)
    r, c = i.shape[-2:]
    n = r * c
    rho = torch.fft.ifft2(psi)
    o = 4.0
    sx, sy = int((o - 1) / 2 * r / o - 1), int((o - 1) / 2 * c / o - 1)
    spt = torch.zeros_like(i)
    spt[:, sx:r - sx, sy:c - sy] = 1
    thr, avg, sig = torch.full((i.shape[0], 1, 1), 0.5, device="cuda", dtype=torch.float64), None, np.float32(3)
    fy, fx = (torch.fft.fftfreq(m, 1.0 / m, device="cuda", dtype=torch.float64) for m in (r, c))
    for count, name in _steps(case["algo"]):
        for _ in range(count):
            if name == "shrinkWrap":
                sf = float(np.float32(r >> 2) / sig)
                f = torch.exp(-(fy[:, None] ** 2 + fx[None, :] ** 2) / (2 * sf * sf))
                spt = (torch.fft.ifft2(psi * f) * n).abs() ** 2
                top = spt.amax((1, 2), keepdim=True)
                avg = spt.sum((1, 2), keepdim=True) * 4 / n if avg is None else avg
                thr = torch.minimum(top, 5 * avg) * float(np.float32(SHRINK))
                sig = np.float32(float(sig) * float(np.float32(0.99))) if sig > 2 else sig
                continue
            p = torch.fft.ifft2(_project(case, psi, i, bs))
            rho = _algo_update(name, spt > thr, rho, p)
            psi = torch.fft.fft2(rho)
    a = i.sqrt()
    return rho * math.sqrt(n), psi, spt, (psi.abs() - a).abs().sum((1, 2)) / a.sum((1, 2))


def _coin(seed, count):
    """The library's documented start coin: SplitMix64 of (seed, pixel), true for a phase of pi."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15) + np.arange(1, count + 1, dtype=np.uint64)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    return torch.from_numpy(((z >> np.uint64(40)) + np.uint64(1)) > np.uint64(1 << 23)).cuda()


def _net_layers(n, levels, base):
    """The network's layers in parameter order: 3x3 blocks, stride-2 down, 2x2 transposed up, 1x1 head."""
    out = []

    def add(kind, ins, cin, cout, k, s, h):
        out.append(dict(kind=kind, ins=ins, cin=cin, cout=cout, k=k, s=s, h=h, oh=2 * h if kind == "convt" else h // s,
                        shape=(cin, k, k, cout) if kind == "convt" else (cout, k, k, cin)))
        return len(out) - 1

    add("conv", [-1], 1, base, 3, 1, n)
    cur, h, ch = add("conv", [0], base, base, 3, 1, n), n, base
    skip = [cur]
    for _ in range(1, levels):
        cur = add("conv", [cur], ch, 2 * ch, 3, 2, h)
        h, ch = h // 2, 2 * ch
        cur = add("conv", [cur], ch, ch, 3, 1, h)
        skip.append(cur)
    for l in range(levels - 2, -1, -1):
        up = add("convt", [cur], ch, ch // 2, 2, 2, h)
        h, ch = 2 * h, ch // 2
        cur = add("conv", [up, skip[l]], 2 * ch, ch, 3, 1, h)
    add("head", [cur], ch, 4, 1, 1, h)
    return out


def _net64(case, p, i):
    """Head output [batch, 4, n, n] of the network in 64 bits (differentiable in p)."""
    x = torch.log1p(i.double())
    x = torch.fft.fftshift(x / x.amax((1, 2), keepdim=True), dim=(1, 2))[:, None]
    acts, at = [], 0

    def take(count):
        nonlocal at
        at += count
        return p[at - count:at]

    for d in _net_layers(case["n"], case["levels"], case["base"]):
        w = take(math.prod(d["shape"])).reshape(d["shape"]).permute(0, 3, 1, 2)
        v = torch.cat([x if k < 0 else acts[k] for k in d["ins"]], 1)
        if d["kind"] == "convt":
            v = torch.nn.functional.conv_transpose2d(v, w, stride=2)
        else:
            v = torch.nn.functional.conv2d(v, w, stride=d["s"], padding=d["k"] // 2)
        if d["kind"] == "head":
            return v + take(4)[:, None, None]
        v = torch.nn.functional.group_norm(v, 8, take(d["cout"]), take(d["cout"]))
        acts.append(torch.nn.functional.leaky_relu(v, 0.01))


def _net_loss64(out, amp, ph, sup):
    """Per-pixel loss of the nearer of the object and its twin, averaged over the patterns given."""
    def one(a, q, t):
        e = (out[:, 0] - a) ** 2 + a * ((out[:, 1] - q.cos()) ** 2 + (out[:, 2] - q.sin()) ** 2)
        e = e + 0.1 * torch.nn.functional.binary_cross_entropy_with_logits(out[:, 3], t, reduction="none")
        return e.mean((1, 2))

    def twin(v):
        return torch.roll(v.flip((1, 2)), (1, 1), (1, 2))

    return torch.minimum(one(amp, ph, sup), one(twin(amp), -twin(ph), twin(sup)))


def _window(o, px, py, r):
    """The r x r window of o at the rounded position, zero outside; and its slices in o and in the window."""
    x, y = (int(math.floor(abs(float(v)) + 0.5)) * (1 if v >= 0 else -1) for v in (px, py))
    at = (slice(max(0, x), min(o.shape[0], x + r)), slice(max(0, y), min(o.shape[1], y + r)))
    to = tuple(slice(a.start - b, a.stop - b) for a, b in zip(at, (x, y)))
    w = torch.zeros(r, r, dtype=o.dtype, device="cuda")
    w[to] = o[at]
    return w, at, to


def _spectrum64(f, distance, res):
    """Angular-spectrum propagation of a centred field (negative distances back)."""
    y, x = (v.double() for v in _grid(*f.shape))
    q = 1 - (y * y + x * x) * (OPTICS["lam"] / (res * f.shape[0])) ** 2
    ph = 2 * math.pi * distance / OPTICS["lam"] * q.clamp(min=0).sqrt()
    return torch.fft.ifft2(torch.fft.fft2(f) * torch.fft.ifftshift(torch.polar((q >= 0).double(), ph)))


def _tv64(o):
    """One TV proximal step of the complex object (its two components separately), lambda 0.01."""
    def part(b):
        v = b * 12.5
        p, q = v.clone(), v.clone()
        p[:-1] -= v[1:]
        q[:, :-1] -= v[:, 1:]
        m = torch.hypot(p, q).clamp(min=1)
        p, q = p / m, q / m
        l = p + q
        l[1:] -= p[:-1]
        l[:, 1:] -= q[:, :-1]
        return b - 0.01 * l
    return torch.complex(part(o.real), part(o.imag))


def _ptycho64(case, seed):
    sx, sy, pd, probe, pats, o, order = _pty_inputs(case, seed)
    r, n = case["probe"], len(sx)
    pats, o, probe = pats.double(), o.to(torch.complex128), probe.to(torch.complex128)
    prev, pprev, y, x = torch.zeros_like(o), torch.zeros_like(probe), *_grid(r, r)
    disk, cover = (y * y + x * x).sqrt() < pd / 2, torch.zeros(o.shape, device="cuda")
    for px, py in zip(sx, sy):
        _, at, to = _window(cover, int(px), int(py), r)
        cover[at] += disk[to]
    cover = cover > 0.5
    full, tk = 0.95 * float(np.float32(1) / np.float32(OPTICS["exposure"])), 0.5 + math.sqrt(1.25)
    res, d = OPTICS["lam"] * OPTICS["d"] / OPTICS["pixelsize"] / r, int(pd)
    cut = torch.arange(d, device="cuda") - (d + 1) // 2
    pupil = torch.zeros(r, r, dtype=torch.bool, device="cuda")
    at0 = (r - d) // 2
    pupil[at0:at0 + d, at0:at0 + d] = (cut[:, None] ** 2 + cut[None, :] ** 2).double().sqrt() < d / 2
    for it in range(case["sweeps"]):
        late = case["first"] + it >= 400
        pmax = (probe.abs() ** 2).max()
        if late:
            omax = (o.abs() ** 2 * cover).max()
            top, m2 = omax.sqrt(), o.abs() ** 2
            o = torch.where(m2 > top, o * (top / m2.clamp(min=1e-300)).sqrt(), o)
            f = (pmax / omax) ** 0.25
            o, prev, probe, pprev = o * f, prev * f, probe / f, pprev / f
            omax = pmax = (omax * pmax).sqrt()
            step = torch.zeros_like(probe)
        den = (1 if not late else 0.5) / (0.9 * probe.abs() ** 2 + 0.1 * pmax.clamp(min=1e-5))
        for k in order[it]:
            w, at, to = _window(o, sx[k], sy[k], r)
            e = probe * w
            f = torch.fft.fft2(e) / r
            src, m2 = f.abs() ** 2, pats[k]
            g = torch.where((m2 >= full) & (src >= m2), 1.0, (m2 / torch.where(src == 0, 1.0, src)).sqrt())
            diff = e - torch.fft.ifft2(f * g) * r
            w = w - probe.conj() * diff * den
            if late:
                step -= w.conj() * diff / (0.5 * w.abs() ** 2 + 0.5 * omax.clamp(min=1e-5)) / n
            o[at] = w[to]
        if late:
            probe = torch.where(pupil, _spectrum64(probe + step, -OPTICS["dpupil"], res), 0)
            probe = _spectrum64(probe, OPTICS["dpupil"], res)
            far = torch.fft.fftshift(torch.fft.fft2(probe)).abs() ** 2
            u = (torch.arange(r, device="cuda", dtype=torch.float64) + 0.5) / r - 0.5
            mx, my = (far.sum(1) * u).sum() / far.sum(), (far.sum(0) * u).sum() / far.sum()
            probe = probe * torch.exp(-2j * math.pi * ((mx * r - 0.5) * y.double() + (my * r - 0.5) * x.double()) / r)
        if case["first"] + it < case["zernike"]:
            o = _tv64(o)
        s = (o * cover).sum()
        s = (s / s.abs()).conj()
        tn = 0.5 + math.sqrt(0.25 + tk * tk)
        o, prev = o * s, prev * s
        o, prev = o + (o - prev) * ((tk - 1) / tn), o
        if case["first"] + it < case["zernike"] and (case["first"] + it) % 10 == 0:   # the probe's own momentum
            probe, pprev = probe + (probe - pprev) * (0.8 * (tk - 1) / tn), probe
        tk = tn
    s = o.sum()
    o = o * (s / s.abs()).conj()
    return dict(object=o, probe=probe)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("job", "ccd", "host"):
        i, psi0 = _job_inputs(case, seed)
        bs = _beamstop(*i.shape) if kind == "ccd" else None
        rho, psi, spt, rf = _retrieve64(case, i[None], psi0[None], bs)
        if kind == "host":
            return dict(rho=rho[0].cpu().numpy(), psi=psi[0].cpu().numpy(), spt=spt[0].cpu().numpy())
        return dict(rho=rho[0], spt=spt[0], rfactor=float(rf[0]))
    if kind in ("starts", "group"):
        out = []
        for i in _batch_inputs(case, seed):
            r, c = i.shape[-2:]
            b = case.get("batch", i.shape[0])
            i = i.expand(b, r, c)
            psi0 = torch.where(_coin(int(seed) % 100003, i.numel()).reshape(i.shape), -1.0, 1.0) * i.double().sqrt() + 0j
            out.append(_retrieve64(case, i, psi0)[0])
        return out
    if kind == "fft":
        x = torch.randn(case["batch"], case["rows"], case["cols"], dtype=torch.complex64, device="cuda",
                        generator=_gen(seed)).to(torch.complex128)
        return [torch.fft.fft2(x), x * (case["rows"] * case["cols"])]
    if kind in ("infer", "train"):
        p, i, *targets = _net_inputs(case, seed)
        p = p.double().requires_grad_(kind == "train")
        if kind == "infer":   # the start's phases hang on a thresholded mask: no 64-bit value
            return dict(out=torch.cat([_net64(case, p, v) for v in i.split(4)]), psi0=None, spt=None)
        loss = 0.0
        for k in range(0, case["batch"], 4):
            e = _net_loss64(_net64(case, p, i[k:k + 4]), *(t[k:k + 4].double() for t in targets)).sum() / case["batch"]
            e.backward()
            loss += float(e)
        return dict(loss=loss, grads=p.grad.cpu().numpy())
    out = _ptycho64(case, seed)
    return {k: v.cpu().numpy() for k, v in out.items()}
