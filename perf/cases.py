"""The calls that the speed of this framework is judged by.

A case is one call as a user's program makes it, through the public entry points: a batch of
raw SIM stacks reconstructed by fused plans (device-resident, as one CUDA graph, or from
pinned host buffers), the live path of one camera or several, the parameter fit, the 2D FFT.
`listed()` names fixed ones, `draw()` gives others of the same ranges; `prepare` makes the
seeded inputs and what a program keeps (plans, graphs, buffers), `run` is one call, `work`
its unavoidable bytes and operations, and `exact` the same result in 64 bits from plain
torch, written from the algorithm's definition (Wiener-filtered 2D SIM with fairSIM's
conventions) without the package's code.
"""
import ctypes
import importlib
import math
import random

import numpy as np
import torch

fs = importlib.import_module("fairsim-vigor_gb300")
plan = importlib.import_module("fairsim-vigor_gb300.plan")
N = importlib.import_module("fairsim-vigor_gb300.native")

EMISSIONS = [488.0, 525.0, 600.0]  # nm, the three channels of the mixed and live workloads
BASE = dict(dirs=3, phases=3, bands=2, dtype="f32", na=1.4, emission=525.0, pixel=0.08, k0=0.85, modulation=0.8,
            photons=500.0)


def _case(name, kind, **kw):
    c = dict(BASE)
    c.update(kind=kind, name=name)
    c.update(kw)
    return c


def listed():
    return [
        # one small camera frame set, reconstructed as it arrives: launches and latency count
        _case("offline-256-single", "offline", n=256, batch=1, dtype="u16", plans=1, graph=False, clip=0,
              attenuation=False, widefield=False),
        # a time series of 512^2 stacks reconstructed at once, the benchmark's headline workload
        _case("offline-512-batch64", "offline", n=512, batch=64, plans=16, graph=True, clip=0, attenuation=False,
              widefield=False),
        # 15-frame stacks of a three-band (three-beam) microscope with a 384^2 region of interest
        _case("offline-384-3band", "offline", n=384, batch=7, dtype="u16", phases=5, bands=3, k0=0.45, plans=1,
              graph=False, clip=0, attenuation=False, widefield=False),
        # the display form: OTF attenuation on, negative values clipped, a ragged 3*2^k size
        _case("offline-768-clip", "offline", n=768, batch=4, plans=2, graph=False, clip=1, attenuation=True,
              widefield=False),
        # one large precision-checked stack, 3 angles x 5 phases, the largest image
        _case("offline-2048-3x5", "offline", n=2048, batch=1, phases=5, k0=0.9, modulation=0.6, photons=200.0, plans=1,
              graph=False, clip=0, attenuation=False, widefield=False),
        # reconstruction beside the widefield and the filtered widefield of the same stacks
        _case("widefield-512", "offline", n=512, batch=16, plans=4, graph=False, clip=0, attenuation=False,
              widefield=True),
        # 32 datasets of five sizes and one to three channels each, recorded once and replayed
        _case("mixed-32", "mixed", datasets=32, mix=77),
        # one live stack of one channel with its widefield: the latency of the served form
        _case("live-512-single", "live", n=512, batch=1, dtype="u16", graph=False),
        # live throughput of three channels
        _case("live-512-batch64", "live", n=512, batch=64, dtype="u16", graph=True),
        # the full parameter fit (coarse search, sub-pixel search, phase and modulation)
        _case("fit-1024", "fit", n=1024),
        # spectra of a set of frames with the library's 2D FFT
        _case("fft2d-1024", "fft2d", w=1024, h=1024, batch=16, inverse=False),
        # stacks in pinned host memory to images in pinned host memory, copies overlapped
        _case("host-512-batch24", "host", n=512, batch=24, plans=4),
    ]


_BUDGET = 64 * 512 * 512 * 9  # raw pixels of the largest drawn batch


def draw(rng):
    kind = rng.choice(["offline", "offline", "offline", "mixed", "live", "live", "fit", "fft2d", "host"])
    c = dict(BASE)
    c.update(kind=kind, dtype=rng.choice(["f32", "u16"]), na=rng.choice([1.2, 1.4, 1.49]),
             emission=rng.choice(EMISSIONS), pixel=round(math.exp(rng.uniform(math.log(0.062), math.log(0.1))), 4),
             k0=round(rng.uniform(0.7, 0.9), 3), modulation=round(rng.uniform(0.5, 0.9), 3),
             photons=round(math.exp(rng.uniform(math.log(100), math.log(2000)))))
    # up to a cutoff just beyond the camera's Nyquist frequency
    c["pixel"] = min(c["pixel"], round(0.52 * c["emission"] / (2000.0 * c["na"]), 4))
    if kind == "mixed":
        c.update(datasets=rng.randrange(3, 25), mix=rng.randrange(1, 10 ** 6), dtype="f32", na=1.4, pixel=0.08, k0=0.85)
        return c
    if kind == "fft2d":
        lens = [64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048]
        c.update(w=rng.choice(lens), h=rng.choice(lens), inverse=rng.random() < 0.5)
        top = max(1, min(64, (1 << 24) // (c["w"] * c["h"])))
        c["batch"] = round(math.exp(rng.uniform(0, math.log(top))))
        return c
    if kind == "fit":
        c.update(n=rng.choice([384, 512, 768, 1024]), k0=round(rng.uniform(0.8, 0.9), 3), photons=500.0)
        if rng.random() < 0.3:
            c.update(bands=3, phases=5, k0=round(c["k0"] / 2, 3))
        return c
    c["phases"], c["bands"] = rng.choice([(3, 2), (3, 2), (5, 2), (5, 3)])
    if c["bands"] == 3:
        c["k0"] = round(c["k0"] / 2, 3)
    c["dirs"] = rng.choice([3, 3, 3, 2, 5])
    sizes = [64, 128, 256, 384, 512, 768, 1024] + ([192, 2048] if kind == "offline" else [])
    c["n"] = rng.choice(sizes)
    top = max(1, min(64 if kind != "host" else 24, _BUDGET // (c["n"] ** 2 * c["dirs"] * c["phases"])))
    c["batch"] = round(math.exp(rng.uniform(0, math.log(top))))
    c["graph"] = rng.random() < 0.4
    if kind == "live":
        c["dtype"] = "u16"
    else:
        c.update(plans=rng.randrange(1, 5))
    if kind == "offline":
        c.update(clip=rng.choice([0, 0, 1]), attenuation=rng.random() < 0.3, widefield=rng.random() < 0.25)
    return c


# ---- inputs ---------------------------------------------------------------------------------

def _geometry(case, rng, n, emission):
    """Seeded pattern vectors and phases of one parameter set, in SimParam's convention."""
    cut = 2000.0 * case["na"] / emission
    k0 = case["k0"] * cut * n * case["pixel"]
    hb = case["bands"] - 1
    g = dict(n=n, emission=emission, cutoff=cut, dirs=[])
    for d in range(case["dirs"]):
        th = math.radians(180.0 * d / case["dirs"] + rng.uniform(0, 5.0))
        kx, ky = k0 * math.cos(th), k0 * math.sin(th)
        g["dirs"].append(dict(kx=kx, ky=ky, px=hb * kx, py=-hb * ky, phase=rng.uniform(0, 2 * math.pi)))
    return g


def _sim_param(case, g, known=True):
    otf = fs.OtfProvider.fromEstimate(case["na"], g["emission"], 1.0)
    if case.get("attenuation"):
        otf.switchAttenuation(True)
    sp = fs.SimParam.create(case["bands"], case["dirs"], case["phases"], g["n"], case["pixel"], otf)
    if known:
        for d, v in enumerate(g["dirs"]):
            sp.dir(d).setPxPy(v["px"], v["py"])
            sp.dir(d).setPhaOff(v["phase"])
            for b in range(1, case["bands"]):
                sp.dir(d).setModulation(b, case["modulation"])
    return sp


def _stack(case, g, gen):
    """One raw stack on the GPU: point emitters and random-walk filaments under the pattern,
    blurred by the widefield OTF, with photon and read-out noise."""
    n, dev = g["n"], "cuda"
    area = (n / 512.0) ** 2
    rand = lambda *s: torch.rand(*s, device=dev, generator=gen)  # noqa: E731
    obj = torch.zeros(n * n, dtype=torch.int64, device=dev)  # sums of integers: the same in any order
    units = lambda v: (v * 2.0 ** 20).round_().long()  # noqa: E731
    npt, nfil, steps = max(8, round(2000 * area)), max(2, round(40 * area)), max(64, n // 2)
    at = (rand(npt) * n).long().clamp_(max=n - 1) * n + (rand(npt) * n).long().clamp_(max=n - 1)
    obj.index_add_(0, at, units(torch.exp(0.5 * torch.randn(npt, device=dev, generator=gen))))
    ang = 2 * math.pi * rand(nfil, 1) + torch.cumsum(0.15 * torch.randn(nfil, steps, device=dev, generator=gen), 1)
    fx = torch.remainder(rand(nfil, 1) * n + torch.cumsum(torch.cos(ang), 1), n).long().clamp_(max=n - 1)
    fy = torch.remainder(rand(nfil, 1) * n + torch.cumsum(torch.sin(ang), 1), n).long().clamp_(max=n - 1)
    amp = torch.exp(-1.0 + 0.3 * torch.randn(nfil, 1, device=dev, generator=gen)).expand(nfil, steps)
    obj.index_add_(0, (fy * n + fx).reshape(-1), units(amp).reshape(-1))
    obj = (obj.double() * 2.0 ** -20).float().reshape(n, n)
    f = torch.fft.fftfreq(n, 1.0 / n, device=dev)
    d = (torch.hypot(f[None, :], f[:, None]) / (g["cutoff"] * n * case["pixel"])).clamp_(max=1.0)
    otf = (2 / math.pi) * (torch.acos(d) - d * torch.sqrt(1 - d * d))
    x = torch.arange(n, device=dev, dtype=torch.float64)
    frames = torch.empty(case["dirs"], case["phases"], n, n, device=dev)
    for a, v in enumerate(g["dirs"]):
        ph = (2 * math.pi / n) * (v["kx"] * x[None, :] + v["ky"] * x[:, None])
        for p in range(case["phases"]):
            t = ph + (2 * math.pi * p / case["phases"] + v["phase"])
            pat = 1.0 + case["modulation"] * torch.cos(t)
            for b in range(2, case["bands"]):
                pat += 0.5 * case["modulation"] * torch.cos(b * t)
            frames[a, p] = torch.fft.ifft2(torch.fft.fft2(obj * pat.float()) * otf).real
    frames = frames.clamp_(min=0)
    frames *= case["photons"] / frames.max()
    frames = torch.poisson(frames, generator=gen) + 2.0 * torch.randn(frames.shape, device=dev, generator=gen)
    frames = frames.reshape(-1, n, n)
    if case["dtype"] == "u16":
        return frames.round_().clamp_(0, 65535).to(torch.int32).to(torch.int16)  # the camera's 16 bits
    return frames


def _mix(case):
    """(size, channel) of every stack of a mixed batch."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["datasets"]):
        n, nch = rng.choice([256, 384, 512, 768, 1024]), rng.randrange(1, 4)
        out += [(n, ch) for ch in range(nch)]
    return out


def _sets(case, seed):
    """Parameter sets and, per stack, (parameter set, generator)."""
    rng = random.Random("%d geometry" % seed)
    if case["kind"] == "mixed":
        geo = [_geometry(case, rng, n, EMISSIONS[ch]) for n, ch in _mix(case)]
        idx = list(range(len(geo)))
    else:
        if case["kind"] == "live":
            lam = [case["emission"]] if case["batch"] == 1 else EMISSIONS
        else:
            lam = [case["emission"]] * min(case.get("plans", 1), case.get("batch", 1))
        geo = [_geometry(case, rng, case["n"], e) for e in lam]
        idx = [i % len(geo) for i in range(case.get("batch", 1))]
    return geo, idx


def _groups(sizes):
    """Per image size, ascending: the stacks of that size."""
    return [(n, [j for j, m in enumerate(sizes) if m == n]) for n in sorted(set(sizes))]


def _raw(case, seed):
    geo, idx = _sets(case, seed)
    out = []
    for j, i in enumerate(idx):
        gen = torch.Generator(device="cuda").manual_seed(1000003 * seed + j)
        out.append(_stack(case, geo[i], gen))
    return geo, idx, out


def _fft_input(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((case["batch"], case["h"], case["w"]), dtype=torch.complex64, device="cuda", generator=gen)


def prepare(case, seed):
    kind = case["kind"]
    N.init(torch.cuda.current_device())
    st = dict(case=case, stream=torch.cuda.Stream())
    if kind == "fft2d":
        st["x"] = _fft_input(case, seed)
        st["y"] = torch.empty_like(st["x"])
        torch.cuda.synchronize()
        return st
    geo, idx, raw = _raw(case, seed)
    st["raw"] = raw
    if kind == "fit":
        st["param"] = _sim_param(case, geo[0], known=False)
        torch.cuda.synchronize()
        return st
    path = N.PATH_LIVE if kind == "live" else N.PATH_OFFLINE
    itype = N.INPUT_U16 if case["dtype"] == "u16" else N.INPUT_F32
    st["plans"] = [plan.ReconPlan(_sim_param(case, g), path=path, input_type=itype, fade_px=10) for g in geo]
    if case.get("clip"):
        for p in st["plans"]:
            p.setClipScale(case["clip"])
    pl = [st["plans"][i] for i in idx]
    if kind == "host":
        n = case["n"]
        h = torch.empty((len(raw),) + tuple(raw[0].shape), dtype=raw[0].dtype).pin_memory()
        for i, r in enumerate(raw):
            h[i].copy_(r)
        st["raw"], st["out"] = h, torch.empty((len(raw), 2 * n, 2 * n)).pin_memory()
        st["jobs"] = [(p, h[i].data_ptr(), st["out"][i].data_ptr()) for i, p in enumerate(pl)]
        torch.cuda.synchronize()
        return st
    # per image size one array of every kind of image the call gives
    scale = [2] + ([1] if kind == "live" else [2, 2] if case.get("widefield") else [])
    groups = _groups([p.w for p in pl])
    st["out"] = [[torch.empty((len(g), f * w, f * w), device="cuda") for f in scale] for w, g in groups]
    at = {j: [o[k].data_ptr() for o in os] for (_, g), os in zip(groups, st["out"]) for k, j in enumerate(g)}
    st["jobs"] = [(p, r.data_ptr(), *at[j]) for j, (p, r) in enumerate(zip(pl, raw))]
    st["ws"] = torch.empty(plan.batch_workspace_bytes(pl), dtype=torch.uint8, device="cuda")
    if kind == "mixed" or case.get("graph"):
        st["graph"] = plan.BatchGraph(st["jobs"], st["ws"].data_ptr(), st["ws"].numel(), st["stream"].cuda_stream)
    torch.cuda.synchronize()
    return st


def run(st):
    case, s = st["case"], st["stream"]
    kind = case["kind"]
    if kind == "host":
        plan.recon_batch_host(st["jobs"])
        return st["out"]
    if kind == "fit":
        c = N.to_c_param(st["param"])
        peaks = np.zeros((case["dirs"], 4))
        itype = N.INPUT_U16 if case["dtype"] == "u16" else N.INPUT_F32
        N.check(N.lib().fsim_estimate_raw(ctypes.byref(c), ctypes.c_void_p(st["raw"][0].data_ptr()), itype, 10,
                                          case["bands"] - 1, ctypes.c_double(0.6), peaks.ctypes.data_as(ctypes.c_void_p)))
        p = N.from_c_param(c)
        return [peaks, np.array([p["pX"], p["pY"], p["phaOff"]]),
                np.array([m[1:] for m in p["modulations"]])]
    cur = torch.cuda.current_stream()
    s.wait_stream(cur)
    if kind == "fft2d":
        with torch.cuda.stream(s):
            st["y"].copy_(st["x"])  # the transform is in place
        N.check(N.lib().fsim_fft2d_batch(ctypes.c_void_p(st["y"].data_ptr()), case["w"], case["h"], case["batch"],
                                         int(case["inverse"]), ctypes.c_void_p(s.cuda_stream)))
        out = st["y"]
    else:
        if "graph" in st:
            st["graph"].launch(s.cuda_stream)
        else:
            plan.recon_batch(st["jobs"], st["ws"].data_ptr(), st["ws"].numel(), s.cuda_stream)
        out = st["out"]
    cur.wait_stream(s)
    return out


def _fft_flops(w, h):
    return 5.0 * w * h * math.log2(w * h)


def work(case):
    """Raw frames in and images out once; the transforms of the algorithm as it is defined: one
    complex N x N transform of band 0 and one per band pair, the pair's shift on the 2N grid
    (inverse and forward; on the N grid on the live path) and the inverse of the result."""
    kind = case["kind"]
    if kind == "fft2d":
        el = case["w"] * case["h"] * case["batch"]
        return {"bytes": 16.0 * el, "flops": case["batch"] * _fft_flops(case["w"], case["h"])}
    sizes = [n for n, _ in _mix(case)] if kind == "mixed" else [case["n"]] * case.get("batch", 1)
    pairs = case["dirs"] * (case["bands"] - 1)
    px = 2 if case["dtype"] == "u16" else 4
    b = f = 0.0
    for n in sizes:
        raw = n * n * case["dirs"] * case["phases"]
        b += raw * px
        f += 2.0 * raw * case["bands"]
        if kind == "fit":
            # spectra, coarse correlation, then per search step two inverse transforms and 100 sums
            f += (case["dirs"] * (case["phases"] + 3 + 2 * 4)) * _fft_flops(n, n) + case["dirs"] * 300 * 8.0 * n * n
            continue
        b += 16.0 * n * n
        if kind == "live":
            b += 4.0 * n * n
            f += (1 + 3 * pairs) * _fft_flops(n, n) + 0.5 * _fft_flops(2 * n, 2 * n)
        else:
            f += (1 + pairs) * _fft_flops(n, n) + (2 * pairs + 0.5) * _fft_flops(2 * n, 2 * n)
            if case.get("widefield"):
                b += 32.0 * n * n
                f += _fft_flops(2 * n, 2 * n)
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits, from the definitions --------------------------------------

class _Exact:
    """Wiener-filtered 2D SIM on one parameter set in double precision."""

    def __init__(self, case, g, dev):
        self.case, self.g, self.dev = case, g, dev
        n = g["n"]
        self.cpm = 1.0 / (n * case["pixel"])
        i = np.arange(512) / 512.0
        val = (2 / math.pi) * (np.arccos(i) - i * np.sqrt(1 - i * i))
        att = 1 - 0.99 * np.exp(-((i * g["cutoff"]) ** 2) / (2 * (1.2 / 2.355) ** 2))
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        self.val, self.att = t(val), t(att)
        fade = np.ones(n)
        e = np.sin(np.arange(10) / 10.0 * math.pi / 2) ** 2
        fade[:10] *= e
        fade[-10:] *= e[::-1]
        self.fade = t(fade)[None, :] * t(fade)[:, None]

    def freq(self, n):
        f = torch.arange(n, dtype=torch.float64, device=self.dev)
        return torch.where(f < n / 2, f, f - n)[None, :], torch.where(f < n / 2, -f, n - f)[:, None]

    def radius(self, n, kx=0.0, ky=0.0):
        x, y = self.freq(n)
        return torch.sqrt((x - kx) ** 2 + (y - ky) ** 2) * self.cpm

    def otf(self, n, kx=0.0, ky=0.0, att=False):
        r = self.radius(n, kx, ky)
        pos = r * (512.0 / self.g["cutoff"])
        i = pos.floor().clamp(max=511).long()
        v = self.val[i] * self.att[i] if att else self.val[i]
        return torch.where((r >= self.g["cutoff"]) | (pos.ceil() >= 512), torch.zeros_like(v), v)

    def wiener(self, bend, cut):
        case, w = self.case, 2 * self.g["n"]
        acc = torch.zeros(w, w, dtype=torch.float64, device=self.dev)
        for d in self.g["dirs"]:
            for b in range(case["bands"]):
                kx, ky = self.band(d, b)
                for sg in (1, -1):
                    o = self.otf(w, sg * kx, sg * ky)
                    r = self.radius(w, sg * kx, sg * ky)
                    o = o * o
                    if case.get("attenuation"):
                        o = o * self.att[(r * (512.0 / self.g["cutoff"])).floor().clamp(max=511).long()]
                    acc += o
        fr = self.radius(w) / (self.g["cutoff"] * cut)
        fc = fr.clamp(max=1.0)
        apo = (2 / math.pi) * (torch.acos(fc) - fc * torch.sqrt(1 - fc * fc))
        apo = torch.where(fr > 1, torch.zeros_like(apo), apo) ** bend
        return apo / (acc + 0.05 ** 2)

    def band(self, d, b):
        hb = self.case["bands"] - 1
        return d["px"] / hb * b, d["py"] / hb * b

    def matrix(self, offset, modulation):
        case = self.case
        ph = 2 * math.pi * np.arange(case["phases"]) / case["phases"] + offset
        cols = [np.ones(case["phases"], complex)]
        for b in range(1, case["bands"]):
            cols += [0.5 * modulation * np.exp(1j * b * ph), 0.5 * modulation * np.exp(-1j * b * ph)]
        return np.linalg.pinv(np.stack(cols, 1))

    def frames(self, raw):
        case, n = self.case, self.g["n"]
        r = raw.to(self.dev)
        r = (r.to(torch.int32) & 0xFFFF).double() if case["dtype"] == "u16" else r.double()
        return r.reshape(case["dirs"], case["phases"], n, n) * self.fade

    def separate(self, fr, a, m):
        mt = torch.tensor(m, dtype=torch.complex128, device=self.dev)
        return torch.fft.fft2(torch.einsum("cp,pyx->cyx", mt, fr[a].to(torch.complex128)))

    def paste(self, v, ox=0, oy=0):
        n = v.shape[-1]
        f = torch.arange(n, device=self.dev)
        f = torch.where(f < n // 2, f, f - n)
        out = torch.zeros(2 * n, 2 * n, dtype=v.dtype, device=self.dev)
        out[((f + oy) % (2 * n))[:, None], ((f + ox) % (2 * n))[None, :]] = v
        return out

    def ramp(self, n, kx, ky):
        x = torch.arange(n, dtype=torch.float64, device=self.dev)
        e = lambda k: torch.polar(torch.ones_like(x), 2 * math.pi * torch.remainder(k * x / n, 1.0))  # noqa: E731
        return e(kx)[None, :] * e(ky)[:, None]

    def shift(self, v, kx, ky):
        return torch.fft.fft2(torch.fft.ifft2(v) * self.ramp(v.shape[-1], kx, ky))

    def offline(self, raw):
        case, w = self.case, 2 * self.g["n"]
        fr, att = self.frames(raw), bool(case.get("attenuation"))
        total = torch.zeros(w, w, dtype=torch.complex128, device=self.dev)
        low = torch.zeros(w // 2, w // 2, dtype=torch.complex128, device=self.dev)
        for a, d in enumerate(self.g["dirs"]):
            sep = self.separate(fr, a, self.matrix(d["phase"], case["modulation"]))
            low += sep[0]
            for b in range(1, case["bands"]):
                kx, ky = self.band(d, b)
                for c, sg in ((2 * b - 1, -1), (2 * b, 1)):
                    total += self.shift(self.paste(sep[c]), sg * kx, -sg * ky) * self.otf(w, sg * kx, sg * ky, att)
        total += self.paste(low) * self.otf(w, att=att)
        img = torch.fft.ifft2(total * self.wiener(0.9, 2.0)).real
        if case.get("clip") == 1:
            img = img.clamp(min=0)
        out = [img]
        if case.get("widefield"):
            o = self.otf(w)
            low = self.paste(low)
            out += [torch.fft.ifft2(low).real, torch.fft.ifft2(low * o / (2 * o * o + 0.05 ** 2)).real]
        return out

    def live(self, raw):
        case, n = self.case, self.g["n"]
        fr, o = self.frames(raw), self.otf(n)
        total = torch.zeros(2 * n, 2 * n, dtype=torch.complex128, device=self.dev)
        for a, d in enumerate(self.g["dirs"]):
            sep = self.separate(fr, a, self.matrix(d["phase"], case["modulation"])) * o
            total += self.paste(sep[0])
            for b in range(1, case["bands"]):
                for c, sg in ((2 * b - 1, -1), (2 * b, 1)):
                    kx, ky = (sg * k for k in self.band(d, b))
                    fx, fy = math.floor(kx), math.floor(-ky)
                    total += self.paste(self.shift(sep[c], kx - fx, -ky - fy), fx, fy)
        return [torch.fft.ifft2(total * self.wiener(1.0, 2.0)).real, fr.mean((0, 1))]

    def common(self, b0, b1, kx, ky):
        """The region of both bands' overlap, divided by the OTF."""
        n = b0.shape[-1]
        x = torch.arange(n, device=self.dev)
        x = torch.where(x < n // 2, x, x - n).double()
        ratio = torch.sqrt(x[None, :] ** 2 + x[:, None] ** 2) / math.hypot(kx, ky)
        w, cut = self.otf(n), (ratio < 0.15) | (ratio > 0.85)
        z = torch.zeros_like(b0)
        b0 = torch.where((w < 0.05) | (self.otf(n, kx, ky) < 0.05) | cut, z, b0 / w)
        b1 = torch.where((w < 0.05) | (self.otf(n, -kx, -ky) < 0.05) |
                         torch.roll(cut, (int(ky), -int(kx)), (0, 1)), z, b1 / w)
        return torch.fft.ifft2(b0), torch.fft.ifft2(b1)

    def correlate(self, b0, b1, kxs, kys):
        n = b0.shape[-1]
        x = torch.arange(n, dtype=torch.float64, device=self.dev)
        e = lambda k: torch.polar(torch.ones_like(x), 2 * math.pi * torch.remainder(k * x / n, 1.0))  # noqa: E731
        tx, ty = torch.stack([e(k) for k in kxs]), torch.stack([e(-k) for k in kys])
        c = ty @ (b1 * b0.conj()) @ tx.T
        return (c / (b0.abs() ** 2).sum()).cpu().numpy()  # [y][x]

    def fit(self, raw):
        case, n = self.case, self.g["n"]
        fr = self.frames(raw)
        att = 1 - 0.99 * torch.exp(-self.radius(n) ** 2 / (2 * (0.15 * self.g["cutoff"] / 2.355) ** 2))
        x = torch.arange(n, device=self.dev)
        x = torch.where(x < n // 2, x, x - n).double()
        rad = torch.sqrt(x[None, :] ** 2 + x[:, None] ** 2)
        hb = 3 if case["bands"] == 3 else 1
        peaks, pars, mods = [], [], []
        for a in range(case["dirs"]):
            sep = self.separate(fr, a, self.matrix(0.0, 1.0))
            c = torch.fft.fft2(torch.fft.ifft2(sep[hb] * att) * torch.fft.ifft2(sep[0] * att).conj()).abs()
            c = torch.where(rad > 0.6 * self.g["cutoff"] / self.cpm, c, torch.full_like(c, -1.0))
            iy, ix = divmod(int(c.argmax()), n)
            kx, ky = -(ix - n if ix > n / 2 else ix), -(n - iy if iy > n / 2 else -iy)
            search = 2.5
            for _ in range(3):
                b0, b1 = self.common(sep[0], sep[hb], kx, ky)
                kxs = [kx + (i - 4.5) / 4.5 * search for i in range(10)]
                kys = [ky + (i - 4.5) / 4.5 * search for i in range(10)]
                g = self.correlate(b0, b1, kxs, kys)
                iy, ix = divmod(int(np.abs(g).argmax()), 10)
                kx, ky, best, search = kxs[ix], kys[iy], g[iy, ix], search / 5
            peaks.append([kx, ky, math.atan2(best.imag, best.real), abs(best)])
            nb = case["bands"] - 1
            pk = []
            for b in range(1, nb + 1):
                q = (kx * b / nb, ky * b / nb)
                b0, b1 = self.common(sep[0], sep[2 * b - 1], *q)
                pk.append(self.correlate(b0, b1, [q[0]], [q[1]])[0, 0])
            pars.append([-kx / nb, -ky / nb, math.atan2(pk[0].imag, pk[0].real)])
            mods.append([abs(p) for p in pk])
        return [np.array(peaks), np.array(pars).T.copy(), np.array(mods)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "fft2d":
        x = _fft_input(case, seed).to(torch.complex128)
        return torch.fft.ifft2(x) if case["inverse"] else torch.fft.fft2(x)
    geo, idx, raw = _raw(case, seed)
    out = []
    for i, r in zip(idx, raw):
        e = _Exact(case, geo[i], r.device)
        if kind == "fit":
            return e.fit(r)
        out.append(e.live(r) if kind == "live" else e.offline(r))
    if kind == "host":
        return torch.stack([o[0] for o in out]).cpu()
    return [[torch.stack([out[j][k] for j in g]) for k in range(len(out[0]))]
            for _, g in _groups([geo[i]["n"] for i in idx])]
