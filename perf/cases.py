"""Performance cases: the reconstruction calls a user of this package makes, through its public
entry points, on seeded synthetic far-field scans.

A pass of a reconstruction case starts from the same estimate (`set_object_device`,
`set_probe_device`, `set_positions`), runs a few epochs or cycles of one algorithm on a handle
the program keeps, and reads the arrays back as a program does; a pass of an adjoint case is one
`autograd.poisson_loss` forward and backward on CUDA tensors. `exact` restates each algorithm in
torch float64 from the published update rules, without this package.
"""
import math

import numpy as np
import torch

from ptyrs_b200 import GpuPtycho, Scan
from ptyrs_b200 import autograd

WAVELENGTH, DETECTOR_PIXEL = 1.0e-10, 75e-6
SIDES = (64, 96, 128, 192, 256)
# sums over pixels x modes x frames x passes that a drawn case may cost: the largest listed one's
BUDGET = 4000 * 256 * 256 * 2 * 2


def _case(algo, n, modes, frames, obj, step, passes, batch=0, photons=1e6, counts="f32",
          masked=False, offsets=False, refine=False, cost="poisson", slices=1):
    return dict(algo=algo, n=n, modes=modes, frames=frames, obj=obj, step=float(step),
                passes=passes, batch=batch, photons=float(photons), counts=counts, masked=masked,
                offsets=offsets, refine=refine, cost=cost, slices=slices)


def listed():
    def named(name, *a, **k):
        return dict(_case(*a, **k), name=name)
    return [
        # a first look at a short scan while it is still being taken: one epoch, one batch;
        # launches and latency are all there is
        named("rpie64_preview", "rpie", 64, 1, 60, 128, 5, 1, batch=100, photons=1e5,
              counts="u16"),
        # the rPIE configuration: 400 frames, 256² object, batches of 100
        named("rpie64_raster", "rpie", 64, 1, 400, 256, 8, 10, batch=100, photons=1e5),
        # rPIE that refines positions on a partially coherent probe, ragged last batch
        named("rpie128_positions", "rpie", 128, 2, 601, 640, 10, 1, batch=150, counts="u16",
              photons=4e5, offsets=True, refine=True),
        # the LSQML configuration: 4096 frames of 128², three modes, Poisson, batches of 256
        named("lsqml128_poisson", "lsqml", 128, 3, 4096, 1024, 6, 2, batch=256),
        # a detector with gaps and dead pixels, 16-bit counts, a side that is no power of two,
        # the amplitude cost, an odd object and frame count
        named("lsqml96_amplitude", "lsqml", 96, 2, 1101, 777, 7, 3, batch=100, photons=2e5,
              counts="u16", masked=True, cost="amplitude"),
        # the multislice configuration's shapes: three slices, two modes
        named("lsqml128_slices", "lsqml", 128, 2, 1500, 1152, 12, 1, batch=256, slices=3),
        # the headline: maximum likelihood refining the positions of 256² frames, two modes
        named("ml256_positions", "ml", 256, 2, 4000, 1536, 12, 2, photons=1e7, offsets=True,
              refine=True),
        # maximum likelihood polishing a masked 192² scan, one mode, odd sizes
        named("ml192_masked", "ml", 192, 1, 997, 1001, 12, 3, masked=True),
        # the carried-wave configuration: DM at 256², two modes
        named("dm256", "dm", 256, 2, 2048, 1280, 12, 4, photons=1e7),
        # many AP cycles of a plain one-mode 128² scan from 16-bit counts
        named("ap128", "ap", 128, 1, 2500, 768, 8, 8, counts="u16", photons=4e5),
        # the adjoint inside a torch program: the loss and the object, probe and position
        # gradients of a mini-batch of frames
        named("adjoint128_positions", "adjoint", 128, 2, 300, 512, 8, 1, offsets=True),
        # the smallest adjoint call: a few frames, object and probe gradients
        named("adjoint64_small", "adjoint", 64, 1, 16, 128, 8, 1, photons=1e5),
    ]


def draw(rng):
    algo = rng.choice(["rpie", "rpie", "lsqml", "lsqml", "slices", "ml", "ml", "dm", "raar",
                       "ap", "adjoint"])
    n = rng.choice(SIDES)
    modes = rng.randint(1, 2 if n >= 192 else 3)
    slices = 1
    if algo == "slices":
        algo, slices, n, modes = "lsqml", rng.randint(2, 3), min(n, 128), min(modes, 2)
    passes = rng.randint(1, 6)
    cost_factor = 3 * slices if slices > 1 else 2
    most = min(4096, BUDGET // (cost_factor * passes * n * n * modes))
    frames = int(round(math.exp(rng.uniform(math.log(16), math.log(max(17, most))))))
    step = rng.uniform(n / 24.0, n / 9.0)
    extent = step * math.sqrt(frames / math.pi)
    obj = n + 2 * int(extent) + rng.randint(12, 75)
    offsets = algo in ("rpie", "ml", "adjoint") and rng.random() < 0.5
    if offsets:
        passes = min(passes, 2)
    return _case(algo, n, modes, frames, obj, step, passes, batch=rng.randint(24, 300),
                 photons=10.0 ** rng.uniform(4.5, 5.6), counts=rng.choice(["u16", "f32"]),
                 masked=rng.random() < 0.4, offsets=offsets,
                 refine=offsets and algo != "adjoint",
                 cost=rng.choice(["poisson", "amplitude"]) if algo == "lsqml" else "poisson",
                 slices=slices)


# Inputs --------------------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _geometry(case):
    """The object pixel of 10 nm at every side: the detector's distance follows."""
    pixel = 1.0e-8
    return pixel, pixel * case["n"] * DETECTOR_PIXEL / WAVELENGTH


def _freq(n):
    return torch.fft.fftfreq(n, dtype=torch.float64, device=_device())


def _smooth_object(side, gen, phase):
    """Unit transmission with smoothed noise in modulus and phase (sigma 3 px)."""
    dev = _device()
    f = _freq(side)
    blur = torch.exp(-2.0 * (math.pi * 3.0) ** 2 * (f[:, None] ** 2 + f[None, :] ** 2))
    g = torch.fft.ifft2(torch.fft.fft2(
        torch.rand(side, side, generator=gen, device=dev, dtype=torch.float64)) * blur).real
    g = (g - g.min()) / (g.max() - g.min())
    return torch.polar(1.0 - 0.2 * g, phase * g)


def _probe(n, modes, defocus):
    """A defocused aperture of radius n/4 with soft edges and its Hermite modes, unit power."""
    x = (torch.arange(n, dtype=torch.float64, device=_device()) - n / 2.0) / (n / 4.0)
    r2 = x[:, None] ** 2 + x[None, :] ** 2
    amp = torch.sigmoid((1.0 - torch.sqrt(r2)) * (n / 4.0) / 1.5)
    base = torch.polar(amp, defocus * r2)
    planes = [base, base * (2.0 * x)[None, :], base * (2.0 * x)[:, None]][:modes]
    power = [[1.0], [0.8, 0.2], [0.8, 0.15, 0.05]][modes - 1]
    return torch.stack([p * math.sqrt(w) / torch.linalg.vector_norm(p)
                        for p, w in zip(planes, power)])


def _scan_positions(case, rng):
    """A Fermat spiral with sub-pixel jitter, in object pixels about its mean."""
    k = np.arange(case["frames"], dtype=np.float64)
    r = case["step"] * np.sqrt(k / np.pi)
    t = k * np.pi * (3.0 - np.sqrt(5.0))
    pos = np.stack([r * np.sin(t), r * np.cos(t)], 1)
    pos += rng.uniform(-0.6, 0.6, pos.shape)
    return pos - pos.mean(axis=0)


def _corners(case, pos):
    """The integer windows: `round_half_even((object - frame)//2 + position)`."""
    c = np.round((case["obj"] - case["n"]) // 2 + pos).astype(np.int64)
    if (c < 0).any() or (c > case["obj"] - case["n"]).any():
        raise ValueError("a window leaves the object")
    return c


def _windows(obj, corners, n):
    """`[B, n, n]` windows of a 2-D array."""
    ar = torch.arange(n, device=obj.device)
    c = torch.as_tensor(corners, device=obj.device)
    return obj[(c[:, 0, None] + ar)[:, :, None], (c[:, 1, None] + ar)[:, None, :]]


def _add_windows(acc, corners, vals):
    n = vals.shape[-1]
    for (y, x), v in zip(corners.tolist(), vals):
        acc[y:y + n, x:x + n] += v


def _chunks(case, total, planes):
    """Ranges of frames of about 256 MB of complex128 per `planes` planes."""
    step = max(1, int(2 ** 28 // (16 * planes * case["n"] ** 2)))
    return [(s, min(total, s + step)) for s in range(0, total, step)]


def _gap(case, pixel, depth):
    """Angular-spectrum transfer function over `depth` metres."""
    f = _freq(case["n"])
    ratio = (f[:, None] ** 2 + f[None, :] ** 2) / (pixel / WAVELENGTH) ** 2
    phase = 2.0 * math.pi * depth / WAVELENGTH * torch.sqrt(torch.clamp(1.0 - ratio, min=0.0))
    return torch.polar((ratio < 1.0).to(torch.float64), phase)


def _inputs(case, seed):
    """The seeded scan: counts (numpy, detector order), positions, windows and the start."""
    dev, n, K = _device(), case["n"], case["modes"]
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * (seed % 2000003) + 17)
    rng = np.random.default_rng([seed, 5])
    pixel, distance = _geometry(case)
    pos = _scan_positions(case, rng)
    corners = _corners(case, pos)
    S = case["slices"]
    truth = torch.stack([_smooth_object(case["obj"], gen, math.pi / (2 * S)) for _ in range(S)])
    probe = _probe(n, K, 10.0)
    gaps = [1.0e-5] * (S - 1)
    offsets = np.zeros((case["frames"], 2))
    near = case["algo"] in ("ml", "adjoint")
    if case["offsets"]:
        true_offsets = rng.normal(0.0, 0.3 if near else 0.7, offsets.shape)
    else:
        true_offsets = offsets
    # the frames: every probe mode moved by the frame's true offset, through the slices
    spec = torch.fft.fft2(probe)
    f = _freq(n)
    P = case["frames"]
    inten = torch.empty((P, n, n), dtype=torch.float32, device=dev)
    props = [_gap(case, pixel, g).to(torch.complex64) for g in gaps]
    t32 = truth.to(torch.complex64)
    for s0, s1 in _chunks(case, P, 2 * K):
        psi = probe.to(torch.complex64)[None].expand(s1 - s0, -1, -1, -1)
        if case["offsets"]:
            d = torch.as_tensor(true_offsets[s0:s1], device=dev)
            ph = -2.0 * math.pi * (f[:, None] * d[:, 0, None, None]
                                   + f[None, :] * d[:, 1, None, None])
            psi = torch.fft.ifft2(spec[None] * torch.polar(torch.ones_like(ph), ph)[:, None])
            psi = psi.to(torch.complex64)
        for s in range(S):
            psi = psi * _windows(t32[s], corners[s0:s1], n)[:, None]
            if s + 1 < S:
                psi = torch.fft.ifft2(torch.fft.fft2(psi) * props[s])
        far = torch.fft.fft2(psi, norm="ortho")
        inten[s0:s1] = torch.fft.fftshift((far.abs() ** 2).sum(dim=1), dim=(-2, -1))
    inten *= case["photons"] / inten.sum(dim=(1, 2)).mean()
    counts = torch.poisson(inten, generator=gen)
    del inten
    if case["masked"]:
        # a module gap across the detector and dead pixels
        bad = torch.rand(n, n, generator=gen, device=dev) < 0.002
        bad[n // 3:n // 3 + 3, :] = True
        counts = torch.where(bad, torch.full_like(counts, -1.0), counts)
    # the start: half the object's contrast, the probe dim, dephased and out of focus; maximum
    # likelihood and its gradients polish an estimate another algorithm has brought near
    start = 1.0 + (0.95 if near else 0.5) * (truth - 1.0)
    probe0 = _probe(n, K, 9.95 if near else 9.0) * (0.9 * math.sqrt(case["photons"]))
    probe0 = probe0 * torch.polar(torch.ones((), dtype=torch.float64, device=dev),
                                  torch.full((), 0.2, dtype=torch.float64, device=dev))
    return dict(counts=counts, pos=pos, corners=corners, object=start, probe=probe0,
                offsets=offsets, gaps=gaps, pixel=pixel, distance=distance)


def prepare(case, seed):
    s = _inputs(case, seed)
    counts = s["counts"]
    if case["counts"] == "u16":
        c = counts.clamp(max=65534.0)
        c = torch.where(counts < 0, torch.full_like(c, 65535.0), c)
        host = c.to(torch.int32).to(torch.uint16).cpu().numpy()
    else:
        host = counts.cpu().numpy()
    s.pop("counts")
    scan = Scan(host, s["pos"][:, 0] * s["pixel"], s["pos"][:, 1] * s["pixel"], WAVELENGTH,
                s["distance"], DETECTOR_PIXEL)
    engine = GpuPtycho(scan, s["object"].cpu().numpy(), s["probe"].cpu().numpy(),
                       gaps=s["gaps"] if case["slices"] > 1 else None)
    state = dict(case=case, engine=engine, object=s["object"].to(torch.complex64).contiguous(),
                 probe=s["probe"].to(torch.complex64).contiguous(),
                 offsets=s["offsets"] if case["offsets"] else None)
    if case["algo"] == "adjoint":
        state["object"].requires_grad_(True)
        state["probe"].requires_grad_(True)
        if case["offsets"]:
            state["offsets"] = torch.as_tensor(s["offsets"], device=_device())
            state["offsets"].requires_grad_(True)
    elif case["offsets"]:
        engine.set_positions(s["offsets"], refine=case["refine"])
    return state


def run(state):
    case, h = state["case"], state["engine"]
    if case["algo"] == "adjoint":
        o, p, d = state["object"], state["probe"], state["offsets"]
        o.grad = p.grad = None
        if d is not None:
            d.grad = None
        loss = autograd.poisson_loss(o, p, d, h)
        loss.backward()
        return dict(loss=loss.detach(), object=o.grad, probe=p.grad,
                    positions=None if d is None else d.grad)
    o, p = state["object"], state["probe"]
    if case["slices"] > 1:
        h.set_objects_device(o.data_ptr(), *o.shape)
    else:
        h.set_object_device(o.data_ptr(), *o.shape)
    h.set_probe_device(p.data_ptr(), *p.shape)
    if case["offsets"]:
        h.set_positions(state["offsets"], refine=case["refine"])
    k = case["passes"]
    if case["algo"] == "rpie":
        h.rpie(k, batch_size=case["batch"])
    elif case["algo"] == "lsqml":
        h.lsqml(k, batch_size=case["batch"], cost=case["cost"])
    elif case["algo"] == "ml":
        h.ml(k, update_probe=True)
    elif case["algo"] == "dm":
        h.dm(k)
    elif case["algo"] == "raar":
        h.raar(k)
    else:
        h.ap(k, probe_inertia=0.01)
    return dict(object=h.objects() if case["slices"] > 1 else h.object(), probe=h.probe(),
                positions=h.positions() if case["refine"] else None)


# Transforms of a pass per frame and mode that the algorithm cannot do without.
TRANSFORMS = dict(rpie=2, lsqml=2, ml=3, dm=2, raar=2, ap=2, adjoint=2)


def work(case):
    n, K, P, S, algo = case["n"], case["modes"], case["frames"], case["slices"], case["algo"]
    passes = case["passes"] if algo != "adjoint" else 1
    transforms = TRANSFORMS[algo] + 4 * (S - 1)
    if case["offsets"]:
        # the probe moved by the offset and its directions moved back
        transforms += {"rpie": 3, "ml": 3, "adjoint": 2}[algo]
        # the position derivatives of one mode (rPIE) or of both axes of every mode
        transforms += {"rpie": 2 + 3.0 / K, "ml": 4, "adjoint": 2}[algo]
    frame = 4 * n * n  # the counts, once per pass over the scan
    if algo in ("dm", "raar"):
        frame += 16 * K * n * n  # the carried waves read and written
    if algo == "raar":
        frame += 16 * K * n * n
    if algo == "ml":
        frame += 4 * n * n  # the line search needs every frame a second time
    arrays = 16 * (S * case["obj"] ** 2 + K * n * n)
    flops = transforms * 5.0 * n * n * math.log2(n * n) * K
    return dict(bytes=float(passes * (P * frame + arrays)), flops=float(passes * P * flops))


def tolerance(case):
    # 32-bit transforms and sums against 64 bits, measured over the listed and some drawn cases:
    # rPIE 1e-7 to 3e-5 (the modulus ratio at the dark pixels of the detector amplifies a
    # transform's rounding, and the batches carry it on), LSQML to 3e-6 (through slices), AP, DM
    # and RAAR to 1.5e-6, ML to 3e-7 after two cycles, the gradients to 3e-6 (1 - I/model where
    # the model is small). Stated with room for draws that amplify more.
    return {"rel": {"rpie": 1e-4, "lsqml": 3e-5, "ml": 2e-5, "adjoint": 2e-5}.get(case["algo"],
                                                                             1e-5)}


# The same algorithms in 64 bits ----------------------------------------------------------------

def _shift(a):
    return torch.fft.fftshift(a, dim=(-2, -1))


def _fft(a):
    return torch.fft.fft2(a, norm="ortho")


def _ifft(a):
    return torch.fft.ifft2(a, norm="ortho")


class _Exact:
    """One scan's float64 state: natural-layout planes, detector planes FFT-shifted."""

    def __init__(self, case, seed):
        s = _inputs(case, seed)
        self.case, self.n, self.P, self.K = case, case["n"], case["frames"], case["modes"]
        c = s["counts"]
        if case["counts"] == "u16":
            c = c.clamp(max=65534.0)
        self.iobs = _shift(c)
        self.corners = s["corners"]
        # the engine's start is the 32-bit one
        self.obj, self.probe = (s[k].to(torch.complex64).to(torch.complex128)
                                for k in ("object", "probe"))
        self.d = torch.as_tensor(s["offsets"], device=_device()) if case["offsets"] else None
        self.tf = [_gap(case, s["pixel"], g) for g in s["gaps"]]
        x = torch.arange(self.n, dtype=torch.float64, device=_device()) - self.n // 2
        f = math.pi / (WAVELENGTH * s["distance"]) * s["pixel"] ** 2
        ph = f * (x[:, None] ** 2 + x[None, :] ** 2)
        self.q = torch.polar(torch.ones_like(ph), ph)
        self.f = _freq(self.n)
        self.cycle = 0

    def counts_of(self, frames):
        c = self.iobs[frames].to(torch.float64)
        return torch.clamp(c, min=0.0), c < 0

    def phase(self, frames):
        d = self.d[frames]
        ph = -2.0 * math.pi * (self.f[:, None] * d[:, 0, None, None]
                               + self.f[None, :] * d[:, 1, None, None])
        return torch.polar(torch.ones_like(ph), ph)[:, None]

    def moved(self, planes, frames, back=False, axis=None):
        """conj(q)·T_d(q·planes), T_{-d} with `back`, or its derivative over one offset."""
        e = self.phase(frames)
        if back:
            e = e.conj()
        if axis is not None:
            e = e * (-2j * math.pi * (self.f[:, None] if axis == 0 else self.f[None, :]))
        return torch.fft.ifft2(torch.fft.fft2(planes * self.q) * e) * self.q.conj()

    def probes(self, frames, probe=None):
        p = self.probe if probe is None else probe
        if self.d is None:
            return p[None].expand(len(frames), -1, -1, -1)
        return self.moved(p[None], frames)

    def windows(self, frames, obj=None):
        o = self.obj[0] if obj is None else obj
        return _windows(o, self.corners[frames.cpu().numpy()], self.n)[:, None]

    def far(self, psi):
        return _fft(_shift(psi * self.q))

    def near(self, far):
        """The exit waves without their phase: conj(q)·shift(IFFT(far))."""
        return _shift(_ifft(far)) * self.q.conj()

    def add(self, acc, frames, vals):
        _add_windows(acc, self.corners[frames.cpu().numpy()], vals)

    def ranges(self, planes=6):
        for a, b in _chunks(self.case, self.P, planes * self.K):
            yield torch.arange(a, b, device=_device())

    def batches(self, size, epoch):
        """Seeded shuffled batches: SplitMix64 Fisher-Yates, each batch sorted."""
        m64 = (1 << 64) - 1

        def mix(z):
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m64
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m64
            return z ^ (z >> 31)
        state, order = (7 ^ mix(epoch)) & m64, list(range(self.P))
        for i in range(self.P - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & m64
            j = (mix(state) * (i + 1)) >> 64
            order[i], order[j] = order[j], order[i]
        return [torch.as_tensor(sorted(order[s:s + size]), device=_device())
                for s in range(0, self.P, size)]

    def zero_phase_ramp(self):
        """The probe's far field centred by a ramp, and its inverse on the object."""
        v = (_shift(torch.fft.fft2(_shift(self.probe))).abs() ** 2).sum(dim=0)
        i = torch.arange(self.n, dtype=torch.float64, device=_device())
        dy = ((v * i[:, None]).sum() / v.sum()).item() - self.n // 2
        dx = ((v * i[None, :]).sum() / v.sum()).item() - self.n // 2

        def ramp(length, sign):
            t = (torch.arange(length, dtype=torch.float64, device=_device())
                 - length // 2) * (sign * 2.0 * math.pi / self.n)
            ph = dy * t[:, None] + dx * t[None, :]
            return torch.polar(torch.ones_like(ph), ph)
        self.probe = self.probe * ramp(self.n, -1.0)
        self.obj = self.obj * ramp(self.obj.shape[-1], 1.0)

    # rPIE ------------------------------------------------------------------------------------
    def rpie(self):
        alpha = 0.1
        for ep in range(self.case["passes"]):
            for frames in self.batches(min(self.case["batch"], self.P), ep):
                iobs, mask = self.counts_of(frames)
                w, o = self.probes(frames), self.windows(frames)
                psi = w * o
                far = self.far(psi)
                r = torch.sqrt(iobs + 1e-7) / (torch.sqrt((far.abs() ** 2).sum(1)) + 1e-7)
                delta = self.near(far * torch.where(mask, torch.ones_like(r), r)[:, None]) - psi
                side = self.obj.shape[-1]
                num = torch.zeros((self.K, side, side), dtype=torch.complex128, device=w.device)
                den = torch.zeros((self.K, side, side), dtype=torch.float64, device=w.device)
                for m in range(self.K):
                    self.add(num[m], frames, w[:, m].conj() * delta[:, m])
                    self.add(den[m], frames, w[:, m].abs() ** 2)
                d_obj = (num / ((1 - alpha) * den + alpha * den.sum(0).max())).sum(0)
                o2 = o.abs() ** 2
                omax = o2.amax(dim=(-2, -1), keepdim=True)
                dp = o.conj() / ((1 - alpha) * o2 + alpha * omax) * delta
                if self.d is not None:
                    dp = self.moved(dp, frames, back=True)
                step = self.position_step(frames, w, o, delta) if self.case["refine"] else None
                self.obj = self.obj + d_obj[None]
                self.probe = self.probe + dp.sum(0) / len(frames)
                if step is not None:
                    self.d[frames] += step

    def position_step(self, frames, w, o, delta):
        """pty-chi's clipped gradient step on the batch, from the main mode."""
        spec = torch.fft.fft2(o[:, 0])
        step = torch.zeros((len(frames), 2), dtype=torch.float64, device=o.device)
        for axis in range(2):
            f = self.f[:, None] if axis == 0 else self.f[None, :]
            u = torch.fft.ifft2(spec * (2j * math.pi * f)) * w[:, 0]
            num = (u.conj() * delta[:, 0]).real.sum(dim=(-2, -1))
            den = (u.abs() ** 2).sum(dim=(-2, -1))
            dx = 0.3 * num / (den + torch.clamp(den.max(), min=1e-6 * self.n ** 2))
            mean = dx.sum() / self.P
            dev = (dx - mean).abs().sum() + (self.P - len(frames)) * mean.abs()
            limit = min(10.0 * (dev / self.P).item(), 0.1)
            step[:, axis] = dx.clamp(-limit, limit)
        return step

    # LSQML -----------------------------------------------------------------------------------
    def lsqml(self):
        n, K, S = self.n, self.K, self.case["slices"]
        poisson = self.case["cost"] == "poisson"
        afar = torch.full((self.P,), 0.5, dtype=torch.float64, device=_device())
        pre = None
        for ep in range(self.case["passes"]):
            illum = torch.zeros(self.obj.shape[1:], dtype=torch.float64, device=_device())
            p2 = (self.probe.abs() ** 2).sum(0)
            for y, x in self.corners.tolist():
                illum[y:y + n, x:x + n] += p2
            if pre is None:
                power = max(self.counts_of(f)[0].sum(dim=(1, 2)).max().item()
                            for f in self.ranges())
                pre = illum * (power / (4.0 * n ** 4))
            pre = (pre + illum) / 2.0
            for frames in self.batches(min(self.case["batch"], self.P), ep):
                self.lsqml_step(frames, afar, torch.sqrt(pre ** 2 + (0.1 * pre.max()) ** 2),
                                poisson, S, K)

    def lsqml_step(self, frames, afar, scale, poisson, S, K):
        n, B = self.n, len(frames)
        iobs, mask = self.counts_of(frames)
        win = [self.windows(frames, self.obj[s]) for s in range(S)]
        waves = [self.probe[None].expand(B, -1, -1, -1)]
        for s in range(S - 1):
            waves.append(torch.fft.ifft2(torch.fft.fft2(waves[s] * win[s]) * self.tf[s]))
        psi = waves[-1] * win[-1]
        far = self.far(psi)
        calc = (far.abs() ** 2).sum(1)
        if poisson:
            a = afar[frames]
            zero = torch.zeros_like(calc)
            for _ in range(2):
                prev = a.mean()
                xi = 1.0 - iobs / (calc + 1e-5)
                num = torch.where(mask, zero, xi * (calc - iobs / (1.0 - prev * xi))).sum((1, 2))
                den = torch.where(mask, zero, xi * xi * calc).sum((1, 2))
                a = (0.5 * prev + 0.5 * torch.where(den > 0, num / den,
                                                    torch.zeros_like(den))).clamp(0.0, 1.0)
            c = 1.0 - iobs / (calc + 1e-6)
            afar[frames] = a
        else:
            a = torch.full((B,), 0.5, dtype=torch.float64, device=calc.device)
            c = 2.0 * (1.0 - torch.sqrt(iobs) / (torch.sqrt(calc) + 1e-9))
        fac = 1.0 - a[:, None, None] * torch.where(mask, torch.zeros_like(c), c)
        chis = [self.near(far * fac[:, None]) - psi]
        for s in range(S - 2, -1, -1):
            back = win[s + 1].conj() * chis[0]
            chis.insert(0, torch.fft.ifft2(torch.fft.fft2(back) * self.tf[s].conj()))
        d_obj = []
        for s in range(S):
            acc = torch.zeros(self.obj.shape[1:], dtype=torch.complex128, device=calc.device)
            self.add(acc, frames, (waves[s].conj() * chis[s]).sum(1))
            d_obj.append(acc / scale)
        d_probe = (win[0].conj() * chis[0]).sum(0) / B
        # Eq. 22 on slice 0 jointly with the probe
        u = waves[0] * self.windows(frames, d_obj[0])
        v = d_probe[None] * win[0]
        dims = (1, 2, 3)
        reg = 1.2e-7 * K * n * n
        a11, a22 = (u.abs() ** 2).sum(dims) + reg, (v.abs() ** 2).sum(dims) + reg
        a12 = (u * v.conj()).sum(dims)
        b1, b2 = ((t.conj() * chis[0]).real.sum(dims) for t in (u, v))
        a11, a22 = a11 + 0.1 * a11.mean(), a22 + 0.1 * a22.mean()
        det = a11 * a22 - a12.abs() ** 2
        x0 = ((a22 * b1 - a12.real * b2) / det).clamp(min=0.0) * 0.9 / (S * K)
        x1 = ((a11 * b2 - a12.real * b1) / det).clamp(min=0.0) * 0.9
        steps = [x0]
        for s in range(1, S):
            du = waves[s] * self.windows(frames, d_obj[s])
            num, den = (du.conj() * chis[s]).real.sum(dims), (du.abs() ** 2).sum(dims)
            steps.append((0.5 * num / den * 0.9 / (S * K)).clamp(min=0.0))
        k = math.ceil(B * 0.1 / 2.0 - 0.5)
        for s in range(S):
            kept = torch.sort(steps[s])[0][k:B - k]
            self.obj[s] += kept.mean() * d_obj[s]
        self.probe = self.probe + x1.mean() * d_probe

    # ML and the adjoint ------------------------------------------------------------------------
    def poisson_gradients(self, refine=False, positions=False):
        """The Poisson sum, its object and probe gradients (real and imaginary parts), and the
        position gradient or, with `refine`, the magnitude projection's position sums."""
        go = torch.zeros_like(self.obj[0])
        gp = torch.zeros_like(self.probe)
        loss, sums = 0.0, torch.zeros((self.P, 4), dtype=torch.float64, device=_device())
        for frames in self.ranges(10):
            iobs, mask = self.counts_of(frames)
            w, o = self.probes(frames), self.windows(frames)
            far = self.far(w * o)
            calc = (far.abs() ** 2).sum(1)
            zero = torch.zeros_like(calc)
            p = torch.where(iobs > 0, calc - iobs + torch.xlogy(iobs, iobs / calc), calc)
            loss += torch.where(mask, zero, p).sum().item()
            r = torch.where(mask, zero, 2.0 * (1.0 - iobs / calc.clamp(min=1e-12)))
            g = self.near(far * r[:, None])
            self.add(go, frames, (w.conj() * g).sum(1))
            y = o.conj() * g
            gp += (y if self.d is None else self.moved(y, frames, back=True)).sum(0)
            if refine or positions:
                c = g
                if refine:
                    r = torch.sqrt(iobs) / torch.sqrt(calc).clamp(min=1e-12) - 1.0
                    c = self.near(far * torch.where(mask, zero, r)[:, None])
                for axis in range(2):
                    u = o * self.moved(self.probe[None], frames, axis=axis)
                    sums[frames, axis] = (c.conj() * u).real.sum(dim=(1, 2, 3))
                    sums[frames, 2 + axis] = (u.abs() ** 2).sum(dim=(1, 2, 3))
        return loss, go, gp, sums

    def line_search(self, d_obj, d_probe):
        num = den = 0.0
        for frames in self.ranges(10):
            iobs, mask = self.counts_of(frames)
            w, o = self.probes(frames), self.windows(frames)
            dw, do = self.probes(frames, d_probe), self.windows(frames, d_obj)
            po, a, b = self.far(w * o), self.far(w * do + dw * o), self.far(dw * do)
            calc = (po.abs() ** 2).sum(1).clamp(min=1e-32)
            r = (po.conj() * a).real.sum(1)
            s = (a.abs() ** 2 + 2.0 * (po.conj() * b).real).sum(1)
            d = 1.0 - iobs / calc
            zero = torch.zeros_like(calc)
            num -= torch.where(mask, zero, 2.0 * r * d).sum().item()
            den += torch.where(mask, zero,
                               2.0 * s * d + iobs * (2.0 * r / calc) ** 2).sum().item()
        return num / den

    def ml(self):
        total = calc = 0.0
        for frames in self.ranges():
            iobs, mask = self.counts_of(frames)
            far = self.far(self.probes(frames) * self.windows(frames))
            keep = (~mask).to(torch.float64)
            total += iobs.sum().item()
            calc += ((far.abs() ** 2).sum(1) * keep).sum().item()
        s = math.sqrt(total / calc)
        so, sp = self.obj.abs().sum().item(), self.probe.abs().sum().item()
        self.probe = self.probe * math.sqrt(so / sp * s)
        self.obj = self.obj * math.sqrt(sp / so * s)
        last = None
        d_obj, d_probe = torch.zeros_like(self.obj[0]), torch.zeros_like(self.probe)
        for _ in range(self.case["passes"]):
            _, go, gp, sums = self.poisson_gradients(refine=self.case["refine"])
            beta = 0.0
            if last is not None:
                num = sum((g.conj() * (g - h)).real.sum().item()
                          for g, h in zip((go, gp), last))
                beta = max(0.0, num / sum((h.abs() ** 2).sum().item() for h in last))
            d_obj, d_probe = d_obj * beta - go, d_probe * beta - gp
            gamma = self.line_search(d_obj, d_probe)
            self.obj = self.obj + gamma * d_obj
            self.probe = self.probe + gamma * d_probe
            last = (go, gp)
            if self.case["refine"]:
                for axis in range(2):
                    den = sums[:, 2 + axis]
                    step = (0.3 * sums[:, axis] / (den + den.max())).clamp(-0.1, 0.1)
                    self.d[:, axis] += step - step.mean()
        self.zero_phase_ramp()

    # AP, DM and RAAR -----------------------------------------------------------------------------
    def carried(self, algo):
        passes, side = self.case["passes"], self.obj.shape[-1]
        pi, mix, h = (0.01 if algo == "ap" else 0.001), 0.02, 0.45
        psi = torch.empty((self.P, self.K, self.n, self.n), dtype=torch.complex128,
                          device=_device())
        it = torch.empty_like(psi) if algo == "raar" else None
        for ic in range(passes):
            o_num = torch.zeros((side, side), dtype=torch.complex128, device=_device())
            p_num = torch.zeros_like(self.probe)
            norm = torch.zeros((self.n, self.n), dtype=torch.float64, device=_device())
            illum = torch.zeros((side, side), dtype=torch.float64, device=_device())
            p2 = (self.probe.abs() ** 2).sum(0)

            def probe_sums():
                for frames in self.ranges():
                    o = self.windows(frames)
                    p_num.add_((o.conj() * psi[frames]).sum(0))
                    norm.add_((o.abs() ** 2).sum((0, 1)))
            for frames in self.ranges():
                iobs, mask = self.counts_of(frames)
                po = self.probes(frames) * self.windows(frames)
                if algo == "ap" or ic == 0:
                    x = po
                elif algo == "dm":
                    x = po * (2.0 - mix) - psi[frames] * (1.0 - mix)
                else:
                    x = psi[frames] * (1.0 - h) + (po * 2.0 - it[frames]) * h
                if it is not None:
                    it[frames] = x
                far = self.far(x)
                r = torch.sqrt(iobs) / torch.sqrt((far.abs() ** 2).sum(1)).clamp(min=1e-12)
                new = self.near(far * torch.where(mask, torch.ones_like(r), r)[:, None])
                if algo == "dm" and ic > 0:
                    new = new + (po - x) * (1.0 - mix)
                psi[frames] = new
                self.add(o_num, frames, (self.probe.conj()[None] * new).sum(1))
            for y, x in self.corners.tolist():
                illum[y:y + self.n, x:x + self.n] += p2
            if algo == "ap":
                probe_sums()
            reg = illum.max() * 0.01
            self.obj = ((o_num + self.obj[0] * reg) / (illum + reg).clamp(min=1e-12))[None]
            if algo != "ap":
                probe_sums()
            reg = norm.max() * pi
            self.probe = (p_num + self.probe * reg) / (norm + reg).clamp(min=1e-12)
        self.zero_phase_ramp()


def exact(case, seed):
    x = _Exact(case, seed)
    algo = case["algo"]
    if algo == "adjoint":
        loss, go, gp, sums = x.poisson_gradients(positions=case["offsets"])
        return dict(loss=torch.tensor(loss, dtype=torch.float64), object=go[None], probe=gp,
                    positions=sums[:, :2].contiguous() if case["offsets"] else None)
    if algo in ("rpie", "lsqml", "ml"):
        getattr(x, algo)()
    else:
        x.carried(algo)
    return dict(object=x.obj.cpu().numpy(), probe=x.probe.cpu().numpy(),
                positions=x.d.cpu().numpy() if case["refine"] else None)
