"""Performance cases of the digHolo batch path, each through the public entry
points of libdigholo_b200: one frame for a live view, ordinary and large
batches in both resolution modes and both pixel types, frame averaging, the
AutoAlign gradient and the power meter.

A case is a plain dict:

  frames, width, height, dtype   the camera batch (12-bit uint16, or float32)
  pols, window, groups           polarisations (side by side in the frame),
                                 FFT-window side, mode groups of the HG basis
  mode                           IFFT resolution mode (0 full, 1 window-sized)
  carrier                        off-axis carrier along x in units of Nyquist
                                 (0.8 of it along y); the Fourier window's
                                 radius is a third of the tilt, so it sets
                                 the IFFT window's size
  average                        frames averaged per batch item
  call                           "batch"     device frames, coefficients left on the device
                                 "host"      pinned host frames, coefficients in host memory
                                 "view"      the same, and the reconstructed fields
                                 "gradient"  IL and its gradient over the alignment parameters
                                 "metrics"   batch, then IL and MDL of its coefficients

listed(), draw(rng), prepare(case, seed), run(state), work(case) and
exact(case, seed) are documented below.
"""
import ctypes as C
import math

import numpy as np
import torch

import digholo_b200
from digholo_b200 import api

WAVELENGTH = 1565e-9
PIXEL = 20e-6
STREAM = []          # the one stream that all handles and this module's programs use


def listed():
    def case(name, frames, width, height, dtype, pols, window, groups, mode, carrier, call="batch", average=1):
        return dict(name=name, frames=frames, width=width, height=height, dtype=dtype, pols=pols, window=window,
                    groups=groups, mode=mode, carrier=carrier, call=call, average=average)
    return [
        # a live alignment view: one camera frame from host memory, coefficients and fields back
        case("view_1_640x512_u16", 1, 640, 512, "uint16", 2, 128, 15, 0, 0.25, "view"),
        # a short acquisition of a small camera, where launches and latency count
        case("batch_16_320x256_f32_lowres", 16, 320, 256, "float32", 1, 64, 9, 1, 0.25),
        # the benchmark's workload: a transfer-matrix acquisition, window-sized fields
        case("batch_1024_640x512_u16_lowres", 1024, 640, 512, "uint16", 2, 128, 15, 1, 0.25),
        # the same acquisition at the default (full) resolution
        case("batch_1024_640x512_u16_full", 1024, 640, 512, "uint16", 2, 128, 15, 0, 0.25),
        # a float camera, a ragged number of frames, and a carrier whose window holds every mode
        case("batch_301_640x512_f32_full", 301, 640, 512, "float32", 2, 128, 15, 0, 0.55),
        # a larger float camera with a wide FFT window (uneven streamed batches)
        case("batch_500_1280x1024_f32_lowres", 500, 1280, 1024, "float32", 2, 256, 9, 1, 0.25),
        # a steep carrier: the IFFT window's side (48) is not a power of two
        case("batch_400_640x512_u16_steep_full", 400, 640, 512, "uint16", 2, 128, 15, 0, 0.8),
        # many modes on a large sensor: 512 x 512 fields, 465 modes
        case("batch_96_2048x2048_u16_full", 96, 2048, 2048, "uint16", 2, 512, 30, 0, 0.25),
        # noisy sources: eight frames averaged per item, phases aligned
        case("average_100x8_640x512_u16_lowres", 100, 640, 512, "uint16", 2, 128, 15, 1, 0.25, "batch", 8),
        # frames arriving in pinned host memory: the copies are part of the call
        case("host_200_640x512_u16_lowres", 200, 640, 512, "uint16", 2, 128, 15, 1, 0.25, "host"),
        # one step of the gradient-driven alignment (forward and adjoint)
        case("gradient_512_640x512_f32_full", 512, 640, 512, "float32", 2, 128, 15, 0, 0.55, "gradient"),
        # one evaluation of an alignment towards mode-dependent loss: batch and singular values
        case("metrics_256_640x512_f32_full", 256, 640, 512, "float32", 2, 128, 10, 0, 0.55, "metrics"),
    ]


# camera: (width, height, types, polarisations, windows, group counts, carriers, most frames)
CAMERAS = [
    (320, 256, ("float32", "uint16"), (1, 2), (32, 64), (3, 9), (0.25, 0.4, 0.55), 512),
    (640, 512, ("uint16", "float32"), (1, 2), (64, 128), (5, 20), (0.25, 0.4, 0.55, 0.8), 1024),
    (1280, 1024, ("float32", "uint16"), (1, 2), (128, 256), (6, 20), (0.25, 0.4, 0.55), 256),
    (2048, 2048, ("uint16",), (2,), (256, 512), (10, 30), (0.25, 0.4), 64),
]


def draw(rng):
    """One more case: camera, window, type, resolution and call at random, the frame count over its logarithm."""
    cam = rng.choices(range(4), (3, 5, 2, 2))[0]
    width, height, types, pols, windows, groups, carriers, most = CAMERAS[cam]
    c = dict(frames=max(1, round(math.exp(rng.uniform(0.0, math.log(most))))), width=width, height=height,
             dtype=rng.choice(types), pols=rng.choice(pols), window=rng.choice(windows), groups=rng.randint(*groups),
             mode=rng.randint(0, 1), carrier=rng.choice(carriers), call="batch", average=1)
    if c["window"] == 64:      # the modes of a 64-pixel window
        c["groups"] = min(c["groups"], 9)
    if c["window"] == 32:
        c["groups"] = min(c["groups"], 4)
    if cam == 1:
        kind = rng.random()
        if kind < 0.15:
            c["average"] = rng.choice((2, 4, 8))
            c["frames"] = max(1, c["frames"] // c["average"])
        elif kind < 0.3:
            c["call"] = "host"
            c["frames"] = min(c["frames"], 200)
        elif kind < 0.4:
            c.update(call="view", frames=min(c["frames"], 8))
        elif kind < 0.55:
            c.update(call="gradient", mode=0, carrier=0.55, window=128, dtype="float32", frames=min(512, max(16, c["frames"])))
        elif kind < 0.65:
            c.update(call="metrics", mode=0, carrier=0.55, window=128, groups=rng.randint(5, 10), pols=2,
                     dtype="float32", frames=rng.randint(150, 256))
    return c


# ------------------------------------------------------------------ inputs

def hg_indices(groups):
    """(m, n) of every mode: group g holds (g - k, k)."""
    return [(g - k, k) for g in range(groups) for k in range(g + 1)]


def hermite_gauss(u, count):
    """Normalised Hermite functions psi_0 .. psi_{count-1} at u (float64)."""
    out = [math.pi ** -0.25 * torch.exp(-0.5 * u * u)]
    if count > 1:
        out.append(math.sqrt(2.0) * u * out[0])
    for n in range(2, count):
        out.append(math.sqrt(2.0 / n) * u * out[n - 1] - math.sqrt((n - 1.0) / n) * out[n - 2])
    return torch.stack(out)


class Settings:
    """The configuration of a case: what its user has set before the call."""

    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        W, H, P, win = case["width"], case["height"], case["pols"], case["window"]
        self.frame_width, self.frame_height, self.pixel_size, self.wavelength = W, H, PIXEL, WAVELENGTH
        self.pol_count, self.fft_window, self.resolution_mode, self.max_mg = P, (win, win), case["mode"], case["groups"]
        self.fill_factor, self.pol_lock_tilt, self.pol_lock_defocus, self.pol_lock_waist = 1, 0, 0, 1
        # 250 um on 128 pixels for 15 groups, and in proportion: the highest modes fill the window
        waist = 250e-6 * (win / 128.0) * min(1.6, math.sqrt(15.0 / max(case["groups"], 3)))
        if case["carrier"] >= 0.5:     # the carriers whose Fourier window is wide: a smaller spot
            waist = min(waist, 250e-6 * max(1.0, win / 256.0))
        centre = [((p - 0.5 * (P - 1)) * (W / P) * PIXEL, 0.0) for p in range(P)]
        self.spot = [(c[0] + rng.uniform(-40e-6, 40e-6), c[1] + rng.uniform(-40e-6, 40e-6)) for c in centre]
        self.spot_waist = waist
        self.carriers = [(case["carrier"] * s, 0.8 * case["carrier"] * s) for s in (1.0, -1.0)[:P]]
        k0 = 2.0 * math.pi / WAVELENGTH
        tilt = [math.degrees(abs(c) * math.pi / PIXEL / k0) for c in self.carriers[0]]
        self.window_radius_deg = math.hypot(*tilt) / 3.0
        off = 1.0 if case["call"] == "gradient" else 0.0      # an alignment begins a little off
        self.beam_centre = [(s[0] + off * rng.uniform(-30e-6, 30e-6), s[1] + off * rng.uniform(-30e-6, 30e-6)) for s in self.spot]
        self.tilt_deg = [(tilt[0] + off * rng.uniform(-0.02, 0.02), tilt[1] + off * rng.uniform(-0.02, 0.02)) for _ in self.spot]
        self.defocus = [off * rng.uniform(-0.3, 0.3) for _ in range(2)]
        self.waist = [waist * (1.0 + off * rng.uniform(-0.1, 0.1))] * 2


def camera_frames(case, seed):
    """A batch of off-axis holograms |reference + signal|^2 + noise on the GPU (12-bit counts):
    complex Gaussian mode coefficients, signal power a tenth of the reference's, 28 dB SNR."""
    s = Settings(case, seed)
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed * 7919 + 13)
    n, W, H, P, G = case["frames"], case["width"], case["height"], case["pols"], case["groups"]
    avg = case["average"]
    region = W // P
    ms, ns = (torch.tensor(v, device=dev) for v in zip(*hg_indices(G)))
    xs = (torch.arange(W, device=dev, dtype=torch.float64) - W // 2) * PIXEL
    ys = (torch.arange(H, device=dev, dtype=torch.float64) - H // 2) * PIXEL
    out = torch.empty((n * avg, H, W), device=dev, dtype=torch.int16 if case["dtype"] == "uint16" else torch.float32)
    step = max(1, (1 << 25) // (H * W))
    coefs = [torch.view_as_complex(torch.randn((n, len(ms), 2), generator=gen, device=dev)).repeat_interleave(avg, 0) for _ in range(P)]
    if avg > 1:                # the phase drifts between the frames of an item
        drift = torch.rand((n * avg, 1), generator=gen, device=dev) * (2 * math.pi)
        coefs = [c * torch.polar(torch.ones_like(drift), drift) for c in coefs]
    for f0 in range(0, n * avg, step):
        f1 = min(n * avg, f0 + step)
        clean = torch.empty((f1 - f0, H, W), device=dev)
        for p in range(P):
            xr = xs[p * region:(p + 1) * region]
            hx = hermite_gauss(math.sqrt(2) * (xr - s.spot[p][0]) / s.spot_waist, G).to(torch.complex64)
            hy = hermite_gauss(math.sqrt(2) * (ys - s.spot[p][1]) / s.spot_waist, G).to(torch.complex64)
            kx, ky = (c * math.pi / PIXEL for c in s.carriers[p])
            ref = (torch.exp(1j * ky * ys)[:, None] * torch.exp(1j * kx * xr)[None, :]).to(torch.complex64)
            c = torch.zeros((f1 - f0, G, G), device=dev, dtype=torch.complex64)
            c[:, ns, ms] = coefs[p][f0:f1]
            sig = hy.T @ c @ hx
            # one scale for the batch (relative frame powers survive): each mode has power (waist / sqrt 2 / pixel)^2
            sig *= math.sqrt(0.1 * ref.numel() / (2.0 * len(ms))) * math.sqrt(2.0) * PIXEL / s.spot_waist
            clean[:, :, p * region:(p + 1) * region] = (ref + sig).abs() ** 2
        clean += torch.randn(clean.shape, generator=gen, device=dev) * (1.1 * 10.0 ** (-28.0 / 20.0))
        clean = torch.clamp(torch.round(clean * 300.0), 0, 4095)
        out[f0:f1] = clean.to(out.dtype)
    return out


# ------------------------------------------------------------------ the calls

class Handle:
    """A digHolo handle, destroyed with the last object that uses it; the arrays that run() returns lie in the
    handle's own buffers and hold it."""

    def __init__(self):
        self.L = digholo_b200.load()
        self.h = self.L.digHoloCreate()

    def __del__(self):
        self.L.digHoloDestroy(self.h)

    def device_complex(self, address, shape):
        view = DeviceView()
        view.owner = self
        view.__cuda_array_interface__ = {"data": (address, False), "shape": shape, "typestr": "<c8", "version": 3}
        return torch.as_tensor(view, device="cuda")

    def host_complex(self, p, shape):
        buf = (C.c_float * (2 * math.prod(shape))).from_address(C.cast(p, C.c_void_p).value)
        buf.owner = self
        return np.frombuffer(buf, dtype=np.complex64).reshape(shape)


class DeviceView:
    pass


class State:
    """A handle configured for the case, and the batch it will be given."""

    def __init__(self, case, seed):
        self.handle = Handle()
        self.L, self.h = self.handle.L, self.handle.h
        L = self.L
        self.call, self.count, self.average = case["call"], case["frames"], case["average"]
        frames = camera_frames(case, seed)
        if self.call in ("host", "view"):
            host = torch.empty(frames.shape, dtype=frames.dtype, pin_memory=True)
            host.copy_(frames)
            frames = host
        self.frames = frames
        u16 = case["dtype"] == "uint16"
        self.set = L.digHoloSetBatchAvgUint16 if u16 else L.digHoloSetBatchAvg
        self.ptr = C.cast(C.c_void_p(frames.data_ptr()), C.POINTER(C.c_ushort if u16 else C.c_float))
        self.tail = (0, 0) if u16 else (0,)     # averaging mode, transpose
        if not STREAM:
            STREAM.append(torch.cuda.Stream())
        torch.cuda.synchronize()
        self.cfg = Settings(case, seed)
        api.configure(L, self.h, self.cfg)
        L.digHoloB200SetStream(self.h, C.c_void_p(STREAM[0].cuda_stream))
        self.b, self.m, self.p = C.c_int(), C.c_int(), C.c_int()
        self.w, self.ht = C.c_int(), C.c_int()
        self.x, self.y = C.POINTER(C.c_float)(), C.POINTER(C.c_float)()
        self.grad, self.value = (C.c_float * 12)(), C.c_float()
        self.view = (0, None)

    def check(self, ok):
        if not ok:
            raise RuntimeError("digholo_b200: %s" % self.L.digHoloB200GetLastError(self.h))

    def device_coefs(self):
        p = self.L.digHoloB200GetCoefsDevice(self.h, C.byref(self.b), C.byref(self.m), C.byref(self.p))
        self.check(bool(p))
        address = C.cast(p, C.c_void_p).value
        if self.view[0] != address:
            self.view = (address, self.handle.device_complex(address, (self.b.value, self.p.value, self.m.value)))
        return self.view[1]


def prepare(case, seed):
    """The frames in device memory (pinned host memory for "host" and "view") and a configured handle."""
    return State(case, seed)


def run(s):
    """One pass: SetBatch, the call, and what it returns."""
    L, h = s.L, s.h
    s.set(h, s.count, s.ptr, s.average, *s.tail)
    if s.call == "batch":
        s.check(L.digHoloB200ProcessBatchDevice(h) == 0)
        return s.device_coefs()
    if s.call == "gradient":
        s.check(L.digHoloB200AutoAlignGradient(h, s.grad, C.byref(s.value)) == 0)
        return {"gradient": np.array(s.grad, dtype=np.float32), "il": float(s.value.value)}
    if s.call == "metrics":
        s.check(L.digHoloB200ProcessBatchDevice(h) == 0)
        s.check(L.digHoloAutoAlignCalcMetrics(h) == 0)
        return {"coefs": s.device_coefs(), "il": float(L.digHoloAutoAlignGetMetric(h, 0)), "mdl": float(L.digHoloAutoAlignGetMetric(h, 1))}
    p = L.digHoloProcessBatch(h, C.byref(s.b), C.byref(s.m), C.byref(s.p))
    s.check(bool(p))
    coefs = s.handle.host_complex(p, (s.b.value, s.p.value, s.m.value))
    if s.call == "host":
        return coefs
    f = L.digHoloGetFields(h, C.byref(s.b), C.byref(s.p), C.byref(s.x), C.byref(s.y), C.byref(s.w), C.byref(s.ht))
    s.check(bool(f))
    return {"coefs": coefs, "fields": s.handle.host_complex(f, (s.b.value, s.p.value, s.ht.value, s.w.value))}


def work(case):
    """Window pixels read once; coefficients and the int16 fields (held for the field getters) written once.
    Operations: the R2C transform of every window's rows, the kept columns', the inverse, the overlap."""
    win, P, G = case["window"], case["pols"], case["groups"]
    kept = 16 * math.ceil(int(2 * math.hypot(1.0, 0.8) * case["carrier"] / 3.0 * win / 2 + 1) / 16)
    n = win if case["mode"] == 0 else kept
    units = case["frames"] * P
    M = G * (G + 1) // 2
    nbytes = units * (case["average"] * win * win * (2 if case["dtype"] == "uint16" else 4) + 8 * M + 4 * n * n)
    lg = math.log2(win)
    flops = units * case["average"] * (2.5 * win * win * lg + 5 * kept * win * lg)
    flops += units * (5 * kept * n * math.log2(n) + 5 * n * n * math.log2(n) + 4 * n * n * G + 4 * n * M)
    if case["call"] == "view":
        nbytes += units * 8 * n * n
    if case["call"] == "gradient":       # the adjoint field, three fields' contractions
        nbytes += units * 4 * n * n
        flops += units * (3 * 5 * n * n * math.log2(n) + 4 * (4 * n * n * G + 4 * n * M))
    if case["call"] == "metrics":
        flops += 8 * case["frames"] * (P * M) ** 2 + 16 / 3 * (P * M) ** 3
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ 64 bits

F = np.float32
PI32 = F(math.pi)
RAD = F(PI32 / F(180.0))


def half_away(v):
    return math.floor(v + 0.5) if v >= 0 else -math.floor(-v + 0.5)


class Exact:
    """The reconstruction in 64 bits with nothing quantised.  Placing the windows, and the tests of which
    Fourier pixels they hold, are single-precision arithmetic by definition."""

    def __init__(self, case, seed):
        self.s = s = Settings(case, seed)
        self.case = case
        self.frames = camera_frames(case, seed)
        self.dev = self.frames.device
        n, W, H = case["window"], case["width"], case["height"]
        self.n, self.P = n, case["pols"]
        p32 = F(PIXEL)
        self.cx, self.cy = [], []
        for p in range(self.P):
            X = F(F(F(s.beam_centre[p][0]) / p32) + F(W // 2))
            Y = F(F(F(s.beam_centre[p][1]) / p32) + F(H // 2))
            x = half_away(float(F(F(X - F(n // 2)) / F(16)))) * 16
            y = half_away(float(F(Y - F(n // 2))))
            self.cx.append(min(max(x, 0), W - n))
            self.cy.append(min(max(y, 0), H - n))
        dk = F(2 * (2.0 * math.pi / float(F(2.0 * float(p32)))) / n)
        self.dk = float(dk)
        self.k = np.array([F(dk) * F(i if i <= n // 2 else i - n) for i in range(n)], dtype=F)
        k0 = F(F(2) * PI32 / F(WAVELENGTH))
        r = F(F(s.window_radius_deg) * RAD)
        self.tilt = [[F(F(t) * RAD) for t in s.tilt_deg[p]] for p in range(self.P)]
        ends, sides = [], []
        for p in range(self.P):
            e = [[F(float(F(F(F(t + sgn * r) * k0) / F(self.k[1] - self.k[0]))) + n / 2.0) for sgn in (1, -1)] for t in self.tilt[p]]
            ends.append([half_away(float(F(a + b)) / 4.0) * 2 for a, b in e])
            sides.append([16 * math.ceil(int(F(F(a - b) + F(1))) / 16) for a, b in e])
        self.w = max(16, max(v[0] for v in sides))
        self.h = max(16, max(v[1] for v in sides))
        self.SX = [min(max(int(ends[p][0] - self.w / 2.0), n // 2), n - self.w) for p in range(self.P)]
        self.SY = [int(ends[p][1] - self.h / 2.0) for p in range(self.P)]
        self.mask, self.rows, self.cols = [], [], []
        kr = F(k0 * F(math.sin(float(r))))
        for p in range(self.P):
            kx0, ky0 = (F(k0 * F(math.sin(float(t)))) for t in self.tilt[p])
            j = np.arange(self.h) + self.SY[p]
            rows, cols = (j + n // 2) % n, np.arange(self.w) + self.SX[p] - n // 2
            turn = F(abs(float(F(self.k[1] - self.k[0])) * n))
            shift = np.where(j < 0, turn, np.where(j > n, -turn, F(0))).astype(F)
            dy = (self.k[rows] - (ky0 + shift)).astype(F)
            dx = (self.k[cols] - kx0).astype(F)
            self.mask.append(((dx * dx)[None, :] + (dy * dy)[:, None]).astype(F) <= F(kr * kr))
            self.rows.append(rows)
            self.cols.append(cols)
        self.full = case["mode"] == 0
        self.nx, self.ny = (n, n) if self.full else (self.w, self.h)

    def t(self, v):
        return torch.as_tensor(np.asarray(v, dtype=np.float64), device=self.dev)

    def windows(self, p, f0, f1):
        """Masked, normalised Fourier windows (no beam-centre phase) of frames f0..f1."""
        n, case = self.n, self.case
        f = self.frames[f0:f1, self.cy[p]:self.cy[p] + n, self.cx[p]:self.cx[p] + n].double()
        rows, cols = (torch.as_tensor(v, device=self.dev) for v in (self.rows[p], self.cols[p]))
        F2 = torch.fft.rfft2(f)[:, rows][:, :, cols]
        length = n * n if self.full else self.w * self.h
        sinc = [np.where(a == 0, 1.0, a / np.where(a == 0, 1.0, np.sin(a)))
                for a in (self.k[v].astype(np.float64) * 0.5 * float(F(PIXEL)) for v in (self.rows[p], self.cols[p]))]
        F2 = F2 * self.t(self.mask[p] * sinc[0][:, None] * sinc[1][None, :] / math.sqrt(float(n * n) * length))
        A = case["average"]
        if A == 1:
            return F2
        F2 = F2.reshape(-1, A, self.h, self.w)
        acc = F2[:, 0] / A
        for k in range(1, A):
            c = (acc * F2[:, k].conj()).sum(dim=(1, 2), keepdim=True)
            acc = acc + F2[:, k] * (c / c.abs()) / A
        return acc

    def axis(self, size):
        step = F(PIXEL) if self.full else F(F(F(PIXEL) * F(self.n)) / F(size))
        return np.array([F(i - size // 2) * F(step) for i in range(size)], dtype=F).astype(np.float64)

    def settings(self):
        """The alignment parameters as the library holds them (single precision)."""
        s = self.s
        return {"tilt": [[float(F(v)) for v in s.tilt_deg[p]] for p in range(self.P)],
                "centre": [[float(F(v)) for v in s.beam_centre[p]] for p in range(self.P)],
                "defocus": [float(F(v)) for v in s.defocus], "waist": float(F(s.waist[0]))}

    def field(self, p, win, q):
        """-conj(A ref) of one polarisation's windows for the alignment q."""
        n = self.n
        kx, ky = (self.t(self.k[v]) for v in (self.cols[p], self.rows[p]))
        x0 = (self.cx[p] + n // 2 - self.case["width"] // 2) * float(F(PIXEL))
        y0 = (self.cy[p] + n // 2 - self.case["height"] // 2) * float(F(PIXEL))
        ph = torch.exp(1j * (ky * (q["centre"][p][1] - y0)))[:, None] * torch.exp(1j * (kx * (q["centre"][p][0] - x0)))[None, :]
        win = win * ph
        if self.full:
            big = torch.zeros((win.shape[0], n, n), dtype=torch.complex128, device=self.dev)
            r, c = (torch.as_tensor(v, device=self.dev) for v in (self.rows[p], self.cols[p] % n))
            big[:, r[:, None], c[None, :]] = win
            win = big
        E = torch.fft.ifft2(win, norm="forward")
        k0 = 2.0 * math.pi / float(F(WAVELENGTH))
        focal = -math.pi * q["defocus"][p] / float(F(WAVELENGTH))
        wave = []
        for a, size in ((0, self.nx), (1, self.ny)):
            off = 0.0 if self.full else ((self.SX[p], self.SY[p])[a] - n / 2.0) * float(F(self.k[1] - self.k[0]))
            t = math.radians(1.0) * q["tilt"][p][a]
            r = self.t(self.axis(size))
            wave.append(torch.exp(1j * ((-k0 * t + off) * r - k0 * t * q["centre"][p][a] + focal * r * r)))
        return -(E * wave[1][:, None] * wave[0][None, :]).conj()

    def coefs(self, p, V, q):
        G = self.case["groups"]
        m, n = (torch.tensor(v, device=self.dev) for v in zip(*hg_indices(G)))
        hs = []
        for size in (self.nx, self.ny):
            r = self.t(self.axis(size))
            dx = float(abs(r[-1] - r[0])) / (size - 1)
            hs.append(hermite_gauss(math.sqrt(2) * r / q["waist"], G) * math.sqrt(dx / q["waist"]) * 2.0 ** 0.25)
        c = hs[1].to(torch.complex128) @ V @ hs[0].T.to(torch.complex128)
        return c[:, n, m]

    def chunks(self):
        n, A = self.case["frames"], self.case["average"]
        step = max(1, (1 << 24) // (self.n * self.n * A))
        return [(b, min(n, b + step)) for b in range(0, n, step)]

    def batch(self, q, fields=False):
        A = self.case["average"]
        cs, vs = [], []
        for b0, b1 in self.chunks():
            row, fl = [], []
            for p in range(self.P):
                V = self.field(p, self.windows(p, b0 * A, b1 * A), q)
                row.append(self.coefs(p, V, q))
                fl.append(V if fields else None)
            cs.append(torch.stack(row, 1))
            if fields:
                vs.append(torch.stack(fl, 1))
        return torch.cat(cs), torch.cat(vs) if fields else None

    def gradient(self):
        """IL = 10 log10 sum |c|^2 and its central differences in every alignment parameter, the Fourier-window
        selection held; the waist is one parameter of both polarisations."""
        base = self.settings()
        power = [0.0] * self.P
        names = [(k, a) for k in ("tilt", "centre") for a in (0, 1)] + [("defocus", 0), ("waist", 0)]
        step = {"tilt": 2e-5, "centre": 2e-8, "defocus": 2e-4, "waist": 2e-8}
        place = {("tilt", 0): 0, ("tilt", 1): 1, ("defocus", 0): 2, ("centre", 0): 3, ("centre", 1): 4, ("waist", 0): 5}
        moved = {}
        for b0, b1 in self.chunks():
            for p in range(self.P):
                win = self.windows(p, b0, b1)
                power[p] += float((self.coefs(p, self.field(p, win, base), base).abs() ** 2).sum())
                for key in names:
                    for sgn in (1, -1):
                        q = {k: [list(v) if isinstance(v, list) else v for v in x] if isinstance(x, list) else x for k, x in base.items()}
                        d = sgn * step[key[0]]
                        if key[0] == "waist":
                            q["waist"] += d
                        elif key[0] == "defocus":
                            q["defocus"][p] += d
                        else:
                            q[key[0]][p][key[1]] += d
                        moved[p, key, sgn] = moved.get((p, key, sgn), 0.0) + float((self.coefs(p, self.field(p, win, q), q).abs() ** 2).sum())
        total = sum(power)
        out = np.zeros(12)
        for p in range(self.P):
            for key in names:
                g = 10.0 / math.log(10.0) * (moved[p, key, 1] - moved[p, key, -1]) / (2 * step[key[0]]) / total
                out[(0 if key[0] == "waist" else 6 * p) + place[key]] += g
        return {"gradient": out, "il": 10.0 * math.log10(total)}


def exact(case, seed):
    """What run() returns, in 64 bits."""
    e = Exact(case, seed)
    if case["call"] == "gradient":
        return e.gradient()
    q = e.settings()
    c, v = e.batch(q, case["call"] == "view")
    if case["call"] == "view":
        return {"coefs": c.cpu().numpy(), "fields": v.cpu().numpy()}
    if case["call"] == "metrics":
        s2 = torch.linalg.svdvals(c.reshape(c.shape[0], -1)) ** 2
        return {"coefs": c, "il": 10.0 * math.log10(float(s2.mean())), "mdl": 10.0 * math.log10(float(s2.min() / s2.max()))}
    return c
