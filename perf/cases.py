"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the package's public entry points: the Python front end (`engine.Series`, `psf`, `fno`) or
the C ABI of `include/*.h` where a host program calls that directly.  Sizes are those of the benchmark's workloads,
the tests and the command line defaults, or lie in the ranges the headers state.

A case is a dict of plain values; "kind" selects one of

  series   the frame loop: (wavelength, direction) instances propagated through frozen-flow layers
  fresnel  one Fresnel hop of a complex field on the device (allocating or allocation-free entry point)
  fft      one unnormalised 2-D transform on the device
  expo     an exposure PSF accumulated from device frames
  chromat  the chromatic PSF of a pupil (host buffers)
  screen   master-screen synthesis (host buffers)
  infer    surrogate inference from layer windows to amplitude and phase
  train    one surrogate training pass: forward, loss, gradients
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

ARCSEC = math.pi / 180.0 / 3600.0
LAM_REF = 0.5e-6
PUPIL = 0.01
DT = 0.001
BIN = 100.0
SEEING = LAM_REF / 0.15 / ARCSEC      # r0 = 15 cm at the reference wavelength
ALT = [0.0, 500.0, 1000.0, 2000.0, 4000.0, 8000.0, 16000.0, 3000.0, 6000.0, 12000.0]
CN2 = [0.45, 0.15, 0.10, 0.10, 0.08, 0.07, 0.05, 0.06, 0.05, 0.04]
REF, SCI, PHASE = 0, 1, 2


def listed():
    return [
        # one 256^2 frame per call, one turbulent layer, as a real-time loop asks for it: the smallest series call
        series("rt_frame_256", n="256", crop=256, layers=1, master=1024, lam_lo=1.6e-6, sink="dev"),
        # four wavelengths of one direction at 512^2 through seven layers, frames delivered to pinned host buffers:
        # an ordinary simulation run
        series("multilayer_512", n="512", crop=512, nlam=4, lam_lo=0.5e-6, lam_hi=2.2e-6, steps=8, sink="host"),
        # 16 wavelengths x 9 directions on mixed grids, frames left on the device: the benchmark's workload
        series("batched_mixed", n="256,512,1024", crop=0, nlam=16, ndir=9, lam_lo=0.5e-6, lam_hi=2.4e-6, steps=2,
               sink="none"),
        # the largest grid, cropped to a ragged size, with a per-layer phase multiplier and a reference-wavelength
        # instance beside the science one
        series("large_2048_crop", n="2048", crop=1803, lam_lo=1.65e-6, master=4096, ref=True, vary=True, sink="dev"),
        # geometric phases only (WAVEFRONT_AMPLITUDE 0) for a fan of directions: tomography and guide-star fields
        series("phase_only_fan", n="512", crop=512, nlam=1, ndir=16, lam_lo=0.8e-6, layers=10, steps=4, amp=0,
               sink="dev"),
        # one hop of a 256^2 field inside a control loop that may not allocate
        {"name": "fresnel_noalloc_256", "kind": "fresnel", "n": 256, "entry": "noalloc"},
        # the transform behind the largest master screens
        {"name": "fft2d_8192", "kind": "fft", "n": 8192, "sign": -1},
        # a 64-frame exposure of 512^2 frames under one pupil
        {"name": "expo_512x64", "kind": "expo", "w": 512, "frames": 64, "per_frame": False},
        # a broad-band PSF
        {"name": "chromat_512", "kind": "chromat", "n": 512, "steps": 40, "apo": 0.0},
        # the master screens of a simulation are made one call per pair
        {"name": "screen_2048", "kind": "screen", "m": 2048},
        # the surrogate in place of the propagation, a batch of 256^2 frames
        {"name": "infer_16", "kind": "infer", "batch": 16},
        # one optimiser step's forward and backward at the default training batch
        {"name": "train_8", "kind": "train", "batch": 8},
    ]


def series(name, *, n, crop, nlam=1, ndir=1, lam_lo=0.5e-6, lam_hi=0.0, layers=7, master=2048, steps=1, amp=1,
           ref=False, vary=False, sink="dev"):
    c = {"kind": "series", "n": n, "crop": crop, "nlam": nlam, "ndir": ndir, "lam_lo": lam_lo,
         "lam_hi": lam_hi or lam_lo, "layers": layers, "master": master, "steps": steps, "amp": amp, "ref": ref,
         "vary": vary, "sink": sink}
    return dict(c, name=name) if name else c


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["series"] * 5 + ["fresnel", "fft", "expo", "chromat", "screen", "infer", "train"])
    if kind == "series":
        n = rng.choice([64, 128, 256, 256, 512, 512, 1024, 1024, 2048])
        crop = rng.choice([n, n, rng.randint(n // 2, n), 4 * rng.randint(n // 8, n // 4)])
        amp = rng.choice([1, 1, 1, 0])
        ndir = max(1, min(int(log(1, 24)), (24 << 20) // (n * n)))
        nlam = max(1, min(int(log(1, 17)), (24 << 20) // (n * n * ndir)))
        lo = log(0.5e-6, 2.0e-6) if n < 2048 else 1.65e-6
        return series("", n=str(n), crop=crop, nlam=nlam, ndir=ndir, lam_lo=lo, lam_hi=max(lo, log(0.8e-6, 2.4e-6)),
                      layers=rng.randint(1, 10), master=rng.choice([1024, 2048, 4096]) if n < 1024 else 4096,
                      steps=rng.randint(1, 4), amp=amp, ref=n <= 256 and rng.random() < 0.3, vary=rng.random() < 0.4,
                      sink=rng.choice(["dev", "dev", "host", "none"]))
    if kind == "fresnel":
        entry = rng.choice(["noalloc", "dev"])
        return {"kind": "fresnel", "n": rng.choice([64, 128, 256, 512] + ([1024, 2048] if entry == "dev" else [])),
                "entry": entry}
    if kind == "fft":
        return {"kind": "fft", "n": rng.choice([64, 128, 256, 512, 1024, 2048, 4096, 8192]), "sign": rng.choice([-1, 1])}
    if kind == "expo":
        w = rng.choice([32, 64, 128, 256, 512, 1024])
        return {"kind": "expo", "w": w, "frames": max(1, int(log(1, min(300, (16 << 20) // (w * w))))),
                "per_frame": rng.random() < 0.5}
    if kind == "chromat":
        return {"kind": "chromat", "n": rng.choice([64, 128, 256, 512]), "steps": rng.randint(3, 40),
                "apo": rng.choice([0.0, 0.35, 1.0])}
    if kind == "screen":
        return {"kind": "screen", "m": rng.choice([128, 256, 512, 1024, 2048])}
    return {"kind": kind, "batch": rng.randint(1, 16 if kind == "infer" else 8)}


# ---------------------------------------------------------------------------
# inputs that a user's program has in hand
# ---------------------------------------------------------------------------
def gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + salt)


def kolmogorov(count, M, seed, outer=2000.0):
    """Periodic von Karman screens (float32, unit-ish scale) from seeded noise."""
    f = torch.fft.fftfreq(M, device="cuda", dtype=torch.float64) * M
    r2 = f[:, None] ** 2 + f[None, :M // 2 + 1] ** 2 + (M / outer) ** 2
    a = r2 ** (-11.0 / 12.0)
    a[0, 0] = 0.0
    a = a.float()
    g = gen(seed, 1)
    out = []
    for _ in range(count):
        z = torch.randn((M, M // 2 + 1, 2), device="cuda", generator=g)
        out.append(torch.fft.irfft2(torch.view_as_complex(z) * a, s=(M, M)).mul_(M * M / 4.0).contiguous())
    return out


def wave(count, n, seed, rms):
    """Turbulent phases of about `rms` radians, [count][n][n]."""
    m = min(2048, max(256, 2 * n))
    s = kolmogorov(min(count, 4), m, seed)
    out = torch.empty((count, n, n), device="cuda")
    for k in range(count):
        p = torch.roll(s[k % len(s)], shifts=(37 * k, 61 * k), dims=(0, 1))[:n, :n]
        p = p - p.mean()
        out[k] = p * (rms / p.std())
    return out


def series_setup(case, seed):
    """Profile, winds, directions and instances of a series case."""
    rng = np.random.default_rng(int(seed))
    L = case["layers"]
    if L == 1:
        # one turbulent layer over a Cn2 = 0 layer at the ground, so that the field is propagated to the ground
        alt, cn2 = [0.0, 5000.0], [0.0, 1.0]
    else:
        order = sorted(range(L), key=lambda k: ALT[k])
        alt, cn2 = [ALT[k] for k in order], [CN2[k] for k in order]
    speed = [float(v) for v in rng.uniform(5.0, 30.0, len(alt))]
    direction = [float(v) for v in rng.uniform(0.0, 2 * np.pi, len(alt))]
    side = math.ceil(math.sqrt(case["ndir"]))
    dirs = [((k % side - (side - 1) / 2) * 10 * ARCSEC, (k // side - (side - 1) / 2) * 10 * ARCSEC)
            for k in range(case["ndir"])]
    nl = case["nlam"]
    lams = [case["lam_lo"] * (case["lam_hi"] / case["lam_lo"]) ** (k / max(1, nl - 1)) for k in range(nl)]
    grids = [int(v) for v in case["n"].split(",")]
    sizes = np.random.default_rng(0).choice(grids, size=nl * len(dirs))
    inst = []
    if case["ref"]:
        inst.append((LAM_REF, REF, dirs[0], int(sizes[0])))
    k = 0
    for d in dirs:
        for lam in lams:
            inst.append((float(lam), SCI, d, int(sizes[k])))
            k += 1
    out = []
    for lam, mode, d, n in inst:
        sc = np.full(len(alt), np.float32(LAM_REF / lam), np.float32)
        if case["vary"]:
            sc = (sc * (1.0 - 2e-3 * (1.0 - LAM_REF / lam) * np.exp(-np.asarray(alt) / 8000.0))).astype(np.float32)
        out.append({"lam": lam, "mode": mode if case["amp"] else PHASE, "src": d, "n": n,
                    "crop": case["crop"] or n, "sc": sc})
    return alt, cn2, speed, direction, out


class DeviceFrames:
    """The engine's own frame buffer, seen as a CUDA array; it holds the engine as long as a tensor holds it."""

    def __init__(self, series, ptr, n):
        self.series = series
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False), "version": 3}


def prepare_series(case, seed):
    from atmosphericturbulencesimul_gb300 import InstanceSpec, Series
    alt, cn2, speed, direction, inst = series_setup(case, seed)
    specs = [InstanceSpec(lam=I["lam"], mode=I["mode"], src_x=I["src"][0], src_y=I["src"][1], wf_raw_size=I["n"],
                          wf_size=I["crop"], scoeff=I["sc"]) for I in inst]
    M = case["master"]
    s = Series(alt, cn2, speed, direction, master_size=M, instances=specs, pupil_scale=PUPIL, time_step=DT,
               fresnel_bin=BIN, amplitude=case["amp"], fresnel=1, ring=2 if case["sink"] == "host" else 1)
    screens = kolmogorov(len(alt), M, seed)
    torch.cuda.synchronize()
    for l, scr in enumerate(screens):
        s.load_screen_dev(l, scr.data_ptr(), M)
    s.normalize(np.float32(LAM_REF), np.float32(SEEING))
    s.run(0)   # the run's plan: windows, tile shapes, the step's graph
    state = {"case": case, "series": s, "frames": sum(I["crop"] ** 2 for I in inst)}
    shape = (case["steps"], state["frames"])
    if case["sink"] == "host":
        state["pha"], state["amp"] = (torch.empty(shape, pin_memory=True) for _ in range(2))
    elif case["sink"] == "dev":
        state["pha"], state["amp"] = (torch.empty(shape, device="cuda") for _ in range(2))
    return state


def run_series(state):
    case, s = state["case"], state["series"]
    if case["sink"] == "none":
        s.run(case["steps"])
        if "pha" not in state:
            state["pha"], state["amp"] = (torch.as_tensor(DeviceFrames(s, p, state["frames"]), device="cuda")
                                          for p in s.frame_dev(0))
    else:
        s.run(case["steps"], pha_ptr=state["pha"].data_ptr(), amp_ptr=state["amp"].data_ptr())
    return {"pha": state["pha"], "amp": state["amp"]}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "series":
        return prepare_series(case, seed)
    from atmosphericturbulencesimul_gb300 import _lib
    st = {"case": case, "lib": _lib.load()}
    if kind == "fresnel":
        # a pupil field after some propagation: amplitude around one, phase of a few radians
        n = case["n"]
        p = wave(2, n, seed, 3.0)
        st["in"] = torch.polar(1.0 + 0.1 * torch.tanh(p[1]), p[0]).contiguous()
        st["out"] = torch.empty_like(st["in"])
    elif kind == "fft":
        n = case["n"]
        st["in"] = torch.view_as_complex(torch.randn((n, n, 2), device="cuda", generator=gen(seed)))
        st["out"] = torch.empty_like(st["in"])
    elif kind == "expo":
        w = case["w"]
        st["pha"] = wave(case["frames"], w, seed, 1.5)
        r = torch.linspace(-1.0, 1.0, w, device="cuda")
        pupil = ((r[:, None] ** 2 + r[None, :] ** 2) < 0.96).float()
        st["amp"] = pupil if not case["per_frame"] else (
            pupil * (1.0 + 0.1 * torch.tanh(wave(case["frames"], w, seed + 1, 1.0)))).contiguous()
        st["acc"] = torch.empty((2 * w, 2 * w), device="cuda")
        st["img"] = torch.empty((2 * w, 2 * w), device="cuda")
    elif kind == "chromat":
        n = case["n"]
        r = torch.linspace(-1.0, 1.0, n, device="cuda")
        st["amp"] = ((r[:, None] ** 2 + r[None, :] ** 2) < 0.2).float().cpu().numpy()
        st["pha"] = wave(1, n, seed, 1.0)[0].cpu().numpy()
    elif kind == "screen":
        st["seed"] = int(seed)
    else:
        from atmosphericturbulencesimul_gb300 import fno as F
        st["F"] = F
        st["model"] = F.Surrogate(F.FnoConfig())
        st["model"].set_params(network(seed)[0].cpu().numpy())
        st.update(network_inputs(case, seed))
        if kind == "train":
            st["grads"] = torch.empty(st["model"].num_params, pin_memory=True)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "series":
        return run_series(st)
    lib = st["lib"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "fresnel":
        fn = lib.atmwfs_fresnel_noalloc if case["entry"] == "noalloc" else lib.atmwfs_fresnel_dev
        ok(fn(st["in"].data_ptr(), st["out"].data_ptr(), case["n"], PUPIL, 4000.0, 1.65e-6, stream))
        return st["out"]
    if kind == "fft":
        ok(lib.atmwfs_fft2d_dev(st["in"].data_ptr(), st["out"].data_ptr(), case["n"], case["sign"], stream))
        return st["out"]
    if kind == "expo":
        from atmosphericturbulencesimul_gb300 import psf
        st["acc"].zero_()
        psf.expo_accumulate_dev(st["pha"], st["amp"], st["acc"], stream)
        psf.expo_image_dev(st["acc"], st["img"], stream)
        return st["img"]
    if kind == "chromat":
        from atmosphericturbulencesimul_gb300 import psf
        return psf.chromat_psf(st["amp"], st["pha"], 0.8, 1.25, case["steps"], case["apo"])
    if kind == "screen":
        from atmosphericturbulencesimul_gb300 import master_screen
        o1, o2, c = master_screen(st["seed"], case["m"], 20.0 / PUPIL, 0.01 / PUPIL)
        return [o1, o2, c]
    F, model = st["F"], st["model"]
    if kind == "infer":
        x, phi = F.prepare(st["win"], st["lam"], stream)
        out = model.forward(x, stream=stream)
        amp, pha = F.assemble(out, phi, stream)
        return {"out": out, "amp": amp, "pha": pha}
    model.zero_grads(stream)
    out = torch.empty((case["batch"], 2, 256, 256), device="cuda")
    loss = model.loss_grad(st["x"], st["target"], out, stream)
    ok(lib.atmwfs_fno_get_grads(model._h, C.cast(st["grads"].data_ptr(), C.POINTER(C.c_float))))
    return {"out": out, "loss": loss, "grads": st["grads"]}


def ok(status):
    if status:
        raise RuntimeError(f"status {status}")


# ---------------------------------------------------------------------------
# the surrogate's parameters and inputs
# ---------------------------------------------------------------------------
NIN, W, MODES, LAYERS, PROJ, NOUT, G = 8, 64, 32, 4, 128, 2, 256


def network(seed):
    """A parameter vector in the library's order (and its pieces), of the size training reaches: spectral weights
    that carry a few percent of a layer's output, pointwise weights of order 1 / sqrt(fan in)."""
    g = gen(seed, 5)

    def uni(*shape, s):
        return (torch.rand(shape, device="cuda", generator=g) * 2 - 1) * s

    p = {"lift_W": uni(W, NIN, s=NIN ** -0.5), "lift_b": uni(W, s=0.05)}
    for l in range(LAYERS):
        p[f"R{l}"] = uni(MODES * MODES, W, W, 2, s=8.0 / W ** 2)
        p[f"W{l}"] = uni(W, W, s=W ** -0.5)
        p[f"b{l}"] = uni(W, s=0.05)
    p |= {"proj1_W": uni(PROJ, W, s=W ** -0.5), "proj1_b": uni(PROJ, s=0.05),
          "proj2_W": uni(NOUT, PROJ, s=PROJ ** -0.5), "proj2_b": uni(NOUT, s=0.02)}
    return torch.cat([v.reshape(-1) for v in p.values()]), p


def network_inputs(case, seed):
    B = case["batch"]
    win = wave(B * (NIN - 1), G, seed + 3, 2.0).reshape(B, NIN - 1, G, G)
    lam = (0.5e-6 + 1.7e-6 * torch.rand(B, device="cuda", generator=gen(seed, 6)))
    if case["kind"] == "infer":
        return {"win": win, "lam": lam}
    x = torch.cat([win * 0.1, ((lam - 1.35e-6) / 0.5e-6).reshape(B, 1, 1, 1).expand(B, 1, G, G)], 1).contiguous()
    t = 0.2 * torch.tanh(wave(B * 2, G, seed + 4, 1.0)).reshape(B, 2, G, G)
    return {"x": x, "target": t.contiguous()}


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "series":
        _, _, _, _, inst = series_setup(case, 0)
        L = max(2, case["layers"])
        wins = {}
        for I in inst:
            wins[I["src"]] = max(wins.get(I["src"], 0), I["n"])
        # the screens under the windows read once, every frame written once
        b = sum(4.0 * L * n * n for n in wins.values()) + sum(8.0 * I["crop"] ** 2 for I in inst)
        # per hop a forward and an inverse 2-D transform and the transfer multiply; per layer the bicubic and phasor
        f = sum(I["n"] ** 2 * ((L - 1) * (20.0 * math.log2(I["n"]) + 6) * (1 if case["amp"] else 0) + 6.0 * L)
                for I in inst) + sum(40.0 * L * n * n for n in wins.values())
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind in ("fresnel", "fft"):
        n = case["n"]
        return {"bytes": 16.0 * n * n, "flops": n * n * (10.0 * math.log2(n)) * (2 if kind == "fresnel" else 1)}
    if kind == "expo":
        w, f = case["w"], case["frames"]
        n = 2 * w
        return {"bytes": 4.0 * w * w * (f + (f if case["per_frame"] else 1)) + 4.0 * n * n,
                "flops": f * (5.0 * n * w * math.log2(n) + 5.0 * n * n * math.log2(n) + 4.0 * n * n)}
    if kind == "chromat":
        n, s = case["n"], case["steps"]
        return {"bytes": 12.0 * n * n, "flops": s * n * n * (10.0 * math.log2(n) + 30.0)}
    if kind == "screen":
        m = case["m"]
        return {"bytes": 8.0 * m * m, "flops": m * m * (10.0 * math.log2(m) + 80.0)}
    B, P = case["batch"], G * G
    point = 2.0 * P * (W * NIN + LAYERS * W * W + PROJ * W + NOUT * PROJ)
    spec = LAYERS * (2 * 2.0 * W * G * G * 2 * MODES + 2 * 8.0 * W * MODES * MODES * G + 8.0 * W * W * MODES * MODES)
    params = LAYERS * MODES * MODES * W * W * 2.0
    if kind == "infer":
        return {"bytes": 4.0 * B * P * (NIN - 1 + NOUT + 2) + 2.0 * params, "flops": B * (point + spec)}
    return {"bytes": 4.0 * B * P * (NIN + 2 * NOUT) + 6.0 * params, "flops": 3.0 * B * (point + spec)}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def keys(t):
    return [0.5 * (-t ** 3 + 2 * t * t - t), 0.5 * (3 * t ** 3 - 5 * t * t + 2), 0.5 * (-3 * t ** 3 + 4 * t * t + t),
            0.5 * (t ** 3 - t * t)]


def window(S, x, y, n):
    """Keys bicubic samples of the periodic screen S at (x + i, y + j)."""
    M = S.shape[0]
    ix, iy = int(math.fmod(x, M)), int(math.fmod(y, M))
    wx, wy = keys(math.fmod(x, M) - ix), keys(math.fmod(y, M) - iy)
    k = torch.arange(-1, n + 2, device=S.device)
    t = S[(iy + k) % M][:, (ix + k) % M]
    h = sum(wx[a] * t[:, a:a + n] for a in range(4))
    return sum(wy[a] * h[a:a + n] for a in range(4))


def relax(pb):
    """The science unwrap's bin relaxation of the bin phases pb [nb][nb]."""
    nb = pb.shape[0]
    sweeps = [(1, 0, .2), (0, 1, .2), (1, 1, .2), (1, -1, .2), (2, 0, .15), (0, -2, .15), (-1, -2, .15), (1, -2, .15),
              (-2, -2, .15), (2, -2, .15), (2, -1, .15), (-2, -1, .15)]
    inner = np.zeros((nb, nb), bool)
    inner[2:nb - 2, 2:nb - 2] = True
    plim, it, quiet = 1.0, 0, 0
    while plim > 0.51 and it < 1000 and quiet < 5:
        it += 1
        ch = np.zeros((nb, nb))
        for dx, dy, c in sweeps:
            if abs(dx) >= nb or abs(dy) >= nb:
                continue
            y1, x1 = slice(max(0, -dy), nb - max(0, dy)), slice(max(0, -dx), nb - max(0, dx))
            y2, x2 = slice(max(0, dy), nb - max(0, -dy)), slice(max(0, dx), nb - max(0, -dx))
            d = pb[y2, x2] - pb[y1, x1]
            v = c * ((d > math.pi).astype(float) - (d < -math.pi))
            ch[y1, x1] += v
            ch[y2, x2] -= v
        plim = max(0.5, np.abs(ch).max() - 0.001)
        up, down = ch > plim, ch < -plim
        pb = pb + 2 * math.pi * (up.astype(float) - down)
        quiet = 0 if ((up | down) & inner).any() else quiet + 1
    return pb


def exact_series(case, seed):
    alt, cn2, speed, direction, inst = series_setup(case, seed)
    dx, dt, M, L = float(np.float32(PUPIL)), float(np.float32(DT)), case["master"], len(alt)
    scr = [s.double() for s in kolmogorov(L, M, seed)]
    # r0 renormalisation and the layers' Cn2 weights
    r0 = np.mean([50.0 * (float(((s[:, 50:] - s[:, :-50]) ** 2).mean()) / 6.88) ** -0.6 for s in scr])
    target = float(np.float32(LAM_REF)) / (float(np.float32(SEEING)) / 3600.0 / 180.0 * math.pi) / dx
    scr = [s * ((r0 / target) ** (5.0 / 6.0) * math.sqrt(c / sum(cn2))) for s, c in zip(scr, cn2)]
    steps = [case["steps"] - 1] if case["sink"] == "none" else list(range(case["steps"]))
    pha = torch.empty((len(steps), sum(I["crop"] ** 2 for I in inst)), dtype=torch.float64, device="cuda")
    amp = torch.empty_like(pha)
    wins, o = {}, 0
    side = {}
    for I in inst:
        side[I["src"]] = max(side.get(I["src"], 0), I["n"])
    for q, I in enumerate(inst):
        n, no, lam = I["n"], I["crop"], I["lam"]
        off = (n - no) // 2
        if not any(J["src"] == I["src"] for J in inst[:q]):
            wins = {}   # instances come direction by direction
        f = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * n
        for row, k in enumerate(steps):
            sc = [float(v) for v in I["sc"]]
            tot = torch.zeros((n, n), dtype=torch.float64, device="cuda")
            fld = torch.ones((n, n), dtype=torch.complex128, device="cuda")
            for l in range(L - 1, -1, -1):
                if (l, k) not in wins:
                    x = 0.05 * M + float(np.float32(I["src"][0])) * alt[l] / dx
                    y = 0.05 * M + float(np.float32(I["src"][1])) * alt[l] / dx
                    x += (k + 1) * (speed[l] * math.cos(direction[l]) / dx * dt)
                    y += (k + 1) * (speed[l] * math.sin(direction[l]) / dx * dt)
                    wins[l, k] = window(scr[l], x % M, y % M, side[I["src"]])
                p = wins[l, k][:n, :n] * sc[l]
                tot += p
                if case["amp"]:
                    fld = fld * torch.polar(torch.ones_like(p), p)
                    if l > 0:
                        c = math.pi * (alt[l] - alt[l - 1]) * lam / (dx * n) ** 2
                        hk = torch.polar(torch.ones_like(f), torch.remainder(-c * f * f, 2 * math.pi))
                        fld = torch.fft.ifft2(torch.fft.fft2(fld) * hk[:, None] * hk[None, :])
            tot = tot[off:off + no, off:off + no]
            fld = fld[off:off + no, off:off + no]
            if I["mode"] == PHASE:
                out, a = tot, torch.ones_like(tot)
            else:
                raw, a = torch.angle(fld), torch.abs(fld)
                peak = 0.0
                nb = no // 20 if I["mode"] == SCI else 0
                if nb > 0:
                    b = torch.tensor([int(1.0 * i / no * nb) for i in range(no)], device="cuda")
                    z = torch.polar(torch.ones_like(tot), tot - raw)
                    s = torch.zeros((nb, no), dtype=z.dtype, device="cuda").index_add_(0, b, z)
                    s = torch.zeros((nb, nb), dtype=z.dtype, device="cuda").index_add_(1, b, s)
                    pk = torch.from_numpy(relax(torch.angle(s).cpu().numpy())).cuda()
                    peak = pk[b][:, b]
                d = tot if I["mode"] == REF else tot - raw - peak
                out = raw + 2 * math.pi * torch.floor(d / (2 * math.pi) + 0.5)
            pha[row, o:o + no * no] = out.reshape(-1)
            amp[row, o:o + no * no] = a.reshape(-1)
        o += no * no
    if case["sink"] == "none":
        pha, amp = pha[0], amp[0]
    return {"pha": pha, "amp": amp}


def exact_network(x, p):
    """The network's output for x [B][NIN][G][G] with parameters p, in 64 bits."""
    def point(w, b, h):
        return torch.einsum("oc,bcyx->boyx", w, h) + b.reshape(1, -1, 1, 1)

    ky = torch.tensor([j if j < MODES // 2 else j - MODES for j in range(MODES)], device="cuda") % G
    h = point(p["lift_W"], p["lift_b"], x)
    for l in range(LAYERS):
        z = torch.fft.fft2(h)[:, :, ky][..., :MODES]
        R = torch.view_as_complex(p[f"R{l}"].contiguous()).reshape(MODES, MODES, W, W)
        y = torch.einsum("kqoc,bckq->bokq", R, z)
        y = torch.cat([y[..., :1], 2.0 * y[..., 1:]], -1)
        full = torch.zeros((x.shape[0], W, G, MODES), dtype=y.dtype, device="cuda").index_copy(2, ky, y)
        s = torch.fft.ifft2(torch.nn.functional.pad(full, (0, G - MODES))).real
        u = s + point(p[f"W{l}"], p[f"b{l}"], h)
        h = torch.nn.functional.gelu(u, approximate="tanh") if l + 1 < LAYERS else u
    q = torch.nn.functional.gelu(point(p["proj1_W"], p["proj1_b"], h), approximate="tanh")
    return point(p["proj2_W"], p["proj2_b"], q)


def philox(c0, c1, key):
    """Philox4x32-10 of counters (c0, c1, 0, 0), as uint64 arrays of 32-bit words."""
    u = np.uint64
    lo32, s32 = u(0xFFFFFFFF), u(32)
    c = [c0, np.full_like(c0, c1), np.zeros_like(c0), np.zeros_like(c0)]
    k = [key & 0xFFFFFFFF, (key >> 32) & 0xFFFFFFFF]
    for _ in range(10):
        a, b = u(0xD2511F53) * c[0], u(0xCD9E8D57) * c[2]
        c = [(b >> s32) ^ c[1] ^ u(k[0]), b & lo32, (a >> s32) ^ c[3] ^ u(k[1]), a & lo32]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return c


def exact(case, seed):
    kind = case["kind"]
    if kind == "series":
        return exact_series(case, seed)
    if kind == "screen":
        M = case["m"]
        c = philox(np.arange(M * M, dtype=np.uint64), 0, int(seed))
        r = [torch.from_numpy((v >> np.uint64(8)).astype(np.float64)).cuda().reshape(M, M) / 2 ** 24 for v in c[:3]]
        g = torch.sqrt(-2.0 * torch.log(r[1] + 2.0 ** -24)) * torch.cos(2 * math.pi * r[2])
        k = torch.arange(M, device="cuda", dtype=torch.float64) - M // 2
        r2 = k[:, None] ** 2 + k[None, :] ** 2
        fo, fi = M * PUPIL / 20.0, 5.92 / (2 * math.pi) * M * PUPIL / 0.01
        a = g * torch.exp(-r2 / (2 * fi * fi)) / (r2 + fo * fo) ** (11.0 / 12.0)
        a[M // 2, M // 2] = 0.0
        f = torch.fft.fft2(torch.fft.fftshift(torch.polar(torch.ones_like(a), 2 * math.pi * r[0]) * a))
        out, cs = [], []
        for part in (f.real, f.imag):
            v = [math.log10(float(((part - torch.roll(part, (-ly, -lx), (0, 1))) ** 2).mean()))
                 - 5.0 / 3.0 * math.log10(math.hypot(lx, ly)) for ly in (1, 2) for lx in (1, 2)]
            cs.append(10.0 ** (sum(v) / 4))
            out.append(part / math.sqrt(cs[-1]))
        return [out[0], out[1], np.array(cs)]
    if kind in ("infer", "train"):
        p = {k: v.double() for k, v in network(seed)[1].items()}
        i = {k: v.double() for k, v in network_inputs(case, seed).items()}
        if kind == "infer":
            lam = (i["lam"] - 1.35e-6) / 0.5e-6
            x = torch.cat([i["win"] * 0.1, lam.reshape(-1, 1, 1, 1).expand(-1, 1, G, G)], 1)
            out = exact_network(x, p)
            u = torch.complex(1.0 + out[:, 0], out[:, 1])
            return {"out": out, "amp": u.abs(), "pha": i["win"].sum(1) + u.angle()}
        p = {k: v.requires_grad_() for k, v in p.items()}
        out = exact_network(i["x"], p)
        loss = ((out - i["target"]) ** 2).mean()
        loss.backward()
        return {"out": out.detach(), "loss": float(loss), "grads": torch.cat([v.grad.reshape(-1) for v in p.values()])}
    st = prepare(case, seed) if kind != "chromat" else {k: torch.from_numpy(v).cuda() for k, v in prepare(case, seed).items()
                                                        if isinstance(v, np.ndarray)}
    if kind == "fft":
        a = st["in"].to(torch.complex128)
        return torch.fft.fft2(a) if case["sign"] < 0 else torch.fft.ifft2(a, norm="forward")
    if kind == "fresnel":
        n = case["n"]
        f = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * n
        ang = torch.remainder(-math.pi * 4000.0 * 1.65e-6 / (PUPIL * n) ** 2 * f * f, 2 * math.pi)
        hk = torch.polar(torch.ones_like(ang), ang)
        return torch.fft.ifft2(torch.fft.fft2(st["in"].to(torch.complex128)) * hk[:, None] * hk[None, :])
    if kind == "expo":
        w = case["w"]
        acc = torch.zeros((2 * w, 2 * w), dtype=torch.float64, device="cuda")
        for k in range(case["frames"]):
            a = st["amp"][k] if case["per_frame"] else st["amp"]
            z = torch.zeros((2 * w, 2 * w), dtype=torch.complex128, device="cuda")
            z[:w, :w] = torch.polar(a.double(), st["pha"][k].double())
            acc += torch.fft.fft2(z).abs() ** 2
        return torch.fft.fftshift(acc)
    # chromat: the step coefficients and weights are float values of the call
    n, steps, apo = case["n"], case["steps"], float(np.float32(case["apo"]))
    c1, c2 = float(np.float32(0.8)), float(np.float32(1.25))
    amp, pha = st["amp"].double(), st["pha"].double()
    out = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    k = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    for s in range(steps):
        c = float(np.float32(c1 * (float(np.float32(np.float32(c2) / np.float32(c1))) ** (1.0 / (steps - 1))) ** s))
        x = (c - (c1 + c2) / 2.0) / ((c2 - c1) / 2.0)
        m = (1.0 - ((abs(x) - (1.0 - apo)) / apo) ** 2) ** 4 if apo > 1e-5 else 1.0
        m = 0.0 if 1.0 - x * x < 1e-5 else m
        m = 1.0 if abs(x) < apo else m
        img = torch.fft.fftshift(torch.fft.fft2(torch.polar(amp, c * pha)).abs() ** 2)
        pos = k * c + n // 2
        i = torch.trunc(pos)
        inside = (i < n - 1) & (i > -1)
        i = i.clamp(0, n - 2).long()
        u = (pos - i) * inside
        cols = img[:, i] * (1 - u) + img[:, i + 1] * u
        z = cols[i] * (1 - u)[:, None] + cols[i + 1] * u[:, None]
        out += m * z * inside[:, None] * inside[None, :] / c / c
    return out
