"""The work that the engine's performance is judged on: image formation calls of a localisation-microscopy user, from
one previewed frame to a whole two-colour movie, with the PSF libraries, widefield focus series, binned frames and
likelihood gradients around them. Each case goes through the package's public entry points only.

A case is a plain dict; prepare() makes what a program holds before the call (inputs from the seed alone, the engine,
its kernel stacks, camera maps and plans), run() is one call, exact() the float64 value of what it computes, from the
documented model and without the package's code. Kernel stacks are handed to the engine as sampled planes (as a measured
PSF would be), so that the frames of a case depend on its inputs alone.
"""
import math

import numpy as np
import torch

from insiliscope_b200.engine import (BLINK_EVENT_DTYPE, CZT_F16X3, CZT_FP32, EMITTER_DTYPE, FRAME_DTYPE, INTERP_CUBIC,
                                     INTERP_LINEAR, INTERP_NEAREST, BinnedRenderer, CameraParams, Engine, PsfParams,
                                     PsfPlan, WidefieldPlan)
from insiliscope_b200.nll import NllModel, NllSpec, poisson_nll

DEV = "cuda:0"
PIXEL_NM = 108.0
INTERP = {"cubic": INTERP_CUBIC, "linear": INTERP_LINEAR, "nearest": INTERP_NEAREST}
TWO_PI = 2.0 * math.pi


# ------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # One previewed frame of a small window: what a user waits for on every change of a setting. Expected image and
        # camera frame, the engine's default render form.
        {"name": "snap_frame", "kind": "render", "frames": 1, "width": 64, "height": 64, "per_frame": 40,
         "uneven": 0.0, "colours": 1, "half": 8, "os": 4, "nz": 25, "interp": "cubic", "form": 0, "photons": True,
         "emccd": False},
        # The plain dSTORM movie of the benchmark: 200 camera frames of 128 x 128, about 160 emitters on in each, with
        # the form that the autotuner takes for it.
        {"name": "dstorm_movie", "kind": "render", "frames": 200, "width": 128, "height": 128, "per_frame": 160,
         "uneven": 0.0, "colours": 1, "half": 16, "os": 4, "nz": 49, "interp": "cubic", "form": 14, "photons": False,
         "emccd": False},
        # The largest movie: 1,024 frames of 256 x 256, two dye groups, emitter counts heavy-tailed over the frames.
        {"name": "two_colour_movie", "kind": "render", "frames": 1024, "width": 256, "height": 256, "per_frame": 300,
         "uneven": 1.0, "colours": 2, "half": 16, "os": 4, "nz": 49, "interp": "cubic", "form": 14, "photons": False,
         "emccd": False},
        # Blink events on the host to EMCCD frames on the host, an odd window with drift, an illumination profile,
        # linear interpolation and the halo cut: one call of the whole path.
        {"name": "events_ragged", "kind": "events", "frames": 60, "width": 131, "height": 97, "per_frame": 90,
         "half": 12, "os": 3, "nz": 33, "interp": "linear", "emccd": True},
        # The camera's noise on expected images that come from elsewhere (a stack of half-megapixel sCMOS frames).
        {"name": "noise_stack", "kind": "noise", "frames": 16, "width": 512, "height": 512, "emccd": False},
        # The PSF stack of one optical setting, as made when an aberration or the depth changes: 49 planes of 129 x 129.
        {"name": "psf_stack", "kind": "psf", "half": 16, "os": 4, "nz": 49, "pupil": 64, "modes": 12,
         "depth_nm": 400.0},
        # The benchmark's PSF library on its tensor-core plan: 64 planes x 4 wavelengths x 16 aberrations.
        {"name": "psf_library", "kind": "library", "sets": 64, "planes": 64, "pupil": 128, "size": 64},
        # A focus series of a thick specimen at the benchmark's size, with the EMCCD camera.
        {"name": "widefield_series", "kind": "series", "nx": 512, "ny": 512, "nz": 64, "stack": 65, "half": 256},
        # The expected images of a small odd specimen under a measured 3D PSF (no camera).
        {"name": "widefield_ragged", "kind": "widefield", "nx": 186, "ny": 151, "nz": 11, "kx": 61, "ky": 61,
         "kz": 9},
        # One step of a maximum-likelihood fit at the benchmark's size: likelihood and gradients of 256,000 ROIs.
        {"name": "fit_large", "kind": "fit", "frames": 256, "per_frame": 1000, "roi": 32},
        # The same step for the few ROIs of a live fit.
        {"name": "fit_live", "kind": "fit", "frames": 4, "per_frame": 25, "roi": 32},
        # Dense frames in the binned regime, two cells per pixel, with the EMCCD camera.
        {"name": "binned_dense", "kind": "binned", "frames": 200, "width": 128, "height": 128, "per_frame": 2400,
         "half": 16, "os": 4, "nz": 49, "upscale": 2},
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "events", "noise", "psf", "library", "series", "widefield", "fit",
                       "fit", "binned"])
    c = {"kind": kind}
    if kind in ("render", "events"):
        w, h = _log(rng, 32, 256), _log(rng, 32, 256)
        half, os = rng.randint(4, 16), rng.choice([2, 3, 4])
        # the pixels of all frames and the emitters' squares stay within the large movie's
        frames = _log(rng, 1, 1024)
        per = _log(rng, 1, max(1.0, min(0.025 * w * h, 300.0)))
        c.update(frames=frames, width=w, height=h, per_frame=per, half=half, os=os, nz=rng.randint(2, 24) * 2 + 1,
                 interp=rng.choice(["cubic", "cubic", "cubic", "linear", "nearest"]), emccd=rng.random() < 0.3)
        if kind == "events":
            c.update(frames=min(frames, 200))
        else:
            c.update(uneven=rng.choice([0.0, 0.0, 1.0]), colours=rng.choice([1, 1, 2]),
                     form=rng.choice([0, 12, 14, 14, 14]), photons=rng.random() < 0.4)
    elif kind == "noise":
        c.update(frames=_log(rng, 1, 16), width=_log(rng, 32, 512), height=_log(rng, 32, 512),
                 emccd=rng.random() < 0.4)
    elif kind == "psf":
        c.update(half=rng.randint(4, 16), os=rng.randint(1, 4), nz=rng.randint(1, 24) * 2 + 1,
                 pupil=rng.choice([32, 48, 64, 64, 100, 128]), modes=rng.choice([0, 3, 12]),
                 depth_nm=rng.choice([0.0, 400.0]))
    elif kind == "library":
        c.update(sets=_log(rng, 1, 64), planes=_log(rng, 1, 64), pupil=rng.choice([64, 96, 128]),
                 size=rng.choice([32, 48, 57, 64]))
    elif kind == "series":
        half = rng.randint(16, 128)
        c.update(nx=2 * _log(rng, 32, 192), ny=_log(rng, 64, 384), nz=_log(rng, 4, 48), stack=2 * rng.randint(2, 20) + 1,
                 half=half)
    elif kind == "widefield":
        c.update(nx=2 * _log(rng, 20, 150), ny=_log(rng, 40, 300), nz=_log(rng, 1, 32), kx=rng.randint(3, 80),
                 ky=rng.randint(3, 80), kz=rng.randint(1, 16))
    elif kind == "fit":
        c.update(frames=_log(rng, 1, 128), per_frame=_log(rng, 1, 1000), roi=rng.choice([16, 32, 32, 32, 64]))
    else:
        c.update(frames=_log(rng, 1, 200), width=_log(rng, 48, 128), height=_log(rng, 48, 128),
                 per_frame=_log(rng, 60, 2400), half=rng.randint(6, 16), os=4, nz=rng.randint(2, 24) * 2 + 1,
                 upscale=rng.choice([1, 2, 2, 4]))
    return c


# ------------------------------------------------------------------------------------------------------ the optics
def _radial(n, m, rho):
    """The unnormalized Zernike radial polynomial (float64 tensor rho)."""
    r = torch.zeros_like(rho)
    for k in range((n - m) // 2 + 1):
        r = r + (-1.0) ** k * math.comb(n - k, k) * math.comb(n - 2 * k, (n - m) // 2 - k) * rho ** (n - 2 * k)
    return r


def _pupil(p):
    """A request's Gibson-Lanni pupil on its M x M grid, float64: the aperture, the defocus-free phase and the phase per
    metre of stage travel."""
    M = p.pupil_samples
    k0 = TWO_PI / (p.wavelength_nm * 1e-9)
    b_max = min(1.0, p.sample_index / p.na)
    k_max = k0 * p.na * b_max
    dk = 2.0 * k_max / (M - 4)
    k = (torch.arange(M, dtype=torch.float64, device=DEV) - M // 2) * dk
    kx, ky = k[None, :].expand(M, M), k[:, None].expand(M, M)
    kr2 = kx * kx + ky * ky
    inside = kr2 <= k_max * k_max
    rho = torch.sqrt(kr2) / (k0 * p.na)
    phi = torch.atan2(ky, kx)
    depth = p.sample_depth_nm * 1e-9
    root = lambda n: torch.sqrt(torch.clamp(1.0 - (p.na * rho / n) ** 2, min=0.0))
    phase = k0 * p.sample_index * depth * root(p.sample_index)
    for j, coef in enumerate(p.zernike):
        if coef:
            n = 0
            while (n + 1) * (n + 2) // 2 <= j:
                n += 1
            m = 2 * (j - n * (n + 1) // 2) - n
            rn = rho / b_max
            ang = torch.cos(abs(m) * phi) if m >= 0 else torch.sin(abs(m) * phi)
            phase = phase + TWO_PI * coef * torch.where(rn <= 1.0, _radial(n, abs(m), rn), 0.0) * ang
    per_m = k0 * p.immersion_index * root(p.immersion_index)
    return inside, phase, per_m, k


def _planes(p, defocus_nm, size):
    """|E|^2 planes of a request at the given defocus, each normalized to sum 1: float64 (n, size, size)."""
    inside, phase, per_m, k = _pupil(p)
    dx = p.pixel_size_nm / p.oversampling * 1e-9
    s = (torch.arange(size, dtype=torch.float64, device=DEV) - (size - 1) / 2.0) * dx
    a = torch.polar(torch.ones((size, len(k)), dtype=torch.float64, device=DEV), s[:, None] * k[None, :])
    focal = p.sample_depth_nm * 1e-9 * (p.immersion_index / p.sample_index)
    out = []
    step = max(1, int(2 ** 27 // (size * size + len(k) ** 2)) // 2)
    dz = torch.as_tensor(np.asarray(defocus_nm, dtype=np.float64), device=DEV) * 1e-9 - focal
    for i in range(0, len(dz), step):
        ph = phase[None] + dz[i:i + step, None, None] * per_m[None]
        u = torch.where(inside[None], torch.polar(torch.ones_like(ph), ph), 0.0)
        e = torch.matmul(torch.matmul(a, u), a.T)
        pl = e.real ** 2 + e.imag ** 2
        out.append(pl / pl.sum(dim=(1, 2), keepdim=True))
    return torch.cat(out)


def _stack_request(half, os, nz, wavelength=670.0, zernike=(), pupil=64, depth_nm=0.0, na=1.45, pixel_nm=PIXEL_NM,
                   z_step=25.0, interp=INTERP_CUBIC):
    z = [0.0] * 28
    for j, v in zernike:
        z[j] = v
    return PsfParams(wavelength_nm=wavelength, na=na, immersion_index=1.518,
                     sample_index=1.33 if depth_nm else 1.518, sample_depth_nm=depth_nm, pixel_size_nm=pixel_nm,
                     zernike=z, oversampling=os, kernel_half_width_px=half, nz=nz, pupil_samples=pupil,
                     z_step_nm=z_step, interp=interp)


def _stack_planes(p):
    """The request's kernel stack as float32 planes (nz, size, size), plane z at (z - (nz - 1) / 2) z_step."""
    size = 2 * p.kernel_half_width_px * p.oversampling + 1
    dz = (np.arange(p.nz) - (p.nz - 1) / 2.0) * p.z_step_nm
    return _planes(p, dz, size).to(torch.float32).cpu().numpy()


def _movie_stacks(case):
    """The kernel stacks of a movie's dye groups: 670 nm unaberrated, 580 nm astigmatic."""
    out = []
    for c in range(case.get("colours", 1)):
        p = _stack_request(case["half"], case["os"], case["nz"], 670.0 if c == 0 else 580.0,
                           () if c == 0 else ((5, 0.24),))
        out.append(_stack_planes(p))
    return out


# ------------------------------------------------------------------------------------------------------ the camera
def _camera(emccd):
    if emccd:
        return CameraParams(quantum_efficiency=0.95, gain=1.0, read_noise_e=50.0, emccd=True, em_gain=300.0,
                            cic_electrons=0.002, bit_depth=16)
    return CameraParams(quantum_efficiency=1.0, dark_electrons=0.0, gain=2.2, read_noise_e=1.5, emccd=False)


def _static(eng, w, h, emccd, flat_bg, illum=None):
    r = np.random.default_rng(42)
    n = w * h
    off = (100.0 + 2.0 * r.standard_normal(n)).astype(np.float32)
    if emccd:
        eng.set_static(w, h, offset=off, illum=illum, flat_bg=flat_bg)
    else:
        gain = np.maximum(2.2 + 0.1 * r.standard_normal(n), 0.09).astype(np.float32)
        rn = np.maximum(1.5 + 0.3 * r.standard_normal(n), 0.0).astype(np.float32)
        eng.set_static(w, h, offset=off, gain=gain, read_noise=rn, illum=illum, flat_bg=flat_bg)


def _words(adu):
    """Device frames as signed 16-bit words (the same bytes): torch indexes and sums those, not uint16."""
    return adu.view(torch.int16)


# ------------------------------------------------------------------------------------------------------ blink movies
def _frame_counts(case, rng):
    mean = float(case["per_frame"])
    f = case["frames"]
    if case.get("uneven"):
        top = 8000.0 / 300.0 * mean
        mu = np.clip(mean * np.exp(case["uneven"] * rng.standard_normal(f)), min(10.0, mean), top)
    else:
        mu = np.full(f, mean)
    return rng.poisson(mu)


def _emitters(case, seed):
    rng = np.random.default_rng(seed)
    counts = _frame_counts(case, rng)
    n = int(counts.sum())
    em = np.zeros(max(n, 1), EMITTER_DTYPE)
    em["x_px"][:n] = case["width"] * rng.random(n) - 0.5
    em["y_px"][:n] = case["height"] * rng.random(n) - 0.5
    em["photons"][:n] = 2000.0 * np.exp(0.5 * rng.standard_normal(n))
    slot = rng.integers(0, case.get("colours", 1), n)
    em["plane"][:n] = rng.integers(0, case["nz"], n) + slot * 65536
    start = np.concatenate([[0], np.cumsum(counts)])
    fi = np.repeat(np.arange(case["frames"]), counts)
    em[:n] = em[:n][np.lexsort((slot, fi))]          # a frame's dye groups one after the other
    fr = np.zeros(case["frames"], FRAME_DTYPE)
    fr["em_start"], fr["em_count"] = start[:-1], counts
    fr["frame"] = np.arange(case["frames"])
    fr["bg_scale"] = 1.0
    return em, fr, n


def _prepare_render(case, seed):
    em, fr, n = _emitters(case, seed)
    eng = Engine(0)
    for s, planes in enumerate(_movie_stacks(case)):
        eng.kernel_set_planes(s, planes, case["os"], 25.0, INTERP[case["interp"]])
    _static(eng, case["width"], case["height"], case["emccd"], 20.0)
    eng.set_render_config(case["form"])
    shape = (case["frames"], case["height"], case["width"])
    return {"kind": "render", "eng": eng, "frames": case["frames"], "camera": _camera(case["emccd"]),
            "seed": 1000 + seed % 1000, "em": torch.from_numpy(em.view(np.uint8)).to(DEV),
            "fr": torch.from_numpy(fr.view(np.uint8)).to(DEV),
            "adu": torch.empty(shape, dtype=torch.uint16, device=DEV),
            "photons": torch.empty(shape, dtype=torch.float32, device=DEV) if case["photons"] else None}


def _run_render(s):
    s["eng"].render_frames_dev(s["em"], s["fr"], s["frames"], s["camera"], s["seed"], photons_dev=s["photons"],
                               adu_dev=s["adu"])
    return {"adu": _words(s["adu"])} if s["photons"] is None else {"adu": _words(s["adu"]), "photons": s["photons"]}


def _weights(t, interp):
    """(first tap, weights) of tap position t along one axis."""
    if interp == "nearest":
        return math.floor(t + 0.5), [1.0]
    b = math.floor(t)
    f = t - b
    if interp == "linear":
        return b, [1.0 - f, f]
    return b - 1, [-0.5 * f ** 3 + f * f - 0.5 * f, 1.5 * f ** 3 - 2.5 * f * f + 1.0,
                   -1.5 * f ** 3 + 2.0 * f * f + 0.5 * f, 0.5 * f ** 3 - 0.5 * f * f]


def _exact_photons(case, seed):
    """The expected images in float64: every emitter's kernel block sums, interpolated at its sub-pixel position."""
    em, fr, n = _emitters(case, seed)
    os, w, h, interp = case["os"], case["width"], case["height"], case["interp"]
    sums, pad = [], 4 * os
    for planes in _movie_stacks(case):
        p = np.pad(planes.astype(np.float64), ((0, 0), (os - 1 + pad, os - 1 + pad), (os - 1 + pad, os - 1 + pad)))
        c = np.cumsum(np.pad(p, ((0, 0), (1, 0), (0, 0))), axis=1)
        p = c[:, os:] - c[:, :-os]
        c = np.cumsum(np.pad(p, ((0, 0), (0, 0), (1, 0))), axis=2)
        sums.append(c[:, :, os:] - c[:, :, :-os])     # block sums from block -(os - 1) - pad on
    half = case["half"]
    kc, side = half * os, 2 * half + 1
    out = np.full((case["frames"], h, w), 20.0)
    for k in range(case["frames"]):
        for e in em[fr["em_start"][k]:fr["em_start"][k] + fr["em_count"][k]]:
            x0, y0 = math.floor(e["x_px"] + 0.5), math.floor(e["y_px"] + 0.5)
            bx, wx = _weights(kc + (x0 - e["x_px"] - 0.5) * os + 0.5, interp)
            by, wy = _weights(kc + (y0 - e["y_px"] - 0.5) * os + 0.5, interp)
            B = sums[int(e["plane"]) >> 16][int(e["plane"]) & 0xFFFF]
            r0, c0 = by - half * os + os - 1 + pad, bx - half * os + os - 1 + pad
            sq = np.zeros((side, side))
            for j, wj in enumerate(wy):
                for i, wi in enumerate(wx):
                    sq += wj * wi * B[r0 + j:r0 + j + side * os:os, c0 + i:c0 + i + side * os:os][:side, :side]
            ya, yb, xa, xb = max(0, y0 - half), min(h, y0 + half + 1), max(0, x0 - half), min(w, x0 + half + 1)
            if ya < yb and xa < xb:
                out[k, ya:yb, xa:xb] += e["photons"] * sq[ya - y0 + half:yb - y0 + half, xa - x0 + half:xb - x0 + half]
    return out


def _prepare_events(case, seed):
    rng = np.random.default_rng(seed)
    f, w, h = case["frames"], case["width"], case["height"]
    counts = rng.poisson(float(case["per_frame"]), f)
    n = int(counts.sum())
    fi = np.repeat(np.arange(f), counts)
    ev = np.zeros(max(n, 1), BLINK_EVENT_DTYPE)
    ev["x_um"][:n] = w * rng.random(n) * PIXEL_NM / 1000.0
    ev["y_um"][:n] = h * rng.random(n) * PIXEL_NM / 1000.0
    ev["z_nm"][:n] = rng.uniform(-300.0, 300.0, n)
    ev["t_start"][:n] = fi + rng.uniform(-0.6, 0.6, n)       # on for part of the frame
    ev["t_end"][:n] = ev["t_start"][:n] + rng.exponential(1.0, n) + 0.4
    ev["brightness"][:n] = np.exp(0.5 * rng.standard_normal(n))
    ev["excite"][:n] = 1.0
    eng = Engine(0)
    eng.kernel_set_planes(0, _movie_stacks(case)[0], case["os"], 25.0, INTERP[case["interp"]])
    eng.kernel_set_halo(0, 2e-4)
    y, x = np.mgrid[0:h, 0:w]
    r2 = ((x - (w - 1) / 2) / w) ** 2 + ((y - (h - 1) / 2) / h) ** 2
    _static(eng, w, h, case["emccd"], 8.0, illum=np.exp(-1.5 * r2).astype(np.float32))
    pin = lambda a: torch.from_numpy(a).pin_memory().numpy()
    drift = 0.02 * rng.standard_normal((2, f)).cumsum(axis=1)
    return {"kind": "events", "eng": eng, "events": pin(ev.view(np.uint8)).view(BLINK_EVENT_DTYPE)[:n],
            "bucket": np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32), "camera": _camera(case["emccd"]),
            "drift": (np.ascontiguousarray(drift[0]), np.ascontiguousarray(drift[1])), "seed": 2000 + seed % 1000,
            "adu": torch.empty((f, h, w), dtype=torch.uint16).pin_memory().numpy()}


def _run_events(s):
    _, adu, n = s["eng"].render_events(0, s["events"], s["bucket"], 0, PIXEL_NM, 2000.0, s["camera"], s["seed"],
                                       drift_x_px=s["drift"][0], drift_y_px=s["drift"][1], use_illum=True,
                                       min_photons=20.0, adu_out=s["adu"])
    return {"adu": adu, "emitters": n}


# ------------------------------------------------------------------------------------------------------ camera noise
def _prepare_noise(case, seed):
    f, h, w = case["frames"], case["height"], case["width"]
    eng = Engine(0)
    _static(eng, w, h, case["emccd"], 0.0)
    g = torch.Generator(device=DEV).manual_seed(seed)
    ph = 5.0 + 30.0 * torch.rand((f, h, w), generator=g, device=DEV)
    bright = torch.rand((f, h, w), generator=g, device=DEV)
    ph = torch.where(bright < 0.05, ph * (1.0 + 400.0 * bright), ph)     # one pixel in twenty on a spot
    return {"kind": "noise", "eng": eng, "photons": ph, "camera": _camera(case["emccd"]), "seed": 3000 + seed % 1000,
            "frames": torch.arange(f, dtype=torch.int32, device=DEV),
            "adu": torch.empty((f, h, w), dtype=torch.uint16, device=DEV)}


def _run_noise(s):
    return {"adu": _words(s["eng"].noise_frames_dev(s["photons"], s["frames"], s["camera"], s["seed"], out=s["adu"]))}


# ------------------------------------------------------------------------------------------------------ PSFs
def _aberrations(rng, modes, rms):
    return tuple((j, float(rng.normal(0.0, rms))) for j in range(3, 3 + modes))


def _psf_request(case, seed):
    rng = np.random.default_rng(seed)
    return _stack_request(case["half"], case["os"], case["nz"], 670.0, _aberrations(rng, case["modes"], 0.08),
                          case["pupil"], case["depth_nm"], na=1.3 if case["depth_nm"] else 1.45)


def _psf_defocus(case):
    return (np.arange(case["nz"]) - (case["nz"] - 1) / 2.0) * 25.0


def _prepare_psf(case, seed):
    size = 2 * case["half"] * case["os"] + 1
    return {"kind": "psf", "eng": Engine(0), "request": _psf_request(case, seed),
            "sets": np.zeros(case["nz"], np.uint32), "defocus": _psf_defocus(case), "size": size,
            "out": torch.empty((case["nz"], size, size), dtype=torch.float32, device=DEV)}


def _run_psf(s):
    return {"planes": s["eng"].psf_library_dev([s["request"]], s["sets"], s["defocus"], size=s["size"],
                                               method=CZT_FP32, out=s["out"])}


def _exact_psf(case, seed):
    return {"planes": _planes(_psf_request(case, seed), _psf_defocus(case), 2 * case["half"] * case["os"] + 1)}


def _library(case, seed):
    rng = np.random.default_rng(seed)
    wl = (520.0, 580.0, 670.0, 750.0)
    sets = [_stack_request(8, 4, 3, wl[i % 4], _aberrations(rng, 12, 0.1), case["pupil"], pixel_nm=100.0)
            for i in range(case["sets"])]
    dz = np.tile((np.arange(case["planes"]) - case["planes"] // 2) * 25.0, case["sets"])
    return sets, np.repeat(np.arange(case["sets"], dtype=np.int32), case["planes"]), dz


def _prepare_library(case, seed):
    sets, of, dz = _library(case, seed)
    plan = PsfPlan(Engine(0), sets, size=case["size"], method=CZT_F16X3)
    return {"kind": "library", "plan": plan, "set_of": torch.from_numpy(of).to(DEV),
            "defocus": torch.from_numpy(dz).to(DEV),
            "out": torch.empty((len(of), case["size"], case["size"]), dtype=torch.float32, device=DEV)}


def _run_library(s):
    return {"planes": s["plan"].run_dev(s["set_of"], s["defocus"], s["out"])}


def _exact_library(case, seed):
    sets, _, dz = _library(case, seed)
    n = case["planes"]
    return {"planes": torch.cat([_planes(p, dz[i * n:(i + 1) * n], case["size"]) for i, p in enumerate(sets)])}


# ------------------------------------------------------------------------------------------------------ widefield
def _specimen(nx, ny, nz, seed):
    """Dye counts of a specimen of ellipsoidal cells with nuclei and filaments (float32, whole multiples of 0.4)."""
    rng = np.random.default_rng(seed)
    d = torch.zeros((nz, ny, nx), dtype=torch.float32, device=DEV)
    z = torch.arange(nz, dtype=torch.float32, device=DEV)
    y = torch.arange(ny, dtype=torch.float32, device=DEV)
    x = torch.arange(nx, dtype=torch.float32, device=DEV)
    cells = max(3, int(50 * nx * ny / 512 ** 2))
    for _ in range(cells):
        c = rng.random(3) * (nz, ny, nx)
        r = rng.uniform(0.05, 0.15, 3) * (4 * nz, max(nx, ny), max(nx, ny))
        q = (((z - c[0]) / r[0]) ** 2)[:, None, None] + (((y - c[1]) / r[1]) ** 2)[None, :, None] + \
            (((x - c[2]) / r[2]) ** 2)[None, None, :]
        d += (q <= 1.0).float() + 2.0 * (q <= 0.16).float()
    walks = 20 * cells
    p = rng.random((walks, 1, 3)) * (nz, ny, nx) + rng.normal(0.0, (0.1, 0.8, 0.8), (walks, 60, 3)).cumsum(axis=1)
    i = np.floor(p).astype(np.int64).reshape(-1, 3)
    i = i[((i >= 0) & (i < (nz, ny, nx))).all(axis=1)]
    flat = torch.from_numpy((i[:, 0] * ny + i[:, 1]) * nx + i[:, 2]).to(DEV)
    d.view(-1).index_add_(0, flat, torch.full((len(flat),), 4.0, device=DEV))
    return d * 0.4


def _prepare_series(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    eng = Engine(0)
    p = _stack_request(case["half"], 1, case["stack"], 520.0, pupil=320, na=1.4, pixel_nm=100.0, z_step=200.0)
    eng.kernel_set_planes(0, _stack_planes(p), 1, 200.0, INTERP_NEAREST)
    plan = WidefieldPlan.from_kernel(eng, 0, 1, 0.1, 30.0, 200.0, (nz, ny, nx), (0, 0, nx, ny))
    _static(eng, nx, ny, True, 0.0)
    return {"kind": "series", "eng": eng, "plan": plan, "density": _specimen(nx, ny, nz, seed), "camera": _camera(True),
            "seed": 4000 + seed % 1000, "adu": torch.empty(plan.frame_shape, dtype=torch.uint16, device=DEV)}


def _run_series(s):
    s["plan"].render_dev(s["density"], 5.0, s["camera"], s["seed"], adu_dev=s["adu"])
    return {"adu": _words(s["adu"])}


def _measured_psf(case):
    """A 3D PSF of kz x ky x kx samples: a Gaussian beam through its focus."""
    z, y, x = (torch.arange(n, dtype=torch.float64, device=DEV) - n // 2 for n in (case["kz"], case["ky"], case["kx"]))
    s2 = (1.3 ** 2 * (1.0 + (z / 2.0) ** 2))[:, None, None]
    p = torch.exp(-(y[None, :, None] ** 2 + x[None, None, :] ** 2) / (2.0 * s2)) / s2
    return (p / p.sum()).to(torch.float32)


def _prepare_widefield(case, seed):
    shape = (case["nz"], case["ny"], case["nx"])
    plan = WidefieldPlan(Engine(0), shape, _measured_psf(case).cpu().numpy())
    return {"kind": "widefield", "plan": plan, "density": _specimen(case["nx"], case["ny"], case["nz"], seed),
            "image": torch.empty(plan.frame_shape, dtype=torch.float32, device=DEV)}


def _run_widefield(s):
    return {"image": s["plan"].convolve_dev(s["density"], s["image"])}


def _exact_widefield(case, seed):
    v = _specimen(case["nx"], case["ny"], case["nz"], seed).double()
    k = _measured_psf(case).double()
    shape = [a + b - 1 for a, b in zip(v.shape, k.shape)]
    full = torch.fft.irfftn(torch.fft.rfftn(v, shape) * torch.fft.rfftn(k, shape), shape)
    sl = tuple(slice(b // 2, b // 2 + a) for a, b in zip(v.shape, k.shape))
    return {"image": torch.clamp(full[sl], min=0.0)}


# ------------------------------------------------------------------------------------------------------ likelihood fits
NOLL = tuple(range(4, 25))


def _noll_nm(j):
    n, j1 = 0, j - 1
    while j1 > n:
        n += 1
        j1 -= n
    return n, (-1) ** j * ((n % 2) + 2 * ((j1 + ((n + 1) % 2)) // 2))


class _Roi:
    """The ROI model in torch, at the precision given: E = A U A^T from a 32 x 32 pupil to 64 x 64 samples, os x os of
    them per pixel, expected counts N kappa |E|^2 + b."""

    def __init__(self, roi, dtype):
        M, os, px, wl, na, ni = 32, 64 // roi, 108.0, 670.0, 1.45, 1.518
        f64 = torch.float64
        k_max = TWO_PI * na / wl
        dk = 2.0 * k_max / (M - 4)
        k = (torch.arange(M, dtype=f64, device=DEV) - M // 2) * dk
        kx, ky = k[None, :].expand(M, M), k[:, None].expand(M, M)
        kr2 = kx * kx + ky * ky
        inside = kr2 <= k_max * k_max
        u = (torch.arange(64, dtype=f64, device=DEV) + 0.5) / os
        a = u[:, None] * (k * px)[None, :]
        basis = []
        rho, theta = torch.sqrt(kr2) / k_max, torch.atan2(ky, kx)
        for j in NOLL:
            n, m = _noll_nm(j)
            am = abs(m)
            z = _radial(n, am, rho) * math.sqrt((1.0 if m == 0 else 2.0) * (n + 1))
            if m:
                z = z * (torch.cos(am * theta) if m > 0 else torch.sin(am * theta))
            basis.append(torch.where(inside, TWO_PI * z, 0.0))
        L, s = TWO_PI / dk, px / os
        self.kappa = s * s / (L * L * float(inside.sum()))
        self.kz = torch.where(inside, torch.sqrt(torch.clamp((TWO_PI * ni / wl) ** 2 - kr2, min=0.0)), 0.0)
        self.kx, self.ky, self.inside = px * kx, px * ky, inside
        self.basis = torch.stack(basis)
        self.A = torch.polar(torch.ones_like(a), a).to(torch.complex128 if dtype == f64 else torch.complex64)
        self.roi, self.os, self.dtype = roi, os, dtype

    def expected(self, params, b, zern):
        """(n, roi, roi) expected counts of params (n, 4) with background b (n,)."""
        x, y, z, N = (params[:, i].double()[:, None, None] for i in range(4))
        ph = z * self.kz + torch.tensordot(zern.double(), self.basis, 1) - (x * self.kx + y * self.ky)
        ph = ph.to(self.dtype) if self.dtype == torch.float64 else torch.remainder(ph, TWO_PI).to(self.dtype)
        u = torch.polar(torch.where(self.inside, torch.ones_like(ph), torch.zeros_like(ph)), ph)
        e = torch.matmul(self.A, torch.matmul(u, self.A.T))
        i = (e.real ** 2 + e.imag ** 2).reshape(-1, self.roi, self.os, self.roi, self.os).sum(dim=(2, 4))
        return N.to(self.dtype) * self.kappa * i + b.to(self.dtype)[:, None, None]


def _fit_inputs(case, seed):
    rng = np.random.default_rng(seed)
    f, per = case["frames"], case["per_frame"]
    n, c = f * per, case["roi"] / 2.0
    scale = case["roi"] / 32.0
    pt = np.column_stack([rng.uniform(c - 1.5, c + 1.5, n), rng.uniform(c - 1.5, c + 1.5, n),
                          rng.uniform(-500.0, 500.0, n) * scale, 2000.0 * np.exp(0.5 * rng.standard_normal(n))])
    bt, zt = rng.uniform(5.0, 20.0, f), rng.normal(0.0, 0.03, len(NOLL))
    p = pt + np.column_stack([rng.normal(0, 0.3, n), rng.normal(0, 0.3, n), rng.normal(0, 50.0, n),
                              pt[:, 3] * rng.normal(0, 0.1, n)])
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(DEV)
    frame = torch.arange(n, device=DEV) // per
    model = _Roi(case["roi"], torch.float32)
    truth, bg_true, z_true = to(pt), to(bt), to(zt)
    g = torch.Generator(device=DEV).manual_seed(seed)
    counts = torch.empty((n, case["roi"], case["roi"]), dtype=torch.float32, device=DEV)
    for i in range(0, n, 4096):
        mu = model.expected(truth[i:i + 4096], bg_true[frame[i:i + 4096]], z_true)
        counts[i:i + 4096] = torch.poisson(mu, generator=g)
    return {"params": to(p), "bg": to(bt * rng.uniform(0.9, 1.1, f)), "zern": to(zt + rng.normal(0, 0.01, len(zt))),
            "frame": frame.to(torch.int32), "counts": counts}


def _prepare_fit(case, seed):
    s = _fit_inputs(case, seed)
    for k in ("params", "bg", "zern"):
        s[k].requires_grad_(True)
    s["kind"], s["model"] = "fit", NllModel(Engine(0), NllSpec(roi=case["roi"], os=64 // case["roi"], noll=NOLL))
    return s


def _run_fit(s):
    for k in ("params", "bg", "zern"):
        s[k].grad = None
    loss = poisson_nll(s["model"], s["params"], s["bg"], s["zern"], s["counts"], s["frame"])
    loss.backward()
    return {"loss": float(loss.detach()), "params": s["params"].grad, "bg": s["bg"].grad, "zern": s["zern"].grad}


def _exact_fit(case, seed):
    s = _fit_inputs(case, seed)
    model = _Roi(case["roi"], torch.float64)
    n = len(s["params"])
    bg, zern = (s[k].double().requires_grad_(True) for k in ("bg", "zern"))
    grads, total = [], 0.0
    for i in range(0, n, 2048):
        p = s["params"][i:i + 2048].double().requires_grad_(True)
        mu = model.expected(p, bg[s["frame"][i:i + 2048].long()], zern)
        loss = (mu - s["counts"][i:i + 2048].double() * torch.log(mu)).sum()
        loss.backward()
        grads.append(p.grad)
        total += float(loss.detach())
    return {"loss": total, "params": torch.cat(grads), "bg": bg.grad, "zern": zern.grad}


# ------------------------------------------------------------------------------------------------------ binned frames
def _prepare_binned(case, seed):
    em, fr, _ = _emitters(case, seed)
    eng = Engine(0)
    eng.kernel_set_planes(0, _movie_stacks(case)[0], case["os"], 25.0, INTERP_CUBIC)
    _static(eng, case["width"], case["height"], True, 0.0)
    f, h, w = case["frames"], case["height"], case["width"]
    return {"kind": "binned", "eng": eng, "binned": BinnedRenderer(eng, w, h, case["upscale"], slot=0),
            "em": torch.from_numpy(em.view(np.uint8)).to(DEV), "fr": torch.from_numpy(fr.view(np.uint8)).to(DEV),
            "frames": f, "frame_ids": torch.arange(f, dtype=torch.int32, device=DEV), "camera": _camera(True),
            "seed": 5000 + seed % 1000, "image": torch.empty((f, h, w), dtype=torch.float32, device=DEV),
            "adu": torch.empty((f, h, w), dtype=torch.uint16, device=DEV)}


def _run_binned(s):
    s["image"].fill_(5.0)      # the background that the blinks are added to
    s["binned"].render_dev(s["em"], s["fr"], s["frames"], s["image"])
    s["eng"].noise_frames_dev(s["image"], s["frame_ids"], s["camera"], s["seed"], out=s["adu"])
    return {"image": s["image"], "adu": _words(s["adu"])}


def _exact_binned(case, seed):
    """Every emitter's photons in its cell, convolved per plane with the stack summed to the cell pitch."""
    em, fr, n = _emitters(case, seed)
    os, w, h = case["os"], case["width"], case["height"]
    u = max(c for c in range(1, min(case["upscale"], os) + 1) if os % c == 0)
    r = os // u
    P = torch.from_numpy(_movie_stacks(case)[0]).to(DEV).double()
    size = P.shape[1]
    s0 = math.floor((size - 1) / 2.0 - r / 2.0 + 1.0)
    R = max(1, -math.ceil((-s0 - r + 1) / r), math.floor((size - 1 - s0) / r))
    pad = size + r * (R + 1)
    Q = torch.nn.functional.pad(P, (pad, pad, pad, pad))
    a = s0 - R * r + pad
    D = 2 * R + 1
    K = Q[:, a:a + D * r, a:a + D * r].reshape(len(P), D, r, D, r).sum(dim=(2, 4)).float().double()
    gh, gw = h * u + 2 * R, w * u + 2 * R               # the cells whose emitters reach the frame
    fh, fw = gh + 2 * R, gw + 2 * R
    Kf = torch.fft.rfft2(K, (fh, fw))
    cx = np.floor((em["x_px"] + 0.5) * u).astype(np.int64) + R
    cy = np.floor((em["y_px"] + 0.5) * u).astype(np.int64) + R
    fi = np.repeat(np.arange(case["frames"]), fr["em_count"])
    ok = (cx >= 0) & (cx < gw) & (cy >= 0) & (cy < gh)
    ok[n:] = False
    photons = em["photons"].astype(np.float32).astype(np.float64)
    out = torch.empty((case["frames"], h, w), dtype=torch.float64, device=DEV)
    nz = len(P)
    for k in range(0, case["frames"], 4):
        m = min(4, case["frames"] - k)
        sel = np.flatnonzero(ok[:n] & (fi >= k) & (fi < k + m))
        at = (((fi[sel] - k) * nz + em["plane"][sel]) * gh + cy[sel]) * gw + cx[sel]
        g = torch.zeros(m * nz * gh * gw, dtype=torch.float64, device=DEV)
        g.index_add_(0, torch.from_numpy(at).to(DEV), torch.from_numpy(photons[sel]).to(DEV))
        S = (torch.fft.rfft2(g.view(m, nz, gh, gw), (fh, fw)) * Kf[None]).sum(dim=1)
        cells = torch.fft.irfft2(S, (fh, fw))[:, 2 * R:2 * R + h * u, 2 * R:2 * R + w * u]
        out[k:k + m] = 5.0 + torch.clamp(cells, min=0.0).reshape(m, h, u, w, u).sum(dim=(2, 4))
    return out


# ------------------------------------------------------------------------------------------------------ the interface
_PREPARE = {"render": _prepare_render, "events": _prepare_events, "noise": _prepare_noise, "psf": _prepare_psf,
            "library": _prepare_library, "series": _prepare_series, "widefield": _prepare_widefield,
            "fit": _prepare_fit, "binned": _prepare_binned}
_RUN = {"render": _run_render, "events": _run_events, "noise": _run_noise, "psf": _run_psf, "library": _run_library,
        "series": _run_series, "widefield": _run_widefield, "fit": _run_fit, "binned": _run_binned}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind == "render" and case["photons"] and case["frames"] * case["per_frame"] <= 20000:
        return {"adu": None, "photons": _exact_photons(case, seed)}
    if kind == "psf":
        return _exact_psf(case, seed)
    if kind == "library":
        return _exact_library(case, seed)
    if kind == "widefield":
        return _exact_widefield(case, seed)
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "binned":
        return {"image": _exact_binned(case, seed), "adu": None}
    return None                # camera frames: whole numbers


def work(case):
    """One pass's inputs read once and outputs written once, and the arithmetic of the model as it is defined."""
    k = case["kind"]
    if k in ("render", "events", "binned"):
        px = case["frames"] * case["width"] * case["height"]
        em = case["frames"] * case["per_frame"] * (math.exp(0.5) if case.get("uneven") else 1.0)
        bw = 2 * case["half"] * case["os"] + case["os"]
        side = 2 * case["half"] + 1
        stack = case.get("colours", 1) * case["nz"] * bw * bw * 4
        if k == "binned":
            cells = (side * case["upscale"]) ** 2
            return {"bytes": px * 10 + em * 32 + stack, "flops": em * cells * 2.0}
        taps = {"cubic": 16, "linear": 4, "nearest": 1}[case["interp"]]
        out = 2 + (4 if case.get("photons") else 0)
        return {"bytes": px * out + 12 * case["width"] * case["height"] + em * (64 if k == "events" else 32) + stack,
                "flops": em * side * side * (2.0 * taps + 2.0)}
    if k == "noise":
        px = case["frames"] * case["width"] * case["height"]
        return {"bytes": px * 6 + 12 * case["width"] * case["height"], "flops": px * 50.0}
    if k in ("psf", "library"):
        n = case["nz"] if k == "psf" else case["sets"] * case["planes"]
        P, M = (2 * case["half"] * case["os"] + 1 if k == "psf" else case["size"]), case["pupil"]
        return {"bytes": n * (P * P * 4 + 12) + M * M * 8, "flops": n * 8.0 * (M * M * P + M * P * P)}
    if k in ("series", "widefield"):
        vox = case["nx"] * case["ny"] * case["nz"]
        fft = 3 * 2 * 2.5 * math.log2(max(2, 8 * vox)) * 4 * vox
        return {"bytes": vox * (6 if k == "series" else 8), "flops": fft}
    n = case["frames"] * case["per_frame"]
    return {"bytes": 2 * n * (case["roi"] ** 2 * 4 + 20) + n * 16, "flops": n * 8.0 * 3 * (32 * 32 * 64 + 32 * 64 * 64)}
