"""Counter RNG and camera noise chain on the B200 against the reference's golden vectors and the oracle: integer
(pcg4d words, uniforms, ADU) bit for bit."""
import json
import os

import numpy as np
import pytest

from insiliscope_b200 import CameraParams

pytestmark = pytest.mark.gpu


def test_pcg4d_golden(engine, golden_dir):
    import torch
    g = json.load(open(os.path.join(golden_dir, "pcg4d_golden.json")))
    words = np.array([r["in_u32"] for r in g["rng"]], dtype=np.uint32)
    t = torch.from_numpy(words.view(np.int32)).cuda()
    out = engine.pcg4d(t).cpu().numpy().view(np.uint32)
    assert out.tolist() == [r["words"] for r in g["rng"]]


def test_pcg4d_random_vs_oracle(engine, oracle):
    import torch
    rng = np.random.default_rng(1)
    words = rng.integers(0, 2**32, size=(4096, 4), dtype=np.uint64).astype(np.uint32)
    out = engine.pcg4d(torch.from_numpy(words.view(np.int32)).cuda()).cpu().numpy().view(np.uint32)
    for i in range(0, 4096, 37):
        assert np.array_equal(out[i], oracle.pcg4d(*[int(x) for x in words[i]]))


def test_counter_uniforms(engine, oracle):
    got = engine.counter_uniforms(0x9E3779B9 ^ 42, 123, 5000, 257, 11).cpu().numpy()
    want = oracle.counter_uniforms(0x9E3779B9 ^ 42, 123, 5000, 257, 11)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("emccd", [False, True])
def test_noise_chain_bit_exact(engine, oracle, emccd):
    """ADU frames equal the CPU chain's for every pixel: photons spanning both Poisson branches (mean 60 boundary),
    zero, negative, and the saturation clamp; per-pixel maps; a window's pixel base."""
    import torch
    rng = np.random.default_rng(10 + emccd)
    W, H, n = 96, 80, 6
    photons = rng.gamma(1.2, 45.0, size=(n, H, W)).astype(np.float32)
    photons[:, ::9, ::4] *= 40.0
    photons[0, 0, :6] = [0.0, -5.0, 59.999, 60.0, 60.001, 1e6]
    off, gain, rn = oracle.camera_maps(W, H, 42, 100.0, 2.0, 2.2, 0.1 / 2.2, 1.5, 0.2)
    if emccd:
        cam = CameraParams(quantum_efficiency=0.9, dark_electrons=0.02, gain=0.05, read_noise_e=30.0, emccd=True,
                           em_gain=300.0, cic_electrons=0.002, bit_depth=16)
        gain = None
    else:
        cam = CameraParams(quantum_efficiency=1.0, dark_electrons=0.0, gain=2.2, read_noise_e=1.5)
    engine.set_static(W, H, pixel_base=7 * W, offset=off, gain=gain, read_noise=rn, flat_bg=0.0)
    frames = [0, 1, 2, 199, 4096, 2**31 + 5]
    got = engine.noise_frames_dev(torch.from_numpy(photons).cuda(), frames, cam, 42 ^ 0x9E3779B9).cpu().numpy()
    mism = 0
    for k in range(n):
        want = oracle.noise_chain(photons[k], cam, off.reshape(H, W), None if gain is None else gain.reshape(H, W),
                                  rn.reshape(H, W), 42 ^ 0x9E3779B9, frames[k], pixel_base=7 * W)
        mism += int((got[k] != want).sum())
    assert mism == 0


CAMERAS = {
    "scmos_maps": dict(gain=2.2, read_noise_e=1.5),
    "scmos_scalars": dict(quantum_efficiency=0.82, dark_electrons=0.35, gain=0.46, read_noise_e=1.1),
    "scmos_no_read_noise": dict(gain=1.0, read_noise_e=0.0),
    "emccd_maps": dict(quantum_efficiency=0.95, gain=1.0, read_noise_e=50.0, emccd=True, em_gain=300.0,
                       cic_electrons=0.002),
    "emccd_scalars": dict(quantum_efficiency=0.9, dark_electrons=0.02, gain=0.05, read_noise_e=30.0, emccd=True,
                          em_gain=4.0, cic_electrons=0.0, bit_depth=14),
    "negative_dark": dict(dark_electrons=-0.5, gain=2.0, read_noise_e=1.5),   # outside the float32 form's bounds
}


@pytest.mark.parametrize("name", list(CAMERAS))
def test_float_decisions_bit_exact(engine, oracle, name):
    """The float32 decisions over every branch's edges: means spread over 1e-8 .. 1e9 by logarithm, dense around the
    60-photon switch and among small counts, and zero, negative, NaN and infinite ones; every ADU the CPU chain's."""
    import torch
    kw = dict(CAMERAS[name])
    rng = np.random.default_rng(len(name))
    W, H, n = 211, 97, 12
    ph = 10.0 ** rng.uniform(-8.0, 9.0, (n, H, W))
    ph[1:4] = rng.uniform(0.0, 130.0, (3, H, W))
    ph[4:7] = rng.uniform(0.0, 12.0, (3, H, W))
    ph[7] = 60.0 / kw.get("quantum_efficiency", 1.0) + rng.normal(0.0, 2e-4, (H, W))
    ph[8:10] = rng.uniform(100.0, 5000.0, (2, H, W))
    ph = ph.astype(np.float32)
    ph[0, 0, :8] = [0.0, -0.0, -3.0, np.nan, np.inf, -np.inf, 1e-45, 3e38]
    ph[10, :, ::3] = 0.0
    off = gain = rn = None
    if name.endswith("maps"):
        off, gain, rn = oracle.camera_maps(W, H, 5, 100.0, 2.0, 2.2, 0.1 / 2.2, 1.5, 0.2)
        if kw.get("emccd"):
            gain = rn = None
        else:
            gain[3], gain[4], gain[5] = 0.0, -2.0, 1e-38
            rn[6], rn[7] = 0.0, 400.0
            off[8], off[9] = -50.0, 65530.0
    cam = CameraParams(**kw)
    engine.set_static(W, H, pixel_base=3 * W, offset=off, gain=gain, read_noise=rn, flat_bg=0.0)
    frames = [0, 1, 2, 199, 4096, 2**31 + 5, 7, 8, 9, 10, 11, 12]
    got = engine.noise_frames_dev(torch.from_numpy(ph).cuda(), frames, cam, 977).cpu().numpy()
    shaped = [None if a is None else a.reshape(H, W) for a in (off, gain, rn)]
    finite = np.isfinite(ph) & (np.abs(ph) < 1e15)   # beyond, the float64 ADU's own conversion is undefined
    for k in range(n):
        want = oracle.noise_chain(ph[k], cam, *shaped, 977, frames[k], pixel_base=3 * W)
        diff = (got[k] != want) & finite[k]
        if gain is not None:
            diff.reshape(-1)[3] = False              # a zero gain's ADU is not a number
        assert not diff.any(), (k, int(diff.sum()), ph[k][diff][:4], got[k][diff][:4], want[diff][:4])


@pytest.mark.parametrize("gain,em_gain,read,depth", [(1.0, 300.0, 50.0, 16), (0.05, 4.0, 30.0, 14), (40.0, 1.0, 200.0, 16),
                                                     (-3.0, 20.0, 5.0, 12)])
def test_bright_emccd_bit_exact(engine, oracle, gain, em_gain, read, depth):
    """EMCCD means from 150 to 3e6 photons, dense around the 512 electrons from which the register is worked out in
    float64 and around the million from which the whole chain is, clamped and not: every ADU the CPU chain's."""
    import torch
    rng = np.random.default_rng(int(abs(gain) * 100) + depth)
    W, H, n = 203, 101, 8
    ph = 10.0 ** rng.uniform(np.log10(150.0), np.log10(3e6), (n, H, W))
    ph[1] = rng.uniform(480.0, 620.0, (H, W))
    ph[2] = 10.0 ** rng.uniform(5.99, 6.01, (H, W))
    ph[3:5] = rng.uniform(2000.0, 30000.0, (2, H, W))
    ph = ph.astype(np.float32)
    off = rng.uniform(-2000.0, 3000.0, W * H).astype(np.float32)
    cam = CameraParams(quantum_efficiency=0.93, dark_electrons=0.01, gain=gain, read_noise_e=read, emccd=True,
                       em_gain=em_gain, cic_electrons=0.005, bit_depth=depth)
    engine.set_static(W, H, pixel_base=W, offset=off, flat_bg=0.0)
    frames = [3, 77, 2**31 + 1, 4, 5, 6, 7, 8]
    got = engine.noise_frames_dev(torch.from_numpy(ph).cuda(), frames, cam, 311).cpu().numpy()
    for k in range(n):
        want = oracle.noise_chain(ph[k], cam, off.reshape(H, W), None, None, 311, frames[k], pixel_base=W)
        assert np.array_equal(got[k], want), (k, int((got[k] != want).sum()))


def _noise_us(engine, mean, cam):
    """The noise of 8 frames of 512 x 512 px at a mean, in us by the device's clock (the best of ten)."""
    import torch
    W, n = 512, 8
    engine.set_static(W, W, flat_bg=0.0)
    ph = mean * (0.8 + 0.4 * torch.rand((n, W, W), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda"))
    fr = torch.arange(n, dtype=torch.int32, device="cuda")
    out = torch.empty((n, W, W), dtype=torch.uint16, device="cuda")
    best = 1e9
    with torch.cuda.stream(engine.torch_stream()):
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            engine.noise_frames_dev(ph, fr, cam, 7, out=out, sync=False)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
    return best


def test_bright_emccd_frames_take_no_longer(engine):
    """The chain's float32 bounds grow with the electrons; bright frames must not fall through to the float64 chain."""
    cam = CameraParams(quantum_efficiency=0.95, gain=1.0, read_noise_e=50.0, emccd=True, em_gain=300.0,
                       cic_electrons=0.002)
    dim = _noise_us(engine, 300.0, cam)
    for mean in (1e3, 6e3, 1.9e4, 3e4, 2e5):
        assert _noise_us(engine, mean, cam) <= 1.6 * dim, mean


def test_cameras_without_float_bounds_skip_the_float_chain(engine):
    """A camera that the float32 bounds do not hold for (here a negative dark current) takes the float64 chain alone: one
    and a half times the float32 chain's time, twice with both."""
    fast = _noise_us(engine, 20.0, CameraParams(gain=2.2, read_noise_e=1.5, dark_electrons=0.5))
    assert _noise_us(engine, 20.0, CameraParams(gain=2.2, read_noise_e=1.5, dark_electrons=-0.5)) <= 1.75 * fast
