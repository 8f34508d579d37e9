"""The render kernel's forms on an uneven two-colour movie: every tile shape, grid or persistent, the autotuned form
and the captured CUDA graph give the reference's frames bit for bit (the reference's multi-colour frame loop: each
dye group with its own kernel, the later group splatted onto the earlier one, then the noise chain)."""
import numpy as np
import pytest
import torch

from insiliscope_b200 import (BLINK_EVENT_DTYPE, EMITTER_DTYPE, INTERP_CUBIC, INTERP_LINEAR, INTERP_NEAREST,
                              CameraParams, PsfParams, RenderGraph, frames_table)
from insiliscope_b200.workloads import noll_rms_to_osa_waves

pytestmark = pytest.mark.gpu

W, H, F, PX = 72, 56, 23, 108.0
PER_BLINK, BG = 1800.0, 15.0


def _requests():
    common = dict(na=1.45, pixel_size_nm=PX, oversampling=4, kernel_half_width_px=8, nz=9, z_step_nm=100.0,
                  pupil_samples=64, interp=INTERP_CUBIC)
    return [PsfParams(wavelength_nm=670.0, double_helix=True, **common),
            PsfParams(wavelength_nm=580.0, zernike=noll_rms_to_osa_waves({5: 0.1}), **common)]


def _movie(rng, frames=F):
    """Frame f: Poisson(mu_f) emitters, mu_f lognormal (median 40, sigma 1.2) clipped to [0.5, 400]; channel 0 then 1
    within each frame."""
    mu = np.clip(40.0 * np.exp(1.2 * rng.standard_normal(frames)), 0.5, 400.0)
    counts = rng.poisson(mu)
    counts[3] = 0                                  # an empty frame
    n = int(counts.sum())
    fi = np.repeat(np.arange(frames), counts)
    ch = (rng.random(n) < 0.5).astype(np.int32)
    order = np.lexsort((ch, fi))
    ev = np.zeros(n, BLINK_EVENT_DTYPE)
    ev["x_um"] = rng.uniform(-0.5, W * PX / 1000 + 0.5, n)
    ev["y_um"] = rng.uniform(-0.5, H * PX / 1000 + 0.5, n)
    ev["z_nm"] = rng.uniform(-450, 450, n)
    ev["t_start"] = fi.astype(np.float64)
    ev["t_end"] = ev["t_start"] + 1.0
    ev["brightness"] = rng.lognormal(0.0, 0.5, n)
    ev["excite"] = 1.0
    ev["slot"] = ch
    ev = ev[order]
    return ev, np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)


@pytest.fixture(scope="module")
def setup(engine, reference, oracle):
    kernels = [reference.kernel(req=r) for r in _requests()]
    for s, k in enumerate(kernels):
        engine.kernel_set_planes(s, k.planes(), 4, 100.0, INTERP_CUBIC)
    off, gain, rn = oracle.camera_maps(W, H, 42, 100.0, 2.0, 2.2, 0.1 / 2.2, 1.5, 0.2)
    engine.set_static(W, H, offset=off, gain=gain, read_noise=rn, flat_bg=BG)
    cam = CameraParams(gain=2.2, read_noise_e=1.5)
    return kernels, (off, gain, rn), cam


def _batch(engine, ev, bucket):
    ems, frames, _ = engine.collect_emitters(-1, ev, bucket, 0, W, H, PX, PER_BLINK)
    return ems.copy(), frames.copy()


def _dev(engine, ems, frames):
    d_em = torch.from_numpy(np.ascontiguousarray(ems).view(np.uint8)).cuda()
    d_fr = torch.from_numpy(np.ascontiguousarray(frames).view(np.uint8)).cuda()
    n = len(frames)
    d_ph = torch.empty((n, H, W), dtype=torch.float32, device="cuda")
    d_adu = torch.empty((n, H, W), dtype=torch.uint16, device="cuda")
    return d_em, d_fr, d_ph, d_adu


def test_forms_match_reference(engine, reference, setup):
    kernels, (off, gain, rn), cam = setup
    rng = np.random.default_rng(31)
    ev, bucket = _movie(rng)
    ems, frames = _batch(engine, ev, bucket)
    assert ems["plane"].max() >> 16 == 1 and ems["plane"].min() >> 16 == 0
    seed = 1234
    _, want_ph, want_adu = reference.render_movie_groups(kernels, ev, 0, F, W, H, PX, PER_BLINK, BG, cam,
                                                         off, gain, rn, seed, want_photons=True)
    try:
        for config in range(engine.RENDER_CONFIGS):
            engine.set_render_config(config)
            assert engine.render_config()[0] == config
            ph, adu = engine.render_frames(ems, frames, cam, seed)
            assert np.array_equal(ph, want_ph), config
            assert np.array_equal(adu, want_adu), config
            ph2, _ = engine.render_frames(ems, frames, None, 0, want_adu=False)
            assert np.array_equal(ph2, want_ph), config
    finally:
        engine.set_render_config(0)


@pytest.mark.parametrize("emccd", [False, True])
def test_two_pass_noise_without_photons(engine, reference, setup, emccd):
    """The two-pass forms when the caller keeps no photon frames (the tiles' photon values in scratch ahead of the
    pooled noise chain), on an sCMOS and an EMCCD camera: the reference's frames bit for bit."""
    kernels, (off, gain, rn), _ = setup
    cam = CameraParams(quantum_efficiency=0.9, dark_electrons=0.02, gain=2.2 if not emccd else 4.0, read_noise_e=1.5,
                       emccd=emccd, em_gain=150.0, cic_electrons=0.003)
    rng = np.random.default_rng(41)
    ev, bucket = _movie(rng)
    ems, frames = _batch(engine, ev, bucket)
    seed = 99
    _, _, want_adu = reference.render_movie_groups(kernels, ev, 0, F, W, H, PX, PER_BLINK, BG, cam, off, gain, rn,
                                                   seed)
    try:
        for config in range(12, engine.RENDER_CONFIGS):
            engine.set_render_config(config)
            ph, adu = engine.render_frames(ems, frames, cam, seed, want_photons=False)
            assert ph is None
            assert np.array_equal(adu, want_adu), config
    finally:
        engine.set_render_config(0)


def test_autotune_and_graph(engine, reference, setup):
    kernels, (off, gain, rn), cam = setup
    rng = np.random.default_rng(77)
    ev, bucket = _movie(rng)
    ems, frames = _batch(engine, ev, bucket)
    d_em, d_fr, d_ph, d_adu = _dev(engine, ems, frames)
    try:
        ms = engine.render_autotune(d_em, d_fr, F, cam, 5, d_adu)
        assert len(ms) == engine.RENDER_CONFIGS and all(m > 0 for m in ms)
        config = engine.render_config()[0]
        assert ms[config] == min(ms)
        ph_h, adu_h = engine.render_frames(ems, frames, cam, 5)
        for persistent_config in (config, 4, 9, 12, 15):
            engine.set_render_config(persistent_config)
            g = RenderGraph(engine, d_em, d_fr, F, cam, 5, d_ph, d_adu)
            d_ph.zero_()
            d_adu.zero_()
            n0 = engine.launch_count
            g.launch()
            assert engine.launch_count > n0
            assert np.array_equal(d_ph.cpu().numpy(), ph_h)
            assert np.array_equal(d_adu.cpu().numpy(), adu_h)
            # the same buffers refilled in place with another batch of the same size: the replay renders it
            ems2 = ems.copy()
            ems2["photons"] *= 0.5
            d_em.copy_(torch.from_numpy(ems2.view(np.uint8)))
            g.launch()
            ph2, adu2 = engine.render_frames(ems2, frames, cam, 5)
            assert np.array_equal(d_ph.cpu().numpy(), ph2)
            assert np.array_equal(d_adu.cpu().numpy(), adu2)
            d_em.copy_(torch.from_numpy(ems.view(np.uint8)))
            g.close()
        _, _, want_adu = reference.render_movie_groups(kernels, ev, 0, F, W, H, PX, PER_BLINK, BG, cam, off, gain, rn,
                                                       5)
        assert np.array_equal(adu_h, want_adu)
    finally:
        engine.set_render_config(0)


def test_heavy_frame_batch(engine, setup):
    """A batch whose frames run from 0 to 3,000 emitters: the persistent forms equal the grid form."""
    _, _, cam = setup
    rng = np.random.default_rng(5)
    counts = np.array([0, 3000, 2, 900, 40, 1, 2200, 0, 10], np.int64)
    n = int(counts.sum())
    fi = np.repeat(np.arange(len(counts)), counts)
    ev = np.zeros(n, BLINK_EVENT_DTYPE)
    ev["x_um"] = rng.uniform(0, W * PX / 1000, n)
    ev["y_um"] = rng.uniform(0, H * PX / 1000, n)
    ev["z_nm"] = rng.uniform(-400, 400, n)
    ev["t_start"] = fi
    ev["t_end"] = fi + 1.0
    ev["brightness"] = 1.0
    ev["excite"] = 1.0
    ev["slot"] = (rng.random(n) < 0.3).astype(np.int32)
    ev = ev[np.lexsort((ev["slot"], fi))]
    ems, frames = _batch(engine, ev, np.concatenate([[0], np.cumsum(counts)]))
    try:
        engine.set_render_config(0)
        want = engine.render_frames(ems, frames, cam, 9)
        for config in (3, 4, 5, 6, 9, 11, 12, 13, 14, 15, 16, 17):
            engine.set_render_config(config)
            got = engine.render_frames(ems, frames, cam, 9)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), config
    finally:
        engine.set_render_config(0)


def test_two_pass_over_limit_falls_back(engine, reference, setup):
    """A two-pass form whose contributions pass the limit renders in the one-pass form: the same bits."""
    kernels, (off, gain, rn), cam = setup
    ev, bucket = _movie(np.random.default_rng(8))
    ems, frames = _batch(engine, ev, bucket)
    try:
        engine.set_render_config(15)
        want = engine.render_frames(ems, frames, cam, 3)
        engine.set_contrib_limit(1024)
        got = engine.render_frames(ems, frames, cam, 3)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    finally:
        engine.set_contrib_limit(0)
        engine.set_render_config(0)


def test_bad_config_rejected(engine):
    from insiliscope_b200 import IscuError
    with pytest.raises(IscuError):
        engine.set_render_config(engine.RENDER_CONFIGS)
    assert engine.render_config()[0] in range(engine.RENDER_CONFIGS)


@pytest.mark.parametrize("interp", [INTERP_CUBIC, INTERP_LINEAR, INTERP_NEAREST])
@pytest.mark.parametrize("halo", [0.0, 2e-4])
def test_contributions_equal_the_one_pass_sums(engine, interp, halo):
    """The two-pass forms' contributions (fused sums, the reference's order where their rounding is in doubt) against
    the one-pass forms' unfused ones, bit for bit: 4 million (emitter, pixel) sums, of which some 500 are in doubt by
    the midpoint test alone, over planes with zeros, negative values and cancelling taps and photons of every size."""
    import torch
    rng = np.random.default_rng(17 + interp)
    nz, os_, half = 7, 4, 12
    n = 2 * half * os_ + 1
    y, x = np.mgrid[0:n, 0:n] - (n - 1) / 2.0
    planes = np.stack([np.exp(-(x * x + y * y) / (2.0 * (4.0 + 2.0 * z) ** 2)) * (1.0 + 0.3 * np.cos(0.9 * x + z))
                       for z in range(nz)]).astype(np.float32)
    planes /= planes.sum(axis=(1, 2), keepdims=True)
    planes[2] -= planes[2].mean()                        # negative and cancelling values
    planes[3][:, : n // 2] = 0.0
    planes[4] = rng.standard_normal((n, n)) * 1e-4
    planes[5] *= 1e-33
    engine.kernel_set_planes(0, planes, os_, 25.0, interp)
    engine.kernel_set_planes(1, planes[:3], os_, 25.0, interp)
    if halo:
        engine.kernel_set_halo(0, halo)
    w, h, per = 83, 61, np.array([1500, 0, 3, 2500, 64, 65, 2800])
    total = int(per.sum())
    em = np.zeros(total, EMITTER_DTYPE)
    em["x_px"] = rng.uniform(-half - 1.0, w + half, total)
    em["y_px"] = rng.uniform(-half - 1.0, h + half, total)
    em["photons"] = 2000.0 * np.exp(0.7 * rng.standard_normal(total))
    slot = rng.integers(0, 2, total)
    em["plane"] = np.where(slot == 1, rng.integers(0, 3, total), rng.integers(0, nz, total)) + slot * 65536
    em["photons"][:8] = [1e-300, 1e-40, 1e33, 1e39, 1e300, -1.0, 0.0, 1e-20]
    em["x_px"][8], em["y_px"][9] = np.nan, 1e10
    fr = frames_table(per)
    engine.set_static(w, h, flat_bg=20.0)
    cam = CameraParams(gain=2.0, read_noise_e=1.5)
    dem, dfr = (torch.from_numpy(a.view(np.uint8)).cuda() for a in (em, fr))
    out = {}
    for config in (0, 12, 13, 14, 17):
        engine.set_render_config(config)
        ph = torch.empty((len(fr), h, w), dtype=torch.float32, device="cuda")
        adu = torch.empty((len(fr), h, w), dtype=torch.uint16, device="cuda")
        engine.render_frames_dev(dem, dfr, len(fr), cam, 5, ph, adu)
        out[config] = ph.cpu().numpy(), adu.cpu().numpy()
    engine.set_render_config(0)
    if halo:
        engine.kernel_set_halo(0, 0.0)
    for config, (ph, adu) in out.items():
        assert np.array_equal(ph, out[0][0], equal_nan=True), config
        assert np.array_equal(adu, out[0][1]), config


@pytest.mark.parametrize("per", [(1,), (2, 0, 3), (65, 2047, 2049, 64)])
def test_small_batches_equal_the_one_emitter_step(engine, per):
    """A batch whose CTAs are all resident takes two emitters a step where they have the same taps (here cubic, linear,
    nearest and off-band emitters mixed, odd counts, both sides of a chunk); the persistent form takes one: the same
    bits, also next to the same frames in a batch over the line."""
    import torch
    rng = np.random.default_rng(len(per))
    half, os_ = 6, 4
    n = 2 * half * os_ + 1
    planes = rng.uniform(0.0, 1e-3, (3, n, n)).astype(np.float32)
    for slot, interp in enumerate((INTERP_CUBIC, INTERP_LINEAR, INTERP_NEAREST)):
        engine.kernel_set_planes(slot, planes, os_, 25.0, interp)
    w, h, total = 49, 35, sum(per)
    em = np.zeros(total, EMITTER_DTYPE)
    em["x_px"] = rng.uniform(-half, w + half, total)
    em["y_px"] = rng.uniform(-half, h + half, total)
    em["photons"] = rng.uniform(1.0, 3000.0, total)
    em["plane"] = rng.integers(0, 3, total) + 65536 * np.where(rng.uniform(size=total) < 0.7, 0, rng.integers(0, 3, total))
    engine.set_static(w, h, flat_bg=10.0)
    cam = CameraParams(gain=2.0, read_noise_e=1.5)
    dem = torch.from_numpy(em.view(np.uint8)).cuda()
    out = []
    for config, empty in ((0, 0), (3, 0), (0, 60)):
        fr = frames_table(np.concatenate([np.array(per), np.zeros(empty, int)]))
        dfr = torch.from_numpy(fr.view(np.uint8)).cuda()
        ph = torch.empty((len(fr), h, w), dtype=torch.float32, device="cuda")
        adu = torch.empty((len(fr), h, w), dtype=torch.uint16, device="cuda")
        try:
            engine.set_render_config(config)
            engine.render_frames_dev(dem, dfr, len(fr), cam, 5, ph, adu)
        finally:
            engine.set_render_config(0)
        out.append((ph.cpu().numpy()[: len(per)], adu.cpu().numpy()[: len(per)]))
    for got in out[1:]:
        assert np.array_equal(got[0].view(np.uint32), out[0][0].view(np.uint32))
        assert np.array_equal(got[1], out[0][1])


def _mixed_squares(engine, big_half, per, frames):
    """A movie whose emitters are all of a 7 x 7-square stack, beside a stack of squares of big_half (0: alone): device
    emitters and frames, after the stacks are set."""
    import torch
    rng = np.random.default_rng(3)
    planes = rng.uniform(0.0, 1e-3, (5, 25, 25)).astype(np.float32)
    if big_half:
        n = 4 * big_half + 1
        engine.kernel_set_planes(0, rng.uniform(0.0, 1e-5, (3, n, n)).astype(np.float32), 2, 25.0, INTERP_CUBIC)
    engine.kernel_set_planes(1 if big_half else 0, planes, 4, 25.0, INTERP_CUBIC)
    n = per * frames
    em = np.zeros(n, EMITTER_DTYPE)
    em["x_px"], em["y_px"] = rng.uniform(-1.0, 100.0, (2, n))
    em["photons"] = rng.uniform(100.0, 3000.0, n)
    em["plane"] = rng.integers(0, 5, n) + (65536 if big_half else 0)
    engine.set_static(100, 100, flat_bg=20.0)
    return [torch.from_numpy(a.view(np.uint8)).cuda() for a in (em, frames_table(np.full(frames, per)))]


def test_small_squares_beside_large_ones():
    """The contributions of a stack of small squares take no more work for a stack of large squares in another slot that
    no emitter is of, and are the one-pass form's bits."""
    import torch
    from insiliscope_b200 import Engine
    times = {}
    for half in (0, 40):
        with Engine(0) as engine:
            dem, dfr = _mixed_squares(engine, half, 500, 150)
            cam, out = CameraParams(gain=2.0, read_noise_e=1.5), {}
            for config in (0, 12):
                engine.set_render_config(config)
                ph = torch.empty((150, 100, 100), dtype=torch.float32, device="cuda")
                adu = torch.empty((150, 100, 100), dtype=torch.uint16, device="cuda")
                best = 1e9
                for _ in range(6):
                    engine.set_render_timing(True)
                    engine.render_frames_dev(dem, dfr, 150, cam, 5, ph, adu)
                    best = min(best, engine.render_pass_times()[0]["contributions"])
                engine.set_render_timing(False)
                out[config], times[half] = (ph.cpu().numpy(), adu.cpu().numpy()), best
            assert np.array_equal(out[0][0].view(np.uint32), out[12][0].view(np.uint32))
            assert np.array_equal(out[0][1], out[12][1])
    assert times[40] <= 1.5 * times[0], times


def test_cancelling_taps_at_extreme_photons():
    """Taps that cancel to 1e-7 of their magnitude, by emitters of 1e-44 to 1e30 photons on samples that keep the product
    in float's range: the two-pass contributions are the one-pass sums' bits (at 1e-7 the fused and the reference's order
    differ in one pixel in ten, so none may be taken for sure)."""
    import torch
    from insiliscope_b200 import Engine
    rng = np.random.default_rng(29)
    half, n = 6, 13
    for photons in (1e-44, 3e-42, 1e-38, 1e-36, 1.0, 1e30):
        a = 1e-12 / photons if photons < 1.0 else 1e-3 / photons ** 0.5
        planes = np.where(np.arange(n) % 2, -1.0, 1.0) * min(a, 1e31) * (1.0 + 1e-7 * rng.random((3, n, n)))
        with Engine(0) as eng:
            eng.kernel_set_planes(0, planes.astype(np.float32), 1, 25.0, INTERP_LINEAR)
            eng.set_static(40, 40, flat_bg=0.0)
            em = np.zeros(400, EMITTER_DTYPE)
            em["x_px"] = rng.integers(0, 40, 400) + 0.5 + 1e-9 * rng.random(400)
            em["y_px"] = rng.uniform(0.0, 40.0, 400)
            em["photons"], em["plane"] = photons, rng.integers(0, 3, 400)
            fr = frames_table(np.full(100, 4))
            dem, dfr = (torch.from_numpy(t.view(np.uint8)).cuda() for t in (em, fr))
            out = []
            for config in (0, 12):
                eng.set_render_config(config)
                ph = torch.empty((100, 40, 40), dtype=torch.float32, device="cuda")
                eng.render_frames_dev(dem, dfr, 100, None, 5, ph)
                out.append(ph.cpu().numpy().view(np.uint32))
            assert (out[0] != 0).any()
            assert np.array_equal(*out), (photons, int((out[0] != out[1]).sum()))


def test_steep_stacks_take_no_second_sum():
    """A Gaussian stack whose far samples fall by more than the fused sums' bound allows takes about a slowly falling
    stack's time for its contributions (each sum once, in the reference's order), and gives the one-pass bits."""
    import torch
    from insiliscope_b200 import Engine
    rng = np.random.default_rng(31)
    half, os_, frames, per = 16, 4, 150, 160
    n = 2 * half * os_ + 1
    y, x = np.mgrid[0:n, 0:n] - (n - 1) / 2.0
    r2 = (x * x + y * y) / (1.2 * os_) ** 2
    em = np.zeros(frames * per, EMITTER_DTYPE)
    em["x_px"], em["y_px"] = rng.uniform(-0.5, 127.5, (2, len(em)))
    em["photons"], em["plane"] = 2000.0 * np.exp(0.5 * rng.standard_normal(len(em))), rng.integers(0, 25, len(em))
    dem, dfr = (torch.from_numpy(t.view(np.uint8)).cuda() for t in (em, frames_table(np.full(frames, per))))
    cam, times = CameraParams(gain=2.0, read_noise_e=1.5), {}
    for name, plane in (("steep", np.exp(-0.5 * r2)), ("slow", (1.0 + r2) ** -1.5)):
        with Engine(0) as eng:
            eng.kernel_set_planes(0, np.repeat((plane / plane.sum())[None], 25, 0).astype(np.float32), os_, 25.0,
                                  INTERP_CUBIC)
            eng.set_static(128, 128, flat_bg=0.0)
            out = []
            for config in (0, 12):
                eng.set_render_config(config)
                ph = torch.empty((frames, 128, 128), dtype=torch.float32, device="cuda")
                adu = torch.empty((frames, 128, 128), dtype=torch.uint16, device="cuda")
                best = 1e9
                for _ in range(6):
                    eng.set_render_timing(True)
                    eng.render_frames_dev(dem, dfr, frames, cam, 5, ph, adu)
                    best = min(best, eng.render_pass_times()[0]["contributions"])
                eng.set_render_timing(False)
                out.append(ph.cpu().numpy().view(np.uint32))
                times[name] = best
            assert np.array_equal(*out), name
    assert times["steep"] <= 1.45 * times["slow"], times


def test_batches_of_about_one_size_share_the_scratch():
    """Two-pass batches that grow by a few emitters at a time stay in the first one's scratch: no allocation, and so no
    wait for one, between them."""
    import torch
    from insiliscope_b200 import Engine
    rng = np.random.default_rng(37)
    half, os_ = 16, 4
    n = 2 * half * os_ + 1
    with Engine(0) as eng:
        eng.kernel_set_planes(0, rng.uniform(0.0, 1e-4, (3, n, n)).astype(np.float32), os_, 25.0, INTERP_CUBIC)
        eng.set_static(128, 128, flat_bg=5.0)
        eng.set_render_config(12)
        free = []
        for count in (32000, 32001, 32100, 32600, 32900, 20000, 32900):
            em = np.zeros(count, EMITTER_DTYPE)
            em["x_px"], em["y_px"] = rng.uniform(0.0, 127.0, (2, count))
            em["photons"], em["plane"] = 1000.0, rng.integers(0, 3, count)
            per = np.full(200, count // 200)
            per[0] += count - int(per.sum())
            dem, dfr = (torch.from_numpy(t.view(np.uint8)).cuda() for t in (em, frames_table(per)))
            ph = torch.empty((200, 128, 128), dtype=torch.float32, device="cuda")
            eng.render_frames_dev(dem, dfr, 200, None, 5, ph)
            del dem, dfr, ph
            free.append(torch.cuda.mem_get_info()[0])
        assert len(set(free[1:])) == 1, free


@pytest.mark.parametrize("per", [30, 300])
@pytest.mark.parametrize("halo", [0.0, 2e-4])
def test_wide_gather_tiles_at_ragged_edges(engine, per, halo):
    """Frames enough for two and (with more emitters than are staged at once) four tiles a CTA, three pixels wider than a
    whole number of either: the one-pass form's bits, with and without a halo cut, some frames empty."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(per)
    half, os_, w, h = 5, 3, 131, 61
    n = 2 * half * os_ + 1
    y, x = np.mgrid[0:n, 0:n] - (n - 1) / 2.0
    plane = (1.0 + (x * x + y * y) / 20.0) ** -1.5
    engine.kernel_set_planes(0, np.repeat((plane / plane.sum())[None], 3, 0).astype(np.float32), os_, 25.0, INTERP_CUBIC)
    if halo:
        engine.kernel_set_halo(0, halo)
    counts = rng.poisson(per, 12 * sms // 10)
    counts[::7] = 0
    counts[1::7] *= 2
    em = np.zeros(int(counts.sum()), EMITTER_DTYPE)
    em["x_px"] = rng.uniform(-half - 1.0, w + half, len(em))
    em["y_px"] = rng.uniform(-half - 1.0, h + half, len(em))
    em["photons"], em["plane"] = rng.uniform(1.0, 3000.0, len(em)), rng.integers(0, 3, len(em))
    engine.set_static(w, h, flat_bg=7.0)
    cam = CameraParams(gain=2.0, read_noise_e=1.5)
    dem, dfr = (torch.from_numpy(t.view(np.uint8)).cuda() for t in (em, frames_table(counts)))
    out = {}
    try:
        for config in (0, 12, 13, 14):
            engine.set_render_config(config)
            ph = torch.empty((len(counts), h, w), dtype=torch.float32, device="cuda")
            adu = torch.empty((len(counts), h, w), dtype=torch.uint16, device="cuda")
            engine.render_frames_dev(dem, dfr, len(counts), cam, 5, ph, adu)
            out[config] = ph.cpu().numpy().view(np.uint32), adu.cpu().numpy()
    finally:
        engine.set_render_config(0)
        if halo:
            engine.kernel_set_halo(0, 0.0)
    for config in (12, 13, 14):
        assert np.array_equal(out[config][0], out[0][0]) and np.array_equal(out[config][1], out[0][1]), config
