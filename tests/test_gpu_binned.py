"""The binned blink regime on the B200 (iscu_binned_*) against the float64 oracle (the linear convolution
BinnedBlinkRenderer computes) and the reference's own BinnedBlinkRenderer (float FFTs, oracle/_ref): the cell kernels
bit for bit (KernelWidefieldPsf's float64 block sums), the photon images within 1e-6 of the frame maximum of the
oracle and 5e-6 of the reference's (its float FFT's rounding), added into the caller's images."""
import numpy as np
import pytest

from insiliscope_b200 import BinnedRenderer, EMITTER_DTYPE, INTERP_CUBIC, frames_table
from oracle.oracle import binned_cell_kernels_f64, binned_gauss_kernel_f64, binned_render_f64
from test_binned_oracle import H, W, _req, binned_movie

pytestmark = pytest.mark.gpu


def _rel(got, want):
    return float(np.abs(got - want).max() / np.abs(want).max())


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8)).cuda()


def _render(r, em, fr, base):
    import torch
    img = torch.from_numpy(base.copy()).cuda()
    alone = torch.zeros_like(img)
    r.render_dev(_dev(em), _dev(fr), len(fr), img, alone)
    return img.cpu().numpy(), alone.cpu().numpy()


@pytest.mark.parametrize("upscale,halo", [(2, None), (4, 0.002), (1, None), (3, None)])
def test_kernel_regime(engine, reference, upscale, halo):
    k = reference.kernel(req=_req())
    size, nz, os_, _ = k.info()
    engine.kernel_set_planes(0, k.planes(), os_, 100.0, INTERP_CUBIC)
    radius2 = None
    if halo is not None:
        engine.kernel_set_halo(0, halo)
        k = k.halo(halo)
        radius2 = k.spans()[2]
    K, u, R = binned_cell_kernels_f64(k.planes(), os_, upscale, radius2)
    r = BinnedRenderer(engine, W, H, upscale, slot=0)
    assert (r.upscale, r.radius, r.planes) == (u, R, nz)
    assert np.array_equal(r.kernels(), K)
    em, fr = binned_movie(7 + upscale, 3, 60, nz)
    base = np.random.default_rng(1).random((len(fr), H, W)).astype(np.float32) * 10
    img, alone = _render(r, em, fr, base)
    want = binned_render_f64(K, u, R, em, fr, W, H)
    assert _rel(alone, want) <= 1e-6
    assert np.array_equal(img, base + alone)
    ref, _, _, _ = reference.binned_render(k, 0.0, W, H, upscale, em, fr)
    assert _rel(alone, ref) <= 5e-6
    r.close()
    if halo is not None:
        engine.kernel_set_halo(0, 0.0)


def test_gauss_regime(engine, reference):
    K, u, R = binned_gauss_kernel_f64(1.3, 3)
    r = BinnedRenderer(engine, W, H, 3, sigma_px=1.3)
    assert (r.upscale, r.radius, r.planes) == (u, R, 1)
    np.testing.assert_allclose(r.kernels(), K, rtol=1e-6, atol=0)
    em, fr = binned_movie(3, 2, 40, 1)
    _, alone = _render(r, em, fr, np.zeros((len(fr), H, W), np.float32))
    ref, _, _, _ = reference.binned_render(None, 1.3, W, H, 3, em, fr)
    assert _rel(alone, ref) <= 5e-6
    assert _rel(alone, binned_render_f64(K, u, R, em, fr, W, H)) <= 1e-6
    r.close()


def test_dense_frames_128(engine, reference):
    """Frames of the dense regime the reference picks binned for (2,000+ ON emitters on a 128 x 128 camera), the
    SMLM kernel geometry (oversampling 4, 49 planes), u = 2."""
    from insiliscope_b200.workloads import binned_dense
    mv = binned_dense(frames=6)
    k = reference.kernel(req=mv.psf)
    engine.kernel_set_planes(1, k.planes(), 4, mv.psf.z_step_nm, INTERP_CUBIC)
    r = BinnedRenderer(engine, mv.width, mv.height, mv.upscale, slot=1)
    K, u, R = binned_cell_kernels_f64(k.planes(), 4, mv.upscale)
    _, alone = _render(r, mv.emitters, mv.frames, np.zeros((len(mv.frames), mv.height, mv.width), np.float32))
    want = binned_render_f64(K, u, R, mv.emitters, mv.frames, mv.width, mv.height)
    assert _rel(alone, want) <= 1e-6
    r.close()


@pytest.mark.parametrize("half,os_,upscale,w,h,nz,signed", [
    (5, 4, 2, 70, 45, 3, False), (5, 4, 4, 33, 17, 5, False), (8, 2, 1, 130, 66, 3, False), (3, 3, 3, 43, 22, 3, False),
    (4, 4, 2, 64, 32, 3, True), (2, 1, 1, 5, 3, 3, False)])
def test_dense_kernel(engine, half, os_, upscale, w, h, nz, signed):
    """Frames of many emitters per plane (the kernel with the plane's samples in shared memory), tiles' edges and
    remainders, planes with negative samples, more emitters than its buffer: the oracle within 1e-6 of the maximum, and
    within a float's last place of the per-pixel kernel, which the same frames take among many empty ones."""
    rng = np.random.default_rng(half * 7 + upscale)
    n = 2 * half * os_ + 1
    planes = rng.random((nz, n, n)).astype(np.float32) / (n * n)
    planes[:, 0, :] = 0.0
    if signed:
        planes[1] -= 0.3 / (n * n)
    engine.kernel_set_planes(0, planes, os_, 100.0, INTERP_CUBIC)
    r = BinnedRenderer(engine, w, h, upscale, slot=0)
    counts = np.tile([2300, 0, 37, 411], 75)      # 300 frames: tiles for every SM
    total = int(counts.sum())
    em = np.zeros(total, EMITTER_DTYPE)
    em["x_px"] = rng.uniform(-half - 2.0, w + half + 2.0, total)
    em["y_px"] = rng.uniform(-half - 2.0, h + half + 2.0, total)
    em["photons"] = rng.uniform(-50.0, 2000.0, total)
    em["plane"] = rng.integers(0, nz + 1, total)
    fr = frames_table(counts)
    want = binned_render_f64(*binned_cell_kernels_f64(planes, os_, upscale), em, fr[:4], w, h)
    base = rng.random((len(fr), h, w)).astype(np.float32)
    img, alone = _render(r, em, fr, base)
    assert _rel(alone[:4], want) <= 1e-6
    assert np.array_equal(img, base + alone)
    pad = frames_table(np.concatenate([counts[:4], np.zeros(20000, np.int64)]))
    _, sparse = _render(r, em[:int(counts[:4].sum())], pad, np.zeros((len(pad), h, w), np.float32))
    assert np.all(np.abs(sparse[:4] - alone[:4]) <= 1.2e-7 * np.abs(alone[:4]))
    r.close()


def _dense_movie(engine, half, os_, upscale, w, h, nz, per, frames, seed=1, signed=0):
    """A renderer on a slowly falling stack (the first `signed` planes with negative samples) and a movie of even frames."""
    rng = np.random.default_rng(seed)
    n = 2 * half * os_ + 1
    y, x = np.mgrid[0:n, 0:n] - (n - 1) / 2.0
    planes = np.stack([(1.0 + (x * x + y * y) / (30.0 + z)) ** -1.5 for z in range(nz)])
    planes /= planes.sum(axis=(1, 2), keepdims=True)
    planes[:signed] -= 0.1 * planes[0].mean()
    engine.kernel_set_planes(0, planes.astype(np.float32), os_, 100.0, INTERP_CUBIC)
    em = np.zeros(per * frames, EMITTER_DTYPE)
    em["x_px"], em["y_px"] = rng.uniform(-0.5, w - 0.5, len(em)), rng.uniform(-0.5, h - 0.5, len(em))
    em["photons"] = 2000.0 * np.exp(0.5 * rng.standard_normal(len(em)))
    em["plane"] = rng.integers(0, nz, len(em))
    return BinnedRenderer(engine, w, h, upscale, slot=0), em, frames_table(np.full(frames, per))


def _render_ms(engine, r, em, fr):
    """One call's image and its time on the device (the best of five)."""
    import torch
    dem, dfr = (torch.from_numpy(a.view(np.uint8)).cuda() for a in (em, fr))
    img = torch.zeros((len(fr), r.height, r.width), dtype=torch.float32, device="cuda")
    best = 1e9
    with torch.cuda.stream(engine.torch_stream()):
        for _ in range(5):
            img.zero_()
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            r.render_dev(dem, dfr, len(fr), img, sync=False)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
    return img.cpu().numpy(), best


def test_signed_stacks_and_extreme_photons_take_no_detour(engine):
    """Dense frames of a stack with negative samples, and with an emitter here and there whose photons are no normal
    float: within 1e-6 of the oracle, the first in about the per-pixel kernel's time (twice the dense one's), the second
    in the dense one's."""
    args = (16, 4, 2, 128, 128, 20)
    r, em, fr = _dense_movie(engine, *args, 1200, 100)
    _, plain = _render_ms(engine, r, em, fr)
    odd = em.copy()
    odd["photons"][::300] = [1e-39, 1e-44, 1e-300, 1e-41] * (len(em) // 1200)
    img, extreme = _render_ms(engine, r, odd, fr)
    want = binned_render_f64(r.kernels().astype(np.float64), r.upscale, r.radius, odd, fr[:2], 128, 128)
    assert _rel(img[:2], want) <= 1e-6
    r.close()
    r, em, fr = _dense_movie(engine, *args, 1200, 100, signed=20)
    img, signed = _render_ms(engine, r, em, fr)
    want = binned_render_f64(r.kernels().astype(np.float64), r.upscale, r.radius, em, fr[:2], 128, 128)
    assert _rel(img[:2], want) <= 1e-6
    r.close()
    assert extreme <= 1.3 * plain and signed <= 2.4 * plain, (plain, extreme, signed)


def _order_movie(frames):
    """Frames of a 1, a 2^-24 and many 2^-54 photons in one cell, the large ones first and on the last plane: in event
    order the small ones are lost one after the other and the sum is float32's midpoint (1); by plane they come first and
    take it past (1 + 2^-23)."""
    per = 900
    em = np.zeros(per * frames, EMITTER_DTYPE)
    em["x_px"], em["y_px"] = 20.0, 20.0
    em["photons"], em["plane"] = 2.0 ** -54, np.arange(per * frames) % 2
    em["photons"][::per], em["photons"][1::per] = 1.0, 2.0 ** -24
    em["plane"][::per] = em["plane"][1::per] = 2
    return em, frames_table(np.full(frames, per))


def test_images_do_not_depend_on_the_batch(engine):
    """A frame's image is the event-order sum's, to the bit, whether its batch takes the dense kernel or the per-pixel one:
    frames built so that the order of the sum decides the rounding, and 100 frames of a movie."""
    planes = np.zeros((3, 5, 5), np.float32)
    planes[:, 2, 2] = 1.0
    engine.kernel_set_planes(0, planes, 1, 100.0, INTERP_CUBIC)
    r = BinnedRenderer(engine, 64, 48, 1, slot=0)
    em, fr = _order_movie(400)
    img, _ = _render_ms(engine, r, em, fr)
    want = np.zeros((48, 64), np.float32)
    want[20, 20] = 1.0
    assert np.array_equal(img[0], want) and all(np.array_equal(f, want) for f in img)
    r.close()
    r, em, fr = _dense_movie(engine, 8, 4, 2, 96, 80, 9, 700, 300, seed=3)
    whole, _ = _render_ms(engine, r, em, fr)
    for k in range(0, 100, 4):     # four frames at a time: too few for the dense kernel
        part, _ = _render_ms(engine, r, em, fr[k:k + 4])
        assert np.array_equal(part.view(np.uint32), whole[k:k + 4].view(np.uint32)), k
    r.close()


@pytest.mark.parametrize("half,os_,nz", [(60, 1, 500), (3, 1, 4), (100, 1, 3)])
def test_a_renderer_holds_its_kernels_once(engine, half, os_, nz):
    """The plane kernels, read back as the oracle has them, take the device memory of one copy (rows of whole 16 bytes)."""
    import torch
    rng = np.random.default_rng(half)
    n = 2 * half * os_ + 1
    planes = rng.random((nz, n, n)).astype(np.float32) / (n * n)
    engine.kernel_set_planes(0, planes, os_, 100.0, INTERP_CUBIC)
    before = torch.cuda.mem_get_info()[0]
    r = BinnedRenderer(engine, 64, 64, 1, slot=0)
    held = before - torch.cuda.mem_get_info()[0]
    assert held <= 1.05 * r.kernels().nbytes + (4 << 20), (held, r.kernels().nbytes)
    assert np.array_equal(r.kernels(), binned_cell_kernels_f64(planes, os_, 1)[0])
    r.close()


@pytest.mark.parametrize("half,os_,upscale,nz,w,h", [(8, 4, 4, 49, 70, 33), (9, 4, 4, 3, 33, 18), (16, 4, 4, 5, 40, 20),
                                                     (16, 4, 2, 49, 130, 40), (5, 2, 2, 300, 65, 33)])
def test_dense_kernel_geometries(engine, half, os_, upscale, nz, w, h):
    """The dense kernel (as its own query says) at kernels as wide as its row pitches allow (R = 32 and 64), just beyond
    the first (one staged kernel instead of two), and more planes than the sort scans at once: the oracle within 1e-6,
    and the per-pixel kernel's bits, which a few frames alone take."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    probe, _, _ = _dense_movie(engine, half, os_, upscale, w, h, nz, 1, 1)
    tiles = -(-w // (128 // probe.upscale)) * -(-h // (64 // probe.upscale))
    frames = -(-2 * sms // tiles)
    per = probe.dense_from(1 << 30, frames) + 5
    probe.close()
    assert per > 5
    r, em, fr = _dense_movie(engine, half, os_, upscale, w, h, nz, per, frames, seed=half)
    assert 0 < r.dense_from(len(em), frames) <= per and r.dense_from(2 * per, 2) == 0
    whole, _ = _render_ms(engine, r, em, fr)
    want = binned_render_f64(r.kernels().astype(np.float64), r.upscale, r.radius, em, fr[:2], w, h)
    assert _rel(whole[:2], want) <= 1e-6
    for k in (0, frames // 2, frames - 2):
        part, _ = _render_ms(engine, r, em, fr[k:k + 2])
        assert np.array_equal(part.view(np.uint32), whole[k:k + 2].view(np.uint32)), k
    r.close()


def test_each_frame_by_its_own_count(engine):
    """Sparse frames whose emitters are the head of a long array take the time that they take with an array of their own,
    and the image; dense and sparse frames in one call are each the per-pixel kernel's bits."""
    r, em, fr = _dense_movie(engine, 16, 4, 2, 128, 128, 49, 100, 20000)
    assert r.dense_from(len(em), 200) > 0 and r.dense_from(100 * 200, 200) == 0
    own, short = _render_ms(engine, r, em[:100 * 200], fr[:200])
    img, long_ = _render_ms(engine, r, em, fr[:200])
    assert np.array_equal(img.view(np.uint32), own.view(np.uint32))
    assert long_ <= 1.3 * short, (short, long_)
    counts = np.where(np.arange(120) % 3 == 0, 3000, 60)
    mixed = frames_table(counts)
    least = r.dense_from(int(counts.sum()), 120)
    assert 60 < least <= 3000
    whole, _ = _render_ms(engine, r, em[:int(counts.sum())], mixed)
    for k in range(0, 24, 2):
        part, _ = _render_ms(engine, r, em[:int(counts.sum())], mixed[k:k + 2])
        assert np.array_equal(part.view(np.uint32), whole[k:k + 2].view(np.uint32)), k
    r.close()
