"""The Poisson-likelihood gradient on the B200 (FP32 forward, adjoint kernel) against the float64 oracle's adjoint
and float64 central differences (h = 1e-4 max(1, |theta|)): <= 1e-4 relative; the NLL and expected counts within
1e-5."""
import numpy as np
import pytest
import torch

from insiliscope_b200 import IscuError
from insiliscope_b200.nll import NllModel, NllSpec, poisson_nll
from insiliscope_b200.workloads import nll_counts, nll_rois
from oracle.nll_oracle import NllSpec as OSpec, expected, gradient, nll, tables

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem(engine):
    spec = NllSpec()
    model = NllModel(engine, spec)
    prob = nll_rois(seed=7, frames=4, per_frame=24, spec=spec)
    counts = nll_counts(engine, model, prob)
    return model, prob, counts, OSpec(), tables(OSpec())


def _dev(prob, counts):
    return (torch.from_numpy(prob.params).cuda(), torch.from_numpy(prob.frame).cuda(),
            torch.from_numpy(prob.bg).cuda(), counts)


def test_counts_are_poisson_of_expected(problem):
    model, prob, counts, ospec, t = problem
    mu = expected(ospec, prob.params_true.astype(np.float64), prob.frame, prob.bg_true.astype(np.float64),
                  prob.zern_true, t)
    k = counts.cpu().numpy().astype(np.float64)
    assert np.all(k == np.round(k)) and k.min() >= 0
    # the counts scatter about the expectation as Poisson draws do
    z = (k - mu) / np.sqrt(mu)
    assert abs(z.mean()) < 0.05 and 0.9 < z.std() < 1.1


def test_forward_matches_oracle(problem):
    model, prob, counts, ospec, t = problem
    p, fr, bg, k = _dev(prob, counts)
    value, mu, _ = model.evaluate(p, fr, bg, prob.zern, k, want_mu=True)
    pd = prob.params.astype(np.float64)
    want_mu = expected(ospec, pd, prob.frame, prob.bg.astype(np.float64), prob.zern, t)
    got = mu.cpu().numpy()
    assert np.max(np.abs(got - want_mu)) <= 1e-5 * np.max(want_mu)
    want = nll(ospec, pd, prob.frame, prob.bg.astype(np.float64), prob.zern, k.cpu().numpy(), t)
    assert abs(value - want) <= 1e-5 * abs(want)


def test_gradient_matches_oracle_adjoint_and_central_differences(problem):
    model, prob, counts, ospec, t = problem
    p, fr, bg, k = _dev(prob, counts)
    _, _, (gp, gb, gz) = model.evaluate(p, fr, bg, prob.zern, k, grad=True)
    gp, gb, gz = gp.cpu().numpy().astype(np.float64), gb.cpu().numpy(), gz.cpu().numpy()
    pd, bd, kd = prob.params.astype(np.float64), prob.bg.astype(np.float64), k.cpu().numpy().astype(np.float64)
    _, wp, wb, wz = gradient(ospec, pd, prob.frame, bd, prob.zern, kd, t)
    for col in range(4):
        scale = np.max(np.abs(wp[:, col]))
        assert np.max(np.abs(gp[:, col] - wp[:, col])) <= 1e-4 * scale, col
    assert np.max(np.abs(gb - wb)) <= 1e-4 * np.max(np.abs(wb))
    assert np.max(np.abs(gz - wz)) <= 1e-4 * np.max(np.abs(wz))
    # central differences of the float64 NLL on a seeded subset
    rng = np.random.default_rng(3)

    def fd(f, x, i):
        h = 1e-4 * max(1.0, abs(x.flat[i]))
        xp, xm = x.copy(), x.copy()
        xp.flat[i] += h
        xm.flat[i] -= h
        return (f(xp) - f(xm)) / (2 * h)

    for i in rng.choice(pd.size, 12, replace=False):
        d = fd(lambda P: nll(ospec, P, prob.frame, bd, prob.zern, kd, t), pd, i)
        assert abs(gp.flat[i] - d) <= 1e-4 * max(abs(d), 1e-3 * np.max(np.abs(wp[:, i % 4]))), i
    for j in rng.choice(len(prob.zern), 4, replace=False):
        d = fd(lambda Z: nll(ospec, pd, prob.frame, bd, Z, kd, t), prob.zern.copy(), j)
        assert abs(gz[j] - d) <= 1e-4 * max(abs(d), 1e-3 * np.max(np.abs(wz))), j
    d = fd(lambda B: nll(ospec, pd, prob.frame, B, prob.zern, kd, t), bd, 1)
    assert abs(gb[1] - d) <= 1e-4 * abs(d)


def test_autograd_function(problem):
    model, prob, counts, ospec, t = problem
    p, fr, bg, k = _dev(prob, counts)
    p = p.clone().requires_grad_(True)
    bg = bg.clone().requires_grad_(True)
    z = torch.tensor(prob.zern, dtype=torch.float64, requires_grad=True)
    loss = poisson_nll(model, p, bg, z, k, fr)
    (2.0 * loss).backward()
    _, _, (gp, gb, gz) = model.evaluate(p, fr, bg, prob.zern, k, grad=True)
    assert torch.allclose(p.grad, 2.0 * gp, rtol=1e-6, atol=0)
    assert torch.allclose(bg.grad.double(), 2.0 * gb, rtol=1e-6)
    assert torch.allclose(z.grad, 2.0 * gz.cpu(), rtol=1e-12)


def test_bad_frame_reported(problem):
    model, prob, counts, _, _ = problem
    p, fr, bg, k = _dev(prob, counts)
    fr = fr.clone()
    fr[5] = 99
    with pytest.raises(IscuError):
        model.evaluate(p, fr, bg, prob.zern, k)


@pytest.mark.parametrize("roi,n", [(64, 3), (32, 700), (16, 5), (8, 5), (4, 5), (2, 5), (1, 1)])
def test_sample_groupings_match_oracle(engine, roi, n):
    """Every grouping of the 64 x 64 samples into pixels (1 to 64 samples per pixel and axis) and more emitters than
    CTAs: expected counts within 1e-5 of their maximum, each gradient within 1e-4 of its largest entry."""
    kw = dict(roi=roi, os=64 // roi)
    ospec = OSpec(**kw)
    t = tables(ospec)
    model = NllModel(engine, NllSpec(**kw))
    rng = np.random.default_rng(roi)
    c = roi / 2.0
    params = np.column_stack([c + rng.uniform(-0.2, 0.2, (n, 2)) * min(roi, 8), rng.uniform(-400, 400, n),
                              rng.uniform(800, 3000, n)]).astype(np.float32)
    frame = rng.integers(0, 3, n).astype(np.int32)
    bg = rng.uniform(5, 20, 3).astype(np.float32)
    zern = rng.normal(0.0, 0.03, len(ospec.noll))
    pd, bd = params.astype(np.float64), bg.astype(np.float64)
    want_mu = expected(ospec, pd, frame, bd, zern, t)
    counts = rng.poisson(want_mu * rng.uniform(0.8, 1.2, (n, 1, 1))).astype(np.float32)
    value, wp, wb, wz = gradient(ospec, pd, frame, bd, zern, counts.astype(np.float64), t)
    dev = [torch.from_numpy(a).cuda() for a in (params, frame, bg)]
    k = torch.from_numpy(counts).cuda()
    got, mu, g = model.evaluate(*dev, zern, k, grad=True, want_mu=True)
    fwd, mu0, _ = model.evaluate(*dev, zern, k, want_mu=True)
    assert np.max(np.abs(mu.cpu().numpy() - want_mu)) <= 1e-5 * np.max(want_mu)
    assert torch.equal(mu, mu0) and abs(fwd - got) <= 1e-12 * abs(got)
    assert abs(got - value) <= 1e-5 * abs(value)
    for have, want in ((g[0].cpu().numpy(), wp), (g[1].cpu().numpy()[None].T, wb[:, None]),
                       (g[2].cpu().numpy()[:, None], wz[:, None])):
        for col in range(want.shape[1]):
            assert np.max(np.abs(have[:, col] - want[:, col])) <= 1e-4 * np.max(np.abs(want[:, col])), col
    model.close()


def test_autograd_forms(problem):
    """The autograd function's paths: no gradient wanted (the likelihood alone, the same value), Zernike coefficients on
    the device and on the host in either precision, a scaled loss, a second backward, a differentiated backward, and
    an input changed in place in between, which autograd refuses."""
    model, prob, counts, ospec, t = problem
    p, fr, bg, k = _dev(prob, counts)
    want, _, (gp, gb, gz) = model.evaluate(p, fr, bg, prob.zern, k, grad=True)
    with torch.no_grad():
        quiet = poisson_nll(model, p.clone().requires_grad_(True), bg, torch.from_numpy(prob.zern), k, fr)
    assert not quiet.requires_grad and abs(float(quiet) - want) <= 1e-12 * abs(want)
    for device, dtype in (("cuda", torch.float64), ("cuda", torch.float32), ("cpu", torch.float64), ("cpu", torch.float32)):
        z = torch.tensor(prob.zern, dtype=dtype, device=device, requires_grad=True)
        q = p.clone().requires_grad_(True)
        b = bg.clone().requires_grad_(True)
        zval = z.detach().double().cpu().numpy()
        _, _, (wp, wb, wz) = model.evaluate(p, fr, bg, zval, k, grad=True)
        loss = poisson_nll(model, q, b, z, k, fr)
        (0.3 * loss).backward(retain_graph=True)
        (0.7 * loss).backward()
        assert loss.dtype == torch.float64 and loss.dim() == 0 and loss.device == q.device
        assert z.grad.dtype == dtype and z.grad.device.type == device
        assert torch.allclose(q.grad, wp, rtol=1e-6, atol=0)
        assert torch.allclose(b.grad.double(), wb, rtol=1e-6)
        assert torch.allclose(z.grad.double().cpu(), wz.cpu(), rtol=1e-6)
    s = torch.tensor(2.0, dtype=torch.float64, device="cuda", requires_grad=True)
    q = p.clone().requires_grad_(True)
    g, = torch.autograd.grad(s * poisson_nll(model, q, bg, torch.from_numpy(prob.zern), k, fr), q, create_graph=True)
    d, = torch.autograd.grad(g.sum(), s)
    assert torch.allclose(d, gp.double().sum(), rtol=1e-5)
    q = p.clone().requires_grad_(True)
    loss = poisson_nll(model, q, bg, torch.from_numpy(prob.zern), k, fr)
    with torch.no_grad():
        q.add_(1.0)
    with pytest.raises(RuntimeError):
        loss.backward()


def test_gradients_to_a_float_ulp(engine):
    """Each gradient of 1,200 ROIs against the float64 oracle: within 2^-23 of its 2-norm, the place value of the float32
    that the field is formed in (a sine or cosine 2^-21 off in the pupil alone takes the shared sums past it)."""
    ospec = OSpec(roi=32, os=2)
    t = tables(ospec)
    model = NllModel(engine, NllSpec(roi=32, os=2))
    rng = np.random.default_rng(23)
    n = 1200
    params = np.column_stack([rng.uniform(14.5, 17.5, (n, 2)), rng.uniform(-500, 500, n),
                              2000.0 * np.exp(0.5 * rng.standard_normal(n))]).astype(np.float32)
    frame = (np.arange(n) // 300).astype(np.int32)
    bg = rng.uniform(5, 20, 4).astype(np.float32)
    zern = rng.normal(0.0, 0.03, len(ospec.noll))
    truth = params.astype(np.float64) + np.column_stack([rng.normal(0, 0.3, (n, 2)), rng.normal(0, 50, n),
                                                         params[:, 3] * rng.normal(0, 0.1, n)])
    counts = rng.poisson(expected(ospec, truth, frame, 1.1 * bg.astype(np.float64), zern + 0.01, t)).astype(np.float32)
    _, *want = gradient(ospec, params.astype(np.float64), frame, bg.astype(np.float64), zern, counts.astype(np.float64), t)
    dev = [torch.from_numpy(a).cuda() for a in (params, frame, bg)]
    _, _, got = model.evaluate(*dev, zern, torch.from_numpy(counts).cuda(), grad=True)
    for have, w in zip(got, want):
        have = have.cpu().numpy().astype(np.float64)
        assert np.linalg.norm(have - w) <= 2.0 ** -23 * np.linalg.norm(w)
    model.close()
