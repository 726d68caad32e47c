"""Heaviside projection (ft = 3) on the device against the numpy restatement
of top3D125modCuda.m (oracle.prj/deta/dprj and its design loop)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def torch():
    import torch as _torch
    return _torch


def test_heaviside_matches_oracle_newton(oracle, gputo, torch):
    rng = np.random.default_rng(3)
    xt = np.clip(rng.beta(0.6, 2.5, 20000), 0.0, 1.0)
    volfrac, beta, eta0 = 0.15, 4.0, 0.4
    eta = eta0
    f = oracle.prj(xt, eta, beta).mean() - volfrac
    while abs(f) > 1e-6:
        eta = eta - f / oracle.deta(xt, eta, beta).mean()
        f = oracle.prj(xt, eta, beta).mean() - volfrac
    dev = dict(dtype=torch.float64, device="cuda")
    X = torch.as_tensor(xt, **dev)
    P, D = torch.empty_like(X), torch.empty_like(X)
    eta_g = gputo.heaviside_dev(X, P, volfrac, beta, eta0, D)
    assert abs(eta_g - eta) <= 1e-12 * abs(eta)
    np.testing.assert_allclose(P.cpu().numpy(), oracle.prj(xt, eta, beta), rtol=0, atol=1e-13)
    np.testing.assert_allclose(D.cpu().numpy(), oracle.dprj(xt, eta, beta), rtol=1e-12, atol=1e-12)
    Z = torch.empty_like(X)
    gputo.mul_dev(P, D, Z)
    np.testing.assert_allclose(Z.cpu().numpy(), P.cpu().numpy() * D.cpu().numpy(), rtol=0, atol=0)


@pytest.mark.parametrize("n", [5, 4097, 300001])
@pytest.mark.parametrize("beta", [0.5, 64.0, 400.0])
def test_projection_loop_sizes_and_betas(oracle, gputo, torch, n, beta):
    """Fewer elements than a CTA, a partial last pass, more than one pass; beta
    on the exponential and (above 300, and where it overflows) the direct
    formulas.  The sums differ from numpy's by rounding (1e-16 n^(1/2) at
    most), which the Newton steps carry into eta: 1e-12."""
    xt = np.random.default_rng(n).random(n)
    xt[:2] = 0.0, 1.0
    volfrac, eta0 = 0.4, 0.55
    eta = eta0
    for _ in range(60):
        f = oracle.prj(xt, eta, beta).mean() - volfrac
        if abs(f) <= 1e-6:
            break
        eta = eta - f / oracle.deta(xt, eta, beta).mean()
    converged = abs(f) <= 1e-6
    X = torch.as_tensor(xt, dtype=torch.float64, device="cuda")
    P = torch.empty_like(X)
    if not converged:   # no threshold gives this volume: the steps run into NaNs or the call says it did not converge
        try:
            gputo.heaviside_dev(X, P, volfrac, beta, eta0)
            assert torch.isnan(P).any()
        except gputo.GputoError as e:
            assert e.status == gputo.GPUTO_ERR_BREAKDOWN
        return
    eta_g = gputo.heaviside_dev(X, P, volfrac, beta, eta0)
    assert abs(eta_g - eta) <= 1e-12 * abs(eta)
    np.testing.assert_allclose(P.cpu().numpy(), oracle.prj(xt, eta, beta), rtol=0, atol=1e-12 * max(1.0, beta))


@pytest.mark.parametrize("beta", [1e-12, 1e-9, 1e-5, 0.01, 0.3, 0.49])
def test_projection_of_small_betas(oracle, gputo, torch, beta):
    """beta near zero, where the projection is the identity and tanh(beta (v - eta)) has to keep its relative
    accuracy.  The volume is that of eta = 0.45, so below 1e-3 the first threshold stays.  The mean of the projection is
    exact to a few 2^-53 on both sides: eta agrees to 1e-15 over its derivative."""
    xt = np.random.default_rng(17).random(60001)
    volfrac, eta0 = oracle.prj(xt, 0.45, beta).mean(), 0.55
    eta = eta0
    for _ in range(60):
        f = oracle.prj(xt, eta, beta).mean() - volfrac
        if abs(f) <= 1e-6:
            break
        eta = eta - f / oracle.deta(xt, eta, beta).mean()
    assert abs(f) <= 1e-6
    X = torch.as_tensor(xt, dtype=torch.float64, device="cuda")
    P = torch.empty_like(X)
    eta_g = gputo.heaviside_dev(X, P, volfrac, beta, eta0)
    if eta == eta0:
        assert eta_g == eta0
    else:
        assert abs(eta_g - eta) <= 1e-15 / abs(oracle.deta(xt, eta, beta).mean())
    # eight roundings of values up to 1, and a shift of eta moves a projected value by at most |beta| of it
    np.testing.assert_allclose(P.cpu().numpy(), oracle.prj(xt, eta, beta), rtol=0,
                               atol=2e-15 + abs(beta) * abs(eta_g - eta))


@pytest.mark.parametrize("beta", [0.5, 0.55, 1.0, 3.0])
def test_threshold_is_as_accurate_as_the_direct_formulas(gputo, torch, beta):
    """The threshold against the same Newton steps in 80 bits, 300 problems of 300 elements: its error is that of the
    direct formulas in 64 bits, times 1.6 for the spread of the two (2.4 at 0.5 from exponentials)."""
    def newton(v, volfrac, eta, real):
        v, volfrac, eta, b = v.astype(real), real(volfrac), real(eta), real(beta)
        for k in range(60):
            den = np.tanh(b * eta) + np.tanh(b * (1 - eta))
            f = ((np.tanh(b * eta) + np.tanh(b * (v - eta))) / den).astype(np.longdouble).mean() - volfrac
            if abs(f) <= 1e-6:
                return eta, k
            d = -b / np.sinh(b) / np.cosh(b * (v - eta)) ** 2 * np.sinh(v * b) * np.sinh((1 - v) * b)
            eta = real(eta - real(f) / real(d.astype(np.longdouble).mean()))

    rng = np.random.default_rng(23)
    err = {"here": [], "direct": []}
    for _ in range(300):
        v = 1 / (1 + np.exp(2 - 2.5 * rng.standard_normal(300)))
        want = rng.uniform(0.2, 0.7)
        volfrac = float(((np.tanh(beta * want) + np.tanh(beta * (v - want)))
                         / (np.tanh(beta * want) + np.tanh(beta * (1 - want)))).mean())
        eta, k = newton(v, volfrac, want + 0.05, np.longdouble)
        direct, k2 = newton(v, volfrac, want + 0.05, np.float64)
        X = torch.as_tensor(v, device="cuda")
        P = torch.empty_like(X)
        torch.cuda.synchronize()
        got = gputo.heaviside_dev(X, P, volfrac, beta, want + 0.05)
        assert k == k2
        err["here"].append(float(got - eta))
        err["direct"].append(float(direct - eta))
    rms = {q: np.sqrt(np.mean(np.square(e))) for q, e in err.items()}
    assert rms["here"] <= 1.6 * rms["direct"] + 2.0 ** -54   # and the rounding of eta itself


@pytest.mark.parametrize("n", [1, 700, 4097, 300001])
def test_oc_loop_sizes(oracle, gputo, torch, n):
    """The OC update on fewer elements than a CTA, a partial last pass and
    several passes: the multiplier's path is the numpy loop's (its start differs
    by rounding only)."""
    rng = np.random.default_rng(n)
    x, dc = rng.random(n), -np.exp(rng.standard_normal(n))
    dv = np.full(n, 1.0 / n)
    ref, lref = oracle.oc_update(x, dc, dv, 0.3, 0.2)
    X, D, V = (torch.as_tensor(a, dtype=torch.float64, device="cuda") for a in (x, dc, dv))
    out = torch.empty_like(X)
    lm = gputo.oc_update_dev(X, D, V, out, 0.3, 0.2)
    assert abs(lm - lref) <= 1e-13 * abs(lref)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=0, atol=1e-13)


def test_design_loop_with_projection_matches_oracle(oracle, gputo, torch):
    """Six iterations of the 32x16x16 cantilever with ft = 3 on the GPU against
    the oracle loop with the same settings: compliance history within 1e-6,
    design within 1e-6 max-abs, the same iteration counts within 1."""
    p = oracle.cantilever(32, 16, 16)
    cfg = oracle.DesignConfig(nl=3, tol=1e-9, maxit=200, iters=6, ft=3, volfrac=0.12)
    h = oracle.design_loop(p, cfg)
    F, fixed = gputo.cantilever(32, 16, 16)
    dl = gputo.DesignLoop(32, 16, 16, 3, F, fixed, gputo.hex8_stiffness(), volfrac=0.12, tol=1e-9, maxit=200,
                          ft=3, eta=0.4, beta=2.0)
    cs, nits = [], []
    for _ in range(6):
        info = dl.step()
        cs.append(info["c"])
        nits.append(info["nit"])
    np.testing.assert_allclose(cs, h["c"], rtol=1e-6)
    assert max(abs(a - b) for a, b in zip(nits, h["nit"])) <= 1
    assert np.abs(dl.xPhys.cpu().numpy() - h["xPhys"]).max() <= 1e-6
    assert np.abs(dl.x.cpu().numpy() - h["x"]).max() <= 1e-6


def test_design_loop_resume_is_seamless(gputo, torch, tmp_path):
    """Save after three ft = 3 iterations, resume in a fresh loop, run three
    more: the design and compliance match six uninterrupted iterations
    (the drivers' warm start, CrossWalk/crosswalk.m:135)."""
    F, fixed = gputo.cantilever(32, 16, 16)
    kw = dict(volfrac=0.12, tol=1e-9, maxit=200, ft=3, eta=0.4, beta=2.0)
    a = gputo.DesignLoop(32, 16, 16, 3, F, fixed, gputo.hex8_stiffness(), **kw)
    ca = [a.step()["c"] for _ in range(6)]
    b = gputo.DesignLoop(32, 16, 16, 3, F, fixed, gputo.hex8_stiffness(), **kw)
    for _ in range(3):
        b.step()
    path = tmp_path / "it3.gds"
    b.save(path, 3)
    c = gputo.DesignLoop(32, 16, 16, 3, F, fixed, gputo.hex8_stiffness(), volfrac=0.3, tol=1e-9, maxit=200,
                         ft=3, eta=0.5, beta=2.0)
    assert c.resume(path) == 3
    assert c.volfrac == 0.12 and c.eta == b.eta
    cc = [c.step()["c"] for _ in range(3)]
    np.testing.assert_allclose(cc, ca[3:], rtol=1e-9)
    assert np.abs(c.x.cpu().numpy() - a.x.cpu().numpy()).max() <= 1e-9
