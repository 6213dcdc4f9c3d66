"""Stout layers whose exponents are large, as large rho or links off the group
make them: the adjoint is that of the forward pass at any size.

Reference in fp64 by the eigenvectors of X (exp(Q) = exp(iX)): the derivative of
the exponential takes Lambda_ab to i exp(i (x_a + x_b) / 2) sinc((x_a - x_b) / 2)
Lambda_ab. Rounding of X, 1e-16 |X|, turns phases by as much, and the pull-back
carries rho times it: 1e-13 max(1, |X|) of the largest entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = (4, 2, 6, 4)
V = int(np.prod(L))


def dag(a):
    return np.swapaxes(a, -1, -2).conj()


def at(a, mu, d):
    return np.roll(a, -d, axis=3 - mu)


def ta(m):
    a = (m - dag(m)) / 2
    return a - np.trace(a, axis1=-2, axis2=-1)[..., None, None] / 3 * np.eye(3)


def staples(u, rho):
    c = np.zeros_like(u)
    for mu in range(4):
        for nu in range(4):
            if nu != mu:
                c[mu] += u[nu] @ at(u[mu], nu, 1) @ dag(at(u[nu], mu, 1))
                c[mu] += at(dag(u[nu]) @ u[mu] @ at(u[nu], mu, 1), nu, -1)
    return rho * c


def level(u, rho, d):
    """Smeared links, dS/dU of dS = 2 Re tr(dUbar d), and the largest |X|."""
    c = staples(u, rho)
    x, v = np.linalg.eigh(-1j * ta(c @ dag(u)))
    e = (v * np.exp(1j * x)[..., None, :]) @ dag(v)
    s, h = (x[..., :, None] + x[..., None, :]) / 2, (x[..., :, None] - x[..., None, :]) / 2
    lam = dag(v) @ (u @ d) @ v
    grad = v @ (1j * np.exp(1j * s) * np.sinc(h / np.pi) * lam) @ dag(v)
    y = ta(-1j * grad)
    z, out = rho * (dag(u) @ y), d @ e + dag(y @ c)
    for mu in range(4):
        for nu in range(4):
            if nu == mu:
                continue
            a, b, f, zr = u[nu], at(u[mu], nu, 1), at(u[nu], mu, 1), z[mu]
            out[nu] += b @ dag(f) @ zr
            out[mu] += at(dag(f) @ zr @ a, nu, -1)
            out[nu] += at(dag(zr @ a @ b), mu, -1)
            b, zr = u[mu], at(z[mu], nu, 1)
            out[nu] += dag(b @ f @ zr)
            out[mu] += f @ zr @ dag(a)
            out[nu] += at(zr @ dag(a) @ b, mu, -1)
    return e @ u, out, np.abs(x).max()


def layout(m):
    return np.ascontiguousarray(np.swapaxes(m.reshape(4, V, 3, 3), -1, -2))


# |X| up to 0.2, 2, 3.6, 6, 12, 24, 120 and 2e4
@pytest.mark.parametrize("rho", [0.05, 0.5, 0.9, 1.5, 3.0, 6.0, 30.0, 5000.0])
@pytest.mark.parametrize("store", [True, False])
def test_forward_and_adjoint(pkg, oracle, rho, store):
    from gaugefields_gb300 import _lib
    from gaugefields_gb300.api import _StoutStack
    U = pkg.gauge_configuration(L, start="hot", seed=4)
    u = np.swapaxes(U.to_host(), -1, -2).reshape((4,) + L[::-1] + (3, 3))
    rng = np.random.RandomState(5)
    d = rng.normal(size=u.shape) + 1j * rng.normal(size=u.shape)
    want, grad, x = level(u, rho, d)
    stack, top, out = _StoutStack(U.ctx, [rho], "fp64", store=store), U.similar(), pkg.Gaugefields4D(U.ctx, _lib.GF_MAT64)
    D = pkg.Gaugefields4D(U.ctx, _lib.GF_MAT64).from_host(layout(d))
    call = _lib.load()
    _lib.check(call.gf_stout_forward(U.ctx.h, stack.h, U.field.h, top.field.h), U.ctx.h)
    _lib.check(call.gf_stout_backward(U.ctx.h, stack.h, D.field.h, out.field.h), U.ctx.h)
    assert 3 * rho < x < 6 * rho
    tol = 1e-13 * max(1.0, x)
    assert np.abs(top.to_host() - layout(want)).max() <= tol
    assert np.abs(out.to_host() - layout(grad)).max() <= tol * np.abs(grad).max()


def test_a_force_far_off_the_group(pkg, oracle):
    """Links scaled by 3: staples times links by 81, |X| about 30. The force of
    the smeared links is the derivative of their energy."""
    U = pkg.gauge_configuration(L, start="hot", seed=4)
    U.from_host(3.0 * U.to_host())
    u = np.swapaxes(U.to_host(), -1, -2).reshape((4,) + L[::-1] + (3, 3))
    top, _, x = level(u, 0.1, np.zeros_like(u))
    d = oracle.dsdu_loops(list(L), layout(top), 3.0, 0.0)
    _, grad, _ = level(u, 0.1, np.swapaxes(d, -1, -2).reshape(u.shape))
    a = -ta(u @ grad).reshape(4, V, 3, 3) / 3
    want = np.stack([2 * a[..., 0, 1].imag, 2 * a[..., 0, 1].real, (a[..., 0, 0] - a[..., 1, 1]).imag,
                     2 * a[..., 0, 2].imag, 2 * a[..., 0, 2].real, 2 * a[..., 1, 2].imag, 2 * a[..., 1, 2].real,
                     -np.sqrt(3) * a[..., 2, 2].imag], axis=-1)
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    net = pkg.CovNeuralnet(U)
    pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.1))
    P = pkg.update_momenta_(pkg.gauge_momenta(U), U, 1.0, pkg.md_driver(U, action, steps=1, smearing=net))
    assert 20 < x < 80
    assert np.abs(P.to_host() - want).max() <= 1e-13 * x * np.abs(want).max()


def test_exponents_without_digits_give_no_number(pkg):
    """|X| beyond 2^53: the phases are lost in the rounding of X. Smeared links,
    gradients and updated links are NaN and not some unitary matrix."""
    for rho, links in ((1e20, "hot"), (1e20, "weak")):
        U = pkg.gauge_configuration(L, start="hot", seed=4)
        if links == "weak":
            x = U.to_host()
            U.from_host(np.eye(3) + 1e-3 * (x - dag(x)))
        net = pkg.CovNeuralnet(U)
        pkg.push_(net, pkg.STOUT_Layer("plaquette", rho))
        top, history, _ = pkg.calc_smearedU(U, net)
        D = pkg.Gaugefields4D(U.ctx, pkg._lib.GF_MAT64).from_host(U.to_host())
        assert np.isnan(top.to_host()).all()
        assert np.isnan(pkg.back_prop(D, net, history, U).to_host()).any(axis=(-1, -2)).all()
    for size in (L, (14, 8, 8, 8)):
        for start in ("hot", "cold"):
            U = pkg.gauge_configuration(size, start=start, seed=4)
            action = pkg.GaugeAction(U)
            pkg.push_(action, 3.0, "plaquette")
            for reunit in (False, True):
                W = U.similar().from_host(U.to_host())
                pkg.update_gaugefields_(W, pkg.gaussian_momenta(U, seed=1), 1e20,
                                        pkg.md_driver(U, action, steps=1, reunitarize=reunit))
                assert np.isnan(W.to_host()).all()
