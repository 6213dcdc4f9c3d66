"""Links whose small parts carry the physics: near the identity (weak fields,
the first steps after a cold start), near the diagonal, near an SU(2) subgroup.
In fp64 each entry has its own digits, so the small parts of forces and updated
links are right relative to themselves; the kernels must keep that.

Tolerance 1e-13 of the largest small part: chains of up to a dozen products
whose terms are themselves of the small parts' size. References: the oracle
where its formulas keep small parts (products and Taylor exponentials), else
extended precision here.
"""
import functools

import numpy as np
import pytest

from test_gpu_parity import exact_exp_oracle  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu

TOL = 1e-13
# below and above the sizes at which the kernels' forms change (2048, 6144 and
# 40,000 sites): the smallest, and repetitions of it along T
SMALL, TIMES = (2, 4, 6, 2), (1, 22, 66, 420)
KINDS = ["weak-3", "weak-6", "weak-9", "diagonal", "su2", "mixed"]
LD, CLD = np.longdouble, np.clongdouble


def dag(a):
    return np.swapaxes(a, -1, -2).conj()


def hermitian(rng, shape):
    a = rng.normal(size=shape + (3, 3)) + 1j * rng.normal(size=shape + (3, 3))
    a = (a + dag(a)) / 2
    return a - np.trace(a, axis1=-2, axis2=-1)[..., None, None] / 3 * np.eye(3)


def expi(x):
    """exp(i x) by its series, each entry to its own digits when x is small."""
    x = 1j * x.astype(CLD)
    out, term = np.zeros_like(x) + np.eye(3), np.zeros_like(x) + np.eye(3)
    for n in range(1, 60):
        term = term @ x / LD(n)
        out = out + term
    return out


@functools.lru_cache(None)
def start(kind, seed=1):
    """Matrices [mu, lex, i, j]."""
    rng = np.random.RandomState(seed)
    shape = (4, int(np.prod(SMALL)))
    eps = 10.0 ** int(kind[4:]) if kind.startswith("weak") else 1e-7
    u = expi(eps * hermitian(rng, shape))
    if kind == "diagonal":
        u = expi(np.einsum("mva,ab->mvab", hermitian(rng, shape).diagonal(axis1=-2, axis2=-1).real, np.eye(3))) @ u
    if kind == "su2":
        h = hermitian(rng, shape)
        h[..., 2, :] = h[..., :, 2] = 0
        h[..., 0, 0] -= np.trace(h, axis1=-2, axis2=-1) / 2
        h[..., 1, 1] = -h[..., 0, 0]
        u = expi(h) @ u
    if kind == "mixed":  # two generic links among weak ones
        for mu, x in ((0, 7), (2, 50)):
            u[mu, x] = expi(hermitian(rng, ()))
    return u.astype(np.complex128)


# the numbers that are small because of the kind
def parts(a, kind):
    a = np.asarray(a)
    if a.shape[-1] == 8:  # su(3) coefficients
        own = {"diagonal": [0, 1, 3, 4, 5, 6], "su2": [3, 4, 5, 6]}.get(kind, list(range(8)))
        return a[..., own]
    off = ~np.eye(3, dtype=bool)
    if kind == "su2":
        off = np.zeros((3, 3), dtype=bool)
        off[2, :2] = off[:2, 2] = True
    picked = a[..., off]
    out = [picked.real, picked.imag]
    if kind.startswith("weak"):
        out.append(a[..., range(3), range(3)].imag)
    return np.concatenate(out, axis=-1)


def check(got, ref, kind, tol=TOL):
    got, ref = np.asarray(got, dtype=ref.dtype), np.asarray(ref)
    g, r = parts(got, kind), parts(ref, kind)
    off, size = float(np.abs(got - ref).max()), float(np.abs(ref).max())
    assert off <= 1e-13 * max(1.0, size)
    if kind == "mixed":
        # where all is weak: its own size counts
        weak = np.abs(r).max(axis=-1) < 1e-4
        assert weak.any()
        g, r = g[weak], r[weak]
    off, size = float(np.abs(g - r).max()), float(np.abs(r).max())
    assert off <= tol * size


def layout(m):
    """[mu, lex, i, j] <-> the library's [mu, lex, j, i]."""
    return np.ascontiguousarray(np.swapaxes(m, -1, -2))


def device(pkg, m, times):
    """The links, repeated along T."""
    U = pkg.gauge_configuration(SMALL[:3] + (SMALL[3] * times,), start="cold")
    return U.from_host(np.tile(layout(m), (1, times, 1, 1)))


def one(a, times):
    """One of the repetitions of a result, all of them the same."""
    a = a.reshape((4, times, -1) + a.shape[2:])
    assert np.array_equal(a, np.broadcast_to(a[:, :1], a.shape))
    return a[:, 0]


@pytest.mark.parametrize("times", TIMES)
@pytest.mark.parametrize("kind", KINDS)
def test_forces(pkg, oracle, kind, times):
    m = start(kind)
    U = device(pkg, m, times)
    P = pkg.gauge_momenta(U)
    for coefficients in ((3.0, 0.0), (3.648, -0.1655)):
        action = pkg.GaugeAction(U)
        for c, loop in zip(coefficients, ("plaquette", "rectangular")):
            pkg.push_(action, c, loop)
        pkg.md_force_(P, action, U)
        ref = oracle.force_loops(list(SMALL), layout(m), *coefficients)
        check(one(P.to_host(), times), ref, kind)
        pkg.update_momenta_(P, U, 0.5, pkg.md_driver(U, action, steps=1))
        check(one(P.to_host(), times), 1.5 * ref, kind)


@pytest.mark.parametrize("times", TIMES)
@pytest.mark.parametrize("kind", KINDS)
def test_sums(pkg, oracle, kind, times):
    m = start(kind)
    U = device(pkg, m, times)
    size = 18 * np.prod(SMALL) * times
    assert abs(pkg.calculate_Plaquette(U) - times * oracle.plaquette(list(SMALL), layout(m))) <= 1e-13 * size
    assert abs(pkg.rectangle_sum(U) - times * oracle.rectangle_sum(list(SMALL), layout(m))) <= 2e-13 * size


@pytest.mark.parametrize("reunit", [False, True])
@pytest.mark.parametrize("times", TIMES)
@pytest.mark.parametrize("kind", KINDS)
def test_link_update(pkg, kind, times, reunit):
    m = start(kind)
    eps = 10.0 ** int(kind[4:]) if kind.startswith("weak") else 1e-7
    x = eps * hermitian(np.random.RandomState(3), m.shape[:2])
    p = np.stack([2 * x[..., 0, 1].real, -2 * x[..., 0, 1].imag, (x[..., 0, 0] - x[..., 1, 1]).real,
                  2 * x[..., 0, 2].real, -2 * x[..., 0, 2].imag, 2 * x[..., 1, 2].real, -2 * x[..., 1, 2].imag,
                  -np.sqrt(3) * x[..., 2, 2].real], axis=-1)
    U = device(pkg, m, times)
    P = pkg.gauge_momenta(U).from_host(np.tile(p, (1, times, 1)))
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    pkg.update_gaugefields_(U, P, 0.5, pkg.md_driver(U, action, steps=1, reunitarize=reunit))
    check(layout(one(U.to_host(), times)), expi(0.5 * x) @ m, kind)


@pytest.mark.parametrize("times", TIMES[:3])
@pytest.mark.parametrize("kind", KINDS[:3])
def test_cold_start(pkg, kind, times):
    """The identity is no small part; what a momentum makes of it is."""
    eps = 10.0 ** int(kind[4:])
    U = pkg.gauge_configuration(SMALL[:3] + (SMALL[3] * times,), start="cold")
    x = eps * hermitian(np.random.RandomState(3), (4, int(np.prod(SMALL))))
    p = np.zeros(x.shape[:2] + (8,))
    p[..., 0], p[..., 1], p[..., 3] = 2 * x[..., 0, 1].real, -2 * x[..., 0, 1].imag, eps * x[..., 0, 0].real
    h = np.zeros(x.shape, dtype=np.complex128)
    h[..., 0, 1] = (p[..., 0] - 1j * p[..., 1]) / 2
    h[..., 0, 2] = p[..., 3] / 2
    h = h + dag(h)
    P = pkg.gauge_momenta(U).from_host(np.tile(p, (1, times, 1)))
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    pkg.update_gaugefields_(U, P, 1.0, pkg.md_driver(U, action, steps=1, reunitarize=False))
    got, ref = layout(one(U.to_host(), times)), expi(h)
    # two scales: (0, 1) of order eps and (0, 2) of order eps^2
    for el in ((0, 1), (0, 2), (2, 0)):
        assert np.abs(got[..., el[0], el[1]] - ref[..., el[0], el[1]]).max() <= \
            TOL * np.abs(ref[..., el[0], el[1]]).max()


@pytest.mark.parametrize("times", TIMES)
@pytest.mark.parametrize("kind", KINDS[:5])
def test_flow(pkg, exact_exp_oracle, kind, times):
    m = start(kind)
    U = device(pkg, m, times)
    pkg.flow_(U, pkg.gradient_flow(U, steps=2, step_size=0.02))
    ref = layout(m)
    exact_exp_oracle.flow(list(SMALL), ref, 0.02, 2)
    check(layout(one(U.to_host(), times)), layout(ref), kind, 2 * TOL)


# --- stout smearing in extended precision, on [mu, t, z, y, x, i, j] ---------
def grid(m):
    return m.astype(CLD).reshape((4,) + SMALL[::-1] + (3, 3))


def at(a, mu, d):
    return np.roll(a, -d, axis=3 - mu)


def ta(m):
    a = (m - dag(m)) / LD(2)
    return a - np.trace(a, axis1=-2, axis2=-1)[..., None, None] / LD(3) * np.eye(3)


def stout_level(u, rho):
    c = np.zeros_like(u)
    for mu in range(4):
        for nu in range(4):
            if nu == mu:
                continue
            c[mu] += u[nu] @ at(u[mu], nu, 1) @ dag(at(u[nu], mu, 1))
            down = dag(u[nu]) @ u[mu] @ at(u[nu], mu, 1)
            c[mu] += at(down, nu, -1)
    c = LD(rho) * c
    x = -1j * ta(c @ dag(u))
    return c, x, expi(x)


def stout_pull_back(u, rho, d):
    """dS/dU of dS = 2 Re tr(dUbar d)."""
    c, x, e = stout_level(u, rho)
    lam, power, grad, coef = u @ d, np.zeros_like(u) + np.eye(3), np.zeros_like(u), CLD(1)
    for n in range(1, 50):  # sum_n i^n / n! sum_k x^(n-1-k) lam x^k
        part = lam @ power if n == 1 else x @ part + lam @ power
        coef = coef * CLD(1j) / LD(n)
        grad, power = grad + coef * part, power @ x
    y = ta(-1j * grad)
    z, out = dag(u) @ y, d @ e + dag(y @ c)
    for mu in range(4):
        for nu in range(4):
            if nu == mu:
                continue
            a, b, f = u[nu], at(u[mu], nu, 1), at(u[nu], mu, 1)
            zr = LD(rho) * z[mu]
            out[nu] += b @ dag(f) @ zr
            out[mu] += at(dag(f) @ zr @ a, nu, -1)
            out[nu] += at(dag(zr @ a @ b), mu, -1)
            # the staple below, formed at x - nu
            a, b, f, zr = u[nu], u[mu], at(u[nu], mu, 1), at(LD(rho) * z[mu], nu, 1)
            out[nu] += dag(b @ f @ zr)
            out[mu] += f @ zr @ dag(a)
            out[nu] += at(zr @ dag(a) @ b, mu, -1)
    return out


def flat(a):
    return a.reshape(4, -1, 3, 3)


RHOS = (0.1, 0.08)


@functools.lru_cache(None)
def levels_of(kind):
    levels = [grid(start(kind))]
    for rho in RHOS:
        levels.append(stout_level(levels[-1], rho)[2] @ levels[-1])
    return levels


def thin_derivative(kind, d):
    for u, rho in zip(levels_of(kind)[-2::-1], RHOS[::-1]):
        d = stout_pull_back(u, rho, d)
    return flat(d)


def smearing(pkg, U):
    net = pkg.CovNeuralnet(U)
    for rho in RHOS:
        pkg.push_(net, pkg.STOUT_Layer("plaquette", rho))
    return net


@functools.lru_cache(None)
def pulled_back(kind):
    return thin_derivative(kind, grid(start(kind, 2) * 2.5))


@pytest.mark.parametrize("times", TIMES)
@pytest.mark.parametrize("kind", KINDS[:5])
def test_stout_forward_and_backward(pkg, kind, times):
    U = device(pkg, start(kind), times)
    net = smearing(pkg, U)
    Ubar, history, _ = pkg.calc_smearedU(U, net)
    check(layout(one(Ubar.to_host(), times)), flat(levels_of(kind)[-1]), kind)
    # a derivative of the links' own kind, as an action of them has
    d = layout(start(kind, 2) * 2.5)
    D = pkg.Gaugefields4D(U.ctx, pkg._lib.GF_MAT64).from_host(np.tile(d, (1, times, 1, 1)))
    got = one(pkg.back_prop(D, net, history, U).to_host(), times)
    check(layout(got), pulled_back(kind), kind, 2 * TOL)


_FORCES = {}


def smeared_force(oracle, kind, c_rect):
    """Momenta that the force of the smeared action adds in a unit of time."""
    if (kind, c_rect) not in _FORCES:
        top = layout(flat(levels_of(kind)[-1]).astype(np.complex128))
        d = thin_derivative(kind, grid(layout(oracle.dsdu_loops(list(SMALL), top, 3.0, c_rect))))
        a = -ta(flat(levels_of(kind)[0]) @ d) / LD(3)
        _FORCES[kind, c_rect] = np.stack(
            [2 * a[..., 0, 1].imag, 2 * a[..., 0, 1].real, (a[..., 0, 0] - a[..., 1, 1]).imag, 2 * a[..., 0, 2].imag,
             2 * a[..., 0, 2].real, 2 * a[..., 1, 2].imag, 2 * a[..., 1, 2].real,
             -np.sqrt(LD(3)) * a[..., 2, 2].imag], axis=-1)
    return _FORCES[kind, c_rect]


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("times", TIMES)
@pytest.mark.parametrize("kind", KINDS[:5])
def test_stout_force(pkg, oracle, kind, times, recompute):
    U = device(pkg, start(kind), times)
    for c_rect in (0.0, -0.2):
        action = pkg.GaugeAction(U)
        pkg.push_(action, 3.0, "plaquette")
        pkg.push_(action, c_rect, "rectangular")
        drv = pkg.md_driver(U, action, steps=1, smearing=smearing(pkg, U), recompute=recompute)
        P = pkg.update_momenta_(pkg.gauge_momenta(U), U, 1.0, drv)
        check(one(P.to_host(), times), smeared_force(oracle, kind, c_rect), kind, 4 * TOL)


@pytest.mark.parametrize("times", TIMES[:3])
@pytest.mark.parametrize("kind", KINDS[:3])
def test_trajectory(pkg, exact_exp_oracle, kind, times):
    """A weak field stays one along a trajectory with momenta of its size."""
    oracle = exact_exp_oracle
    m = start(kind)
    p = 10.0 ** int(kind[4:]) * np.random.RandomState(6).normal(size=m.shape[:2] + (8,))
    U = device(pkg, m, times)
    P = pkg.gauge_momenta(U).from_host(np.tile(p, (1, times, 1)))
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    drv = pkg.md_driver(U, action, steps=4, trajectory_length=0.4, reunitarize=False)
    pkg.md_trajectory_(U, P, drv)
    u = layout(m)
    oracle.md_trajectory(list(SMALL), u, p, 6.0, 0.4, 4)
    check(layout(one(U.to_host(), times)), layout(u), kind, 4 * TOL)
    check(one(P.to_host(), times), p, kind, 4 * TOL)
