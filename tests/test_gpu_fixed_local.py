"""Two properties of the fixed-point kernels that whole-field tolerances cannot
show: each link keeps the digits of its own size, and the forms of the link
update agree in everything that they write."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2, 2), (4, 6, 10, 14), (34, 2, 2, 6)]
S, B = (14, 8, 8, 4), (14, 8, 8, 8)  # 3,584 sites, rows of a link in three threads; 7,168, in one


def scaled(oracle, L, spread):
    """Unitary links times factors of e^-spread to e^spread: (links, factors)."""
    U = oracle.hot_start(list(L), 11)
    n = np.exp(np.random.RandomState(4).uniform(-spread, spread, size=U.shape[:2]))
    return U * n[:, :, None, None], n


def loops_through(L, n, steps):
    """Per link, the sum over the loops with `steps` (nu steps of a mu x nu loop)
    that hold it of the product of their links' factors."""
    n = n.reshape((4,) + L[::-1])

    def at(a, *moves):
        for mu, d in moves:
            a = np.roll(a, -d, axis=3 - mu)
        return a

    out = np.zeros_like(n)
    for mu in range(4):
        for nu in range(4):
            if mu == nu or (steps == 1 and nu < mu):
                continue
            links = [(mu, ()), (mu, ((nu, steps),))]
            for k in range(steps):
                links += [(nu, ((nu, k),)), (nu, ((mu, 1), (nu, k)))]
            value = np.ones(L[::-1])
            for d, moves in links:
                value = value * at(n[d], *moves)
            for d, moves in links:
                out[d] += at(value, *[(m, -k) for m, k in moves])
    return out.reshape(4, -1)


@pytest.mark.parametrize("coefficients", [(3.0, 0.0), (3.648, -0.1655), (0.0, 1.0)])
@pytest.mark.parametrize("L", SIZES)
def test_forces_to_each_links_own_size(pkg, oracle, L, coefficients):
    """Links off the group by factors e^-3 .. e^3: forces from 1e-5 to 1e5, each
    right to 1e-13 of the norms of the products that enter it."""
    Uh, n = scaled(oracle, L, 3)
    U = pkg.gauge_configuration(L, start="cold").from_host(Uh)
    action = pkg.GaugeAction(U)
    for c, loop in zip(coefficients, ("plaquette", "rectangular")):
        pkg.push_(action, c, loop)
    F = pkg.gauge_momenta(U)
    pkg.md_force_(F, action, U)
    ref = oracle.force_loops(list(L), Uh, *coefficients)
    size = sum(abs(c) * loops_through(L, n, s) for c, s in zip(coefficients, (1, 2)))
    assert (np.abs(F.to_host() - ref).max(axis=-1) <= 1e-13 * size).all()


@pytest.mark.parametrize("coefficients", [(0.0, 1.0), (1e-8, 1.0), (1.0, 1e-8)])
@pytest.mark.parametrize("L", SIZES)
def test_a_small_coefficient_leaves_the_other_term_its_digits(pkg, oracle, L, coefficients):
    """Factors of e^-20 .. e^20: plaquette staples that dwarf the rectangle ones,
    but for their coefficient."""
    Uh, n = scaled(oracle, L, 20)
    U = pkg.gauge_configuration(L, start="cold").from_host(Uh)
    action = pkg.GaugeAction(U)
    for c, loop in zip(coefficients, ("plaquette", "rectangular")):
        pkg.push_(action, c, loop)
    F = pkg.gauge_momenta(U)
    pkg.md_force_(F, action, U)
    ref = oracle.force_loops(list(L), Uh, *coefficients)
    size = sum(abs(c) * loops_through(L, n, s) for c, s in zip(coefficients, (1, 2)))
    assert (np.abs(F.to_host() - ref).max(axis=-1) <= 1e-13 * size).all()


@pytest.mark.parametrize("L", SIZES)
def test_the_adjoint_of_no_smearing_is_the_derivative_itself(pkg, oracle, L):
    """rho = 0 on links off the group by e^-5 .. e^5: what rho multiplies is up to
    e^10 times larger."""
    Uh, _ = scaled(oracle, L, 5)
    U = pkg.gauge_configuration(L, start="cold").from_host(Uh)
    net = pkg.CovNeuralnet(U)
    pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.0))
    rng = np.random.RandomState(2)
    d = rng.normal(size=Uh.shape) + 1j * rng.normal(size=Uh.shape)
    D = pkg.Gaugefields4D(U.ctx, pkg._lib.GF_MAT64).from_host(d)
    _, history, _ = pkg.calc_smearedU(U, net)
    got = pkg.back_prop(D, net, history, U).to_host()
    assert np.abs(got - d).max() <= 1e-15 * np.abs(d).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("reunit", [False, True])
@pytest.mark.parametrize("kind", ["unitary", "scaled", "weak"])
def test_update_forms_write_the_same(pkg, oracle, kind, reunit, precision):
    """The link update also writes what the next force reads: the fixed-point copy
    of the links (plain form) or their fp32 shadow (mixed). A lattice and its
    repetition, on either side of the size where the update changes its form, go
    through the same trajectory, bitwise."""
    if kind == "weak":
        U = pkg.gauge_configuration(S, start="cold")
        action = pkg.GaugeAction(U)
        pkg.push_(action, 3.0, "plaquette")
        pkg.update_gaugefields_(U, pkg.gaussian_momenta(U, seed=2), 1e-5, pkg.md_driver(U, action, steps=1))
        Uh = U.to_host()
    else:
        Uh, _ = scaled(oracle, S, 0.3 if kind == "scaled" else 0.0)
    Ph = 0.3 * np.random.RandomState(8).normal(size=Uh.shape[:2] + (8,))
    out = []
    for L, k in ((S, 1), (B, 2)):
        U = pkg.gauge_configuration(L, start="cold").from_host(np.tile(Uh, (1, k, 1, 1)))
        P = pkg.gauge_momenta(U).from_host(np.tile(Ph, (1, k, 1)))
        action = pkg.GaugeAction(U)
        pkg.push_(action, 3.0, "plaquette")
        drv = pkg.md_driver(U, action, steps=3, trajectory_length=0.3, reunitarize=reunit, precision=precision)
        pkg.md_trajectory_(U, P, drv)
        out.append((U.to_host(), P.to_host()))
    for small, big in zip(*out):
        assert np.isfinite(small).all()
        assert np.array_equal(big, np.concatenate([small, small], axis=1))
