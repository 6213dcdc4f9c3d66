"""GPU parity of the fixed-point kernels (gf_fixed.cu) at the sizes and on the
links where they can go wrong: fewer links than a block, a last block and a
last tile that are nearly empty, links whose exponents differ (not unitary,
over many orders of magnitude), and a NaN.

Tolerances: 1e-13 of the largest entry, two orders above fp64 rounding of the
sums involved (the oracle's own).
"""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import exact_exp_oracle  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2, 2), (2, 4, 2, 6), (6, 2, 10, 2), (4, 6, 10, 14), (34, 2, 2, 6)]
TOL = 1e-13
LARGE = (48, 48, 32, 32)  # 9 2^18 sites, more than 2^21


def start(pkg, oracle, L, kind):
    """Unitary links, or links scaled by random powers: (device field, host copy)."""
    Uh = oracle.hot_start(list(L), 11)
    if kind == "scaled":
        rng = np.random.RandomState(4)
        Uh *= np.exp(rng.uniform(-3, 3, size=Uh.shape[:2]))[:, :, None, None]
    U = pkg.gauge_configuration(L, start="cold")
    U.from_host(Uh)
    return U, Uh


def close(got, ref, tol=TOL):
    assert np.abs(got - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("kind", ["unitary", "scaled"])
@pytest.mark.parametrize("L", SIZES)
def test_wilson_force(pkg, oracle, L, kind):
    U, Uh = start(pkg, oracle, L, kind)
    F = pkg.gauge_momenta(U)
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    pkg.md_force_(F, action, U)
    ref = oracle.force(list(L), Uh, 6.0)
    close(F.to_host(), ref)
    # P += eps F keeps what P holds
    pkg.update_momenta_(F, U, 0.25, pkg.md_driver(U, action, steps=1))
    close(F.to_host(), 1.25 * ref)


def test_wilson_force_with_a_nan(pkg, oracle):
    L = (4, 4, 4, 6)
    U, Uh = start(pkg, oracle, L, "unitary")
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    ref = oracle.force(list(L), Uh, 6.0)
    Uh[2, 37, 1, 1] = np.nan
    U.from_host(Uh)
    F = pkg.gauge_momenta(U)
    pkg.md_force_(F, action, U)
    got = F.to_host()
    hit = np.isnan(got).any(axis=-1)
    # the link itself and the 18 links that share a plaquette with it
    assert hit.sum() == 19 and hit[2, 37]
    close(got[~hit], ref[~hit])


@pytest.mark.parametrize("kind", ["unitary", "scaled"])
@pytest.mark.parametrize("L", SIZES)
def test_plaquette_and_rectangles(pkg, oracle, L, kind):
    U, Uh = start(pkg, oracle, L, kind)
    for got, ref in ((pkg.calculate_Plaquette(U), oracle.plaquette(list(L), Uh)),
                     (pkg.rectangle_sum(U), oracle.rectangle_sum(list(L), Uh))):
        # of the sum of the loops' norms, which bounds what rounding sees
        size = np.abs(Uh).max() ** 6 * 18 * np.prod(L)
        assert abs(got - ref) <= TOL * size


@pytest.mark.parametrize("kind", ["unitary", "scaled"])
@pytest.mark.parametrize("coefficients", [(3.648, -0.1655), (-0.25, 4.0), (0.0, 1.0), (1.5, 0.0)])
@pytest.mark.parametrize("L", SIZES)
def test_rectangle_force(pkg, oracle, L, kind, coefficients):
    U, Uh = start(pkg, oracle, L, kind)
    action = pkg.GaugeAction(U)
    pkg.push_(action, coefficients[0], "plaquette")
    pkg.push_(action, coefficients[1], "rectangular")
    F = pkg.gauge_momenta(U)
    pkg.md_force_(F, action, U)
    close(F.to_host(), oracle.force_loops(list(L), Uh, *coefficients))


def general(pkg, U, L, spread):
    """A dS/dUbar whose matrices differ in size by up to `spread` orders of magnitude."""
    rng = np.random.RandomState(8)
    V = int(np.prod(L))
    D = rng.normal(size=(4, V, 3, 3)) + 1j * rng.normal(size=(4, V, 3, 3))
    D *= 10.0 ** rng.uniform(-spread, 0, size=(4, V))[:, :, None, None]
    d = pkg.Gaugefields4D(U.ctx, pkg._lib.GF_MAT64)
    return d.from_host(D), D


# |Q| from 0.3 to about 6: every scale of the exponential's series that a stack meets
@pytest.mark.parametrize("rho", [0.0, 0.1, 0.45, 1.0])
@pytest.mark.parametrize("L", SIZES)
def test_stout_forward_and_backward(pkg, exact_exp_oracle, L, rho):
    oracle = exact_exp_oracle
    U, Uh = start(pkg, oracle, L, "unitary")
    net = pkg.CovNeuralnet(U)
    for _ in range(2):
        pkg.push_(net, pkg.STOUT_Layer("plaquette", rho))
    Ubar, history, _ = pkg.calc_smearedU(U, net)
    close(Ubar.to_host(), oracle.stout_forward(list(L), Uh, [rho, rho]), 1e-12)
    d, D = general(pkg, U, L, 2)
    got = pkg.back_prop(d, net, history, U).to_host()
    close(got, oracle.stout_backward(list(L), Uh, [rho, rho], D)[0], 1e-11)


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("c_rect", [0.0, -0.2])
@pytest.mark.parametrize("L", SIZES)
def test_stout_force(pkg, exact_exp_oracle, L, c_rect, recompute):
    oracle = exact_exp_oracle
    U, Uh = start(pkg, oracle, L, "unitary")
    net = pkg.CovNeuralnet(U)
    for rho in (0.1, 0.15, 0.05):
        pkg.push_(net, pkg.STOUT_Layer("plaquette", rho))
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    pkg.push_(action, c_rect, "rectangular")
    drv = pkg.md_driver(U, action, steps=1, smearing=net, recompute=recompute)
    P = pkg.update_momenta_(pkg.gauge_momenta(U), U, 1.0, drv)
    close(P.to_host(), oracle.stout_force_loops(list(L), Uh, [0.1, 0.15, 0.05], 3.0, c_rect), 1e-11)


def test_stout_with_links_of_different_exponents(pkg, exact_exp_oracle):
    """Links off the group by factors 0.6 .. 1.7: exponents 0 and 1 side by side in every sum."""
    oracle = exact_exp_oracle
    L = (4, 6, 2, 8)
    Uh = oracle.hot_start(list(L), 21)
    Uh *= np.random.RandomState(2).uniform(0.6, 1.7, size=Uh.shape[:2])[:, :, None, None]
    U = pkg.gauge_configuration(L, start="cold")
    U.from_host(Uh)
    net = pkg.CovNeuralnet(U)
    pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.05))
    Ubar, history, _ = pkg.calc_smearedU(U, net)
    close(Ubar.to_host(), oracle.stout_forward(list(L), Uh, [0.05]), 1e-12)
    d, D = general(pkg, U, L, 6)
    close(pkg.back_prop(d, net, history, U).to_host(), oracle.stout_backward(list(L), Uh, [0.05], D)[0], 1e-11)


def test_stout_with_a_nan(pkg, oracle):
    L = (4, 4, 4, 6)
    U, Uh = start(pkg, oracle, L, "unitary")
    ref = oracle.stout_forward(list(L), Uh, [0.1])
    Uh[1, 50, 0, 2] = np.nan
    U.from_host(Uh)
    got = pkg.smear(U, pkg.stout_smearing(U)).to_host()
    hit = np.isnan(got).any(axis=(-1, -2))
    assert hit.sum() == 19 and hit[1, 50]
    close(got[~hit], ref[~hit], 1e-11)


@pytest.mark.parametrize("reunit", [False, True])
@pytest.mark.parametrize("eps", [0.05, 1.0, -3.0])
@pytest.mark.parametrize("L", SIZES)
def test_link_update(pkg, exact_exp_oracle, L, eps, reunit):
    """|eps P| up to 7 and links off the group by factors 0.5 .. 2."""
    oracle = exact_exp_oracle
    Uh = oracle.hot_start(list(L), 31)
    Uh *= np.random.RandomState(6).uniform(0.5, 2.0, size=Uh.shape[:2])[:, :, None, None]
    U = pkg.gauge_configuration(L, start="cold")
    U.from_host(Uh)
    P = pkg.gaussian_momenta(U, seed=5)
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    drv = pkg.md_driver(U, action, steps=1, reunitarize=reunit)
    pkg.update_gaugefields_(U, P, eps, drv)
    oracle.link_update(list(L), Uh, P.to_host(), eps)
    if reunit:
        oracle.normalize(list(L), Uh)
    close(U.to_host(), Uh, 1e-12)


def test_link_update_keeps_bad_values_where_they_are(pkg, exact_exp_oracle):
    """A NaN momentum, a NaN link and a zero link: those links only are not finite."""
    oracle = exact_exp_oracle
    L = (4, 4, 4, 6)
    Uh = oracle.hot_start(list(L), 31)
    Ph = np.random.RandomState(3).normal(size=(4, 384, 8))
    ref = Uh.copy()
    oracle.link_update(list(L), ref, Ph.copy(), 0.1)
    oracle.normalize(list(L), ref)
    Ph[0, 5, 3] = np.inf
    Uh[1, 60, 2, 0] = np.nan
    Uh[3, 100] = 0.0
    U = pkg.gauge_configuration(L, start="cold")
    U.from_host(Uh)
    P = pkg.gauge_momenta(U).from_host(Ph)
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    pkg.update_gaugefields_(U, P, 0.1, pkg.md_driver(U, action, steps=1))
    got = U.to_host()
    hit = ~np.isfinite(got).all(axis=(-1, -2))
    assert sorted(zip(*np.nonzero(hit))) == [(0, 5), (1, 60), (3, 100)]
    close(got[~hit], ref[~hit], 1e-12)


@pytest.mark.parametrize("L", SIZES + [(8, 8, 16, 18)])
def test_sums_of_few_and_many_blocks(pkg, oracle, L):
    """A sum whose last block adds up the partials and one that needs the
    second kernel (8 x 8 x 16 x 18: 3,456 plaquette items), twice over: bitwise
    repeatable, and P P against numpy."""
    U, Uh = start(pkg, oracle, L, "unitary")
    p = [pkg.calculate_Plaquette(U) for _ in range(3)]
    r = [pkg.rectangle_sum(U) for _ in range(3)]
    assert len(set(p)) == 1 and len(set(r)) == 1
    assert abs(p[0] - oracle.plaquette(list(L), Uh)) <= 1e-13 * abs(18 * np.prod(L))
    assert abs(r[0] - oracle.rectangle_sum(list(L), Uh)) <= 1e-13 * abs(36 * np.prod(L))
    P = pkg.gaussian_momenta(U, seed=3)
    k = (P.to_host() ** 2).sum()
    assert abs(P * P - k) <= 1e-13 * k


@pytest.mark.parametrize("L", [(4, 6, 10, 14), (34, 2, 2, 6), (14, 8, 8, 8)])
@pytest.mark.parametrize("c_rect", [0.0, -0.1])
@pytest.mark.parametrize("reunit", [False, True])
def test_drivers_copy_equals_a_fresh_conversion(pkg, oracle, L, c_rect, reunit):
    """The fixed-point copy that the link update keeps for the next force is
    bitwise what converting the stored links gives: the one-call trajectory and
    the one stepped through md_step_ (which converts each time) agree bitwise
    where they take the same steps (PQP: no half steps merge for one step)."""
    out = []
    for whole in (True, False):
        U, _ = start(pkg, oracle, L, "unitary")
        P = pkg.gaussian_momenta(U, seed=9)
        action = pkg.GaugeAction(U)
        pkg.push_(action, 3.0, "plaquette")
        pkg.push_(action, c_rect, "rectangular")
        drv = pkg.md_driver(U, action, steps=1, trajectory_length=0.3, integrator=pkg.PQP(), reunitarize=reunit)
        if whole:
            pkg.md_trajectory_(U, P, drv)
        else:
            pkg.md_step_(pkg.PQP(), U, P, 0.3, drv)
        out.append((U.to_host(), P.to_host()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("eps", [0.05, -3.0])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("reunit", [False, True])
@pytest.mark.parametrize("kind", ["unitary", "scaled"])
def test_link_update_does_not_depend_on_the_lattice(pkg, oracle, kind, reunit, precision, eps):
    """Up to 6144 sites the update runs a link's rows in three threads, beyond
    in one. A link's result depends on nothing else, so a small lattice's links
    and momenta, repeated over one of 7168 sites, come out bitwise the same,
    NaNs included."""
    S, B = (14, 2, 4, 2), (14, 8, 8, 8)
    n, N = int(np.prod(S)), int(np.prod(B))
    assert n <= 6144 < N
    _, Uh = start(pkg, oracle, S, kind)
    Ph = np.random.RandomState(8).normal(size=(4, n, 8))
    Uh[1, 7] = 0.0
    Uh[2, 9, 1, 1] = np.nan
    Uh[3, 11, 1] = Uh[3, 11, 0]  # rank two: row 2 vanishes under the projection
    Ph[0, 13, 4] = np.inf
    reps = -(-N // n)
    got = []
    for L, k in ((S, 1), (B, reps)):
        V = int(np.prod(L))
        U = pkg.gauge_configuration(L, start="cold")
        U.from_host(np.tile(Uh, (1, k, 1, 1))[:, :V])
        P = pkg.gauge_momenta(U).from_host(np.tile(Ph, (1, k, 1))[:, :V])
        action = pkg.GaugeAction(U)
        pkg.push_(action, 3.0, "plaquette")
        drv = pkg.md_driver(U, action, steps=1, reunitarize=reunit, precision=precision)
        pkg.update_gaugefields_(U, P, eps, drv)
        got.append(U.to_host())
    want = np.tile(got[0], (1, reps, 1, 1))[:, :N]
    assert np.array_equal(got[1], want, equal_nan=True)


@pytest.mark.parametrize("c_rect,recompute", [(0.0, True), (-0.1, False)])
def test_double_float_stacks_of_large_lattices(pkg, c_rect, recompute):
    """Beyond 2^21 sites the double-float form's stacks run through the
    double-float tables, up to there in fixed point. 1e-11 between the forms'
    forces and 5e-13 between their energies, as at the other sizes."""
    U = pkg.gauge_configuration(LARGE, start="hot", seed=3)
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    pkg.push_(action, c_rect, "rectangular")
    net = pkg.CovNeuralnet(U)
    for rho in (0.1, 0.08):
        pkg.push_(net, pkg.STOUT_Layer("plaquette", rho))
    force, energy = [], []
    for precision in ("fp64", "dfloat"):
        P = pkg.gauge_momenta(U)
        drv = pkg.md_driver(U, action, steps=1, smearing=net, precision=precision, recompute=recompute)
        pkg.update_momenta_(P, U, 1.0, drv)
        energy.append(pkg.md_hamiltonian(U, P, drv))
        force.append(P.to_host())
    assert np.linalg.norm(force[1] - force[0]) <= 1e-11 * np.linalg.norm(force[0])
    assert abs(energy[1] - energy[0]) <= 5e-13 * abs(energy[0])


def test_double_float_adjoint_of_large_lattices(pkg):
    """The same for the pull-back of a caller's dS/dUbar, and 1e-11 a link for
    dS/drho, a sum over the links."""
    from gaugefields_gb300 import _lib
    from gaugefields_gb300.api import _StoutStack
    V = int(np.prod(LARGE))
    U = pkg.gauge_configuration(LARGE, start="hot", seed=3)
    rng = np.random.RandomState(5)
    few = rng.randn(4, 9 << 10, 3, 3) + 1j * rng.randn(4, 9 << 10, 3, 3)
    D = pkg.Gaugefields4D(U.ctx, _lib.GF_MAT64)
    D.from_host(np.tile(few, (1, V // few.shape[1], 1, 1)))
    net = pkg.CovNeuralnet(U)
    pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.1))
    grad, drho = [], []
    for precision in ("fp64", "dfloat"):
        stack = _StoutStack(U.ctx, [0.1], precision)
        _lib.check(_lib.load().gf_stout_forward(U.ctx.h, stack.h, U.field.h, None), U.ctx.h)
        out = pkg.Gaugefields4D(U.ctx, _lib.GF_MAT64)
        _lib.check(_lib.load().gf_stout_backward(U.ctx.h, stack.h, D.field.h, out.field.h), U.ctx.h)
        grad.append(out.to_host())
        drho.append(pkg.get_parameter_derivatives(D, net, U, precision)[0])
    assert np.linalg.norm(grad[1] - grad[0]) <= 1e-11 * np.linalg.norm(grad[0])
    assert abs(drho[1] - drho[0]) <= 1e-11 * 4 * V


def test_without_memory_for_the_copy(pkg):
    """The fixed-point copy of the links is what goes when memory is short: a
    field takes its place, and the calls that made it read the links as they
    are. The same
    numbers to 1e-13, and the copy is back when there is memory again."""
    from gaugefields_gb300 import _lib
    torch = pytest.importorskip("torch")
    U = pkg.gauge_configuration((24, 24, 24, 24), start="hot", seed=11)
    V, P = U.similar(), pkg.gauge_momenta(U)
    P0 = pkg.gaussian_momenta(U, seed=3)
    wilson, loops = pkg.GaugeAction(U), pkg.GaugeAction(U)
    pkg.push_(wilson, 3.0, "plaquette")
    pkg.push_(loops, 3.0, "plaquette")
    pkg.push_(loops, -0.1, "rectangular")
    net = pkg.CovNeuralnet(U)
    pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.1))
    smeared = pkg.md_driver(U, loops, steps=1, smearing=net, precision="mixed")

    def launches():
        n = ctypes.c_longlong()
        _lib.check(_lib.load().gf_launch_count(ctypes.byref(n)))
        return n.value

    def numbers():
        out = [pkg.calculate_Plaquette(U), pkg.rectangle_sum(U), pkg.md_hamiltonian(U, P0, smeared)]
        for action in (wilson, loops):
            pkg.md_force_(P, action, U)
            out.append(P.to_host())
        pkg.substitute_U_(V, U)
        P.from_host(P0.to_host())
        r = pkg.md_trajectory_(V, P, pkg.md_driver(U, wilson, steps=1, trajectory_length=0.1))
        out += [V.to_host(), P.to_host(), r.initial_hamiltonian, r.final_hamiltonian]
        pkg.substitute_U_(V, U)
        pkg.flow_(V, pkg.gradient_flow(V, steps=1, step_size=0.01))
        out.append(V.to_host())
        return out

    def plaquette_launches():
        before = launches()
        pkg.calculate_Plaquette(U)
        return launches() - before

    ref = numbers()
    usual = plaquette_launches()
    size = 4 * 24 ** 4 * 144
    filler = torch.empty(torch.cuda.mem_get_info()[0] - size // 2, dtype=torch.uint8, device="cuda")
    try:
        W = U.similar()  # takes the copy's place
        assert plaquette_launches() == usual - 1  # no conversion before the sum
        got = numbers()
        del W
    finally:
        del filler
        torch.cuda.empty_cache()
    for a, b in zip(got, ref):
        close(np.asarray(a), np.asarray(b))
    for a, b in zip(numbers(), ref):
        assert np.array_equal(np.asarray(a), np.asarray(b))


@pytest.mark.parametrize("warm", [False, True])
def test_forces_and_smearing_in_a_graph(pkg, warm):
    """Calls that read nothing back can be captured, with the fixed-point copy
    in place or (lattices whose copy a first call allocates) without one, and a
    replay follows the links."""
    from gaugefields_gb300 import _lib
    from gaugefields_gb300.api import _StoutStack
    torch = pytest.importorskip("torch")
    L = (16, 16, 16, 16)
    U = pkg.gauge_configuration(L, start="hot", seed=5)
    W = pkg.gauge_configuration(L, start="hot", seed=6)
    wilson = pkg.GaugeAction(U)
    pkg.push_(wilson, 3.0, "plaquette")
    stack, top, F = _StoutStack(U.ctx, [0.1], "fp64"), U.similar(), pkg.gauge_momenta(U)
    host = W.to_host()

    def calls():
        pkg.md_force_(F, wilson, U)
        _lib.check(_lib.load().gf_stout_forward(U.ctx.h, stack.h, U.field.h, top.field.h), U.ctx.h)

    stream = torch.cuda.Stream()
    U.ctx.set_stream(stream.cuda_stream)
    U.ctx.torch_stream = stream  # alive as long as the context
    if warm:
        calls()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        calls()
    U.from_host(host)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    got = F.to_host(), top.to_host()
    calls()
    close(got[0], F.to_host())
    close(got[1], top.to_host())


@pytest.mark.parametrize("precision", ["fp64", "dfloat"])
def test_smeared_driver_calls_in_any_order(pkg, precision):
    """The context's stacks read the context's copy of whatever links a call
    is given; energies, forces and trajectories on two configurations in turn
    are bitwise those of fresh contexts."""
    L = (4, 6, 4, 8)

    def run(seeds):
        U = pkg.gauge_configuration(L, start="hot", seed=1)
        other = {k: pkg.gauge_configuration(L, start="hot", seed=k).to_host() for k in set(seeds)}
        action = pkg.GaugeAction(U)
        pkg.push_(action, 3.0, "plaquette")
        pkg.push_(action, -0.1, "rectangular")
        net = pkg.CovNeuralnet(U)
        pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.1))
        pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.08))
        drv = pkg.md_driver(U, action, steps=2, trajectory_length=0.2, smearing=net, precision=precision)
        out = []
        for k in seeds:
            U.from_host(other[k])
            P = pkg.gaussian_momenta(U, seed=k)
            h = pkg.md_hamiltonian(U, P, drv)
            pkg.calculate_Plaquette(U)
            r = pkg.md_trajectory_(U, P, drv)
            pkg.update_momenta_(P, U, 0.1, drv)
            out.append((h, r.initial_hamiltonian, r.final_hamiltonian, U.to_host(), P.to_host()))
        return out

    turns = run([3, 5, 3])
    for got, k in zip(turns, [3, 5, 3]):
        want = run([k])[0]
        assert got[0] == got[1]
        assert all(np.array_equal(np.asarray(a), np.asarray(b)) for a, b in zip(got, want))


@pytest.mark.parametrize("levels,recompute", [(1, False), (2, True)])
def test_smeared_force_forms_its_top_derivative_either_way(pkg, levels, recompute):
    """Above 40,000 sites dS/dUbar of the Wilson action is formed in a kernel
    of its own, below in the adjoint. A lattice of 2 x 20,480 sites that
    repeats one of 20,480 along T has the same force, up to the exponents that
    the two paths choose: 1e-14 of the largest entry."""
    S, B = (16, 10, 8, 16), (16, 10, 8, 32)
    n = int(np.prod(S))
    assert n < 40000 < 2 * n
    Uh = pkg.gauge_configuration(S, start="hot", seed=2).to_host()
    out = []
    for L, k in ((S, 1), (B, 2)):
        U = pkg.gauge_configuration(L, start="cold")
        U.from_host(np.tile(Uh, (1, k, 1, 1)))
        action = pkg.GaugeAction(U)
        pkg.push_(action, 3.0, "plaquette")
        net = pkg.CovNeuralnet(U)
        for rho in (0.1, 0.08)[:levels]:
            pkg.push_(net, pkg.STOUT_Layer("plaquette", rho))
        P = pkg.gauge_momenta(U)
        pkg.update_momenta_(P, U, 1.0, pkg.md_driver(U, action, steps=1, smearing=net, recompute=recompute))
        out.append(P.to_host())
    close(out[1], np.tile(out[0], (1, 2, 1)), 1e-14)
