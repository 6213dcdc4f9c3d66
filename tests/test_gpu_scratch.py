"""The context's scratch memory under pressure, under graph capture and with
several threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L24 = (24, 24, 24, 24)
COPY = 4 * (24 ** 4 // 32) * (9 * 512 + 128)  # bytes of the fixed-point copy of the links


def free_bytes(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def wilson(pkg, U):
    action = pkg.GaugeAction(U)
    pkg.push_(action, 3.0, "plaquette")
    return action


def test_an_idle_copy_gives_way_to_a_trajectory_that_keeps_none(pkg):
    """The mixed form's trajectory holds no fixed-point copy of the links, so
    one that an earlier plaquette left behind must not keep memory from it."""
    torch = pytest.importorskip("torch")

    def trajectory(idle_copy):
        U = pkg.gauge_configuration(L24, start="hot", seed=11)
        P = pkg.gaussian_momenta(U, seed=3)
        net = pkg.CovNeuralnet(U)
        pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.1))
        drv = pkg.md_driver(U, wilson(pkg, U), steps=1, trajectory_length=0.1, smearing=net, precision="mixed")
        filler = None
        before = free_bytes(torch)
        if idle_copy:
            pkg.calculate_Plaquette(U)
            filler = torch.empty(free_bytes(torch) - taken + COPY // 2, dtype=torch.uint8, device="cuda")
        try:
            r = pkg.md_trajectory_(U, P, drv)
        finally:
            del filler
            torch.cuda.empty_cache()
        return before - free_bytes(torch), (r.initial_hamiltonian, r.final_hamiltonian)

    taken, _ = trajectory(False)  # loads every kernel too
    taken, want = trajectory(False)
    assert taken > COPY
    assert trajectory(True)[1] == want


def launches(pkg):
    import ctypes
    from gaugefields_gb300 import _lib
    n = ctypes.c_longlong()
    _lib.check(_lib.load().gf_launch_count(ctypes.byref(n)))
    return n.value


def test_a_captured_force_touches_its_own_fields_only(pkg):
    """A graph may be replayed on any stream beside the context's other calls,
    so captured calls that need no state of the context use none: one launch
    each, no conversion of the links into the context's copy before it. They
    give the same to 1e-13."""
    torch = pytest.importorskip("torch")
    U = pkg.gauge_configuration((16, 16, 16, 16), start="hot", seed=5)
    plain, loops = wilson(pkg, U), wilson(pkg, U)
    pkg.push_(loops, -0.1, "rectangular")
    F = [pkg.gauge_momenta(U) for _ in range(3)]
    pkg.clear_U_(F[2])

    def calls():
        pkg.md_force_(F[0], plain, U)
        pkg.md_force_(F[1], loops, U)
        pkg.add_force_(F[2], U)

    def forces():
        return [f.to_host() for f in F]

    calls()
    want = forces()
    for f in F:
        pkg.gaussian_momenta_(f, seed=1)
    pkg.clear_U_(F[2])
    stream = torch.cuda.Stream()
    U.ctx.set_stream(stream.cuda_stream)
    U.ctx.torch_stream = stream
    graph = torch.cuda.CUDAGraph()
    before = launches(pkg)
    with torch.cuda.graph(graph, stream=stream):
        calls()
    assert launches(pkg) - before == 3
    graph.replay()
    torch.cuda.synchronize()
    for got, ref in zip(forces(), want):
        assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max()


def test_threads_of_one_context_wait_for_one_another(pkg):
    """Forces, plaquettes and smeared links of two configurations from two
    threads that share a context: bitwise those of one thread."""
    import threading
    L = (8, 8, 8, 16)
    U = pkg.gauge_configuration(L, start="hot", seed=5)
    V = U.similar().from_host(pkg.gauge_configuration(L, start="hot", seed=6).to_host())
    action, smearing = wilson(pkg, U), pkg.stout_smearing(U)
    F = {id(W): pkg.gauge_momenta(U) for W in (U, V)}

    def results(W):
        plaq = pkg.calculate_Plaquette(W)
        pkg.md_force_(F[id(W)], action, W)
        return plaq, F[id(W)].to_host(), pkg.smear(W, smearing).to_host()

    want = {id(W): results(W) for W in (U, V)}
    wrong, errors = [], []

    def work(W):
        try:
            for _ in range(200):
                got = results(W)
                wrong.extend(1 for a, b in zip(got, want[id(W)]) if not np.array_equal(a, b))
        except Exception as e:  # reported below: a thread's own would be lost
            errors.append(e)

    threads = [threading.Thread(target=work, args=(W,)) for W in (U, V)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and not wrong


def test_kept_memory_is_given_back(pkg):
    """What a context keeps between calls only to save allocations goes back on
    request, and to an allocation of another context that would fail."""
    torch = pytest.importorskip("torch")
    A = pkg.gauge_configuration(L24, start="hot", seed=11)
    B = pkg.gauge_configuration(L24, start="cold")
    A.ctx.trim()
    idle = free_bytes(torch)
    plaq = pkg.calculate_Plaquette(A)
    top = pkg.smear(A, pkg.stout_smearing(A))
    del top
    assert free_bytes(torch) < idle - COPY  # the copy, and buffers of the stack
    A.ctx.trim()
    assert free_bytes(torch) == idle
    pkg.calculate_Plaquette(A)
    size = 4 * 24 ** 4 * 144
    filler = torch.empty(free_bytes(torch) - size // 2, dtype=torch.uint8, device="cuda")
    try:
        B2 = B.similar()
        assert pkg.calculate_Plaquette(A) == pytest.approx(plaq, rel=1e-13)
        del B2
    finally:
        del filler
        torch.cuda.empty_cache()
    assert pkg.calculate_Plaquette(A) == plaq


def test_a_context_without_memory_for_its_copy(pkg):
    """A new context on a device that is nearly full does without the copy that
    small lattices get at once."""
    torch = pytest.importorskip("torch")
    L = (14, 14, 14, 14)
    want = pkg.calculate_Plaquette(pkg.gauge_configuration(L, start="cold"))
    torch.empty(1, device="cuda")
    filler, keep = [], 12 << 20  # the copy takes 22.8 MB
    while free_bytes(torch) > keep + (2 << 20):
        n = (free_bytes(torch) - keep) >> 21 << 21
        try:
            filler.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            break
    try:
        assert free_bytes(torch) < 20 << 20
        U = pkg.api._Context(L)
    finally:
        del filler
        torch.cuda.empty_cache()
    V = pkg.Gaugefields4D(U)
    pkg._lib.call("gf_cold_start", U.h, V.field.h)
    assert pkg.calculate_Plaquette(V) == want


def test_plain_and_double_float_drivers_share_their_stack(pkg):
    """The two forms' stacks are the same on lattices of this size: a driver of the
    second form takes no memory that the first has not."""
    torch = pytest.importorskip("torch")
    U = pkg.gauge_configuration(L24, start="hot", seed=11)
    net = pkg.CovNeuralnet(U)
    pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.1))
    P, free, energy = pkg.gaussian_momenta(U, seed=3), [], []
    for precision in ("fp64", "dfloat"):
        drv = pkg.md_driver(U, wilson(pkg, U), steps=1, smearing=net, precision=precision)
        energy.append(pkg.md_hamiltonian(U, P, drv))
        pkg.update_momenta_(P, U, 0.0, drv)
        free.append(free_bytes(torch))
    assert free[0] == free[1] and energy[0] == energy[1]


@pytest.mark.parametrize("blocks", [1.015, 1.5])
def test_mixed_energy_in_one_scratch_block(pkg, blocks):
    """The mixed form's smeared energy needs one scratch block of a link field for a
    level of smearing; the fixed-point sums take a second, larger one if there is
    memory, and the fp64 sums do without: the same to 1e-13."""
    torch = pytest.importorskip("torch")
    L = (32, 32, 32, 32)
    link64 = 4 * 32 ** 4 * 144  # 2.8% of it are 17 MB, above the 4 MB that allocations are rounded by

    def energy(fill):
        U = pkg.gauge_configuration(L, start="hot", seed=11)
        P = pkg.gaussian_momenta(U, seed=3)
        net = pkg.CovNeuralnet(U)
        pkg.push_(net, pkg.STOUT_Layer("plaquette", 0.1))
        action = wilson(pkg, U)
        pkg.push_(action, -0.1, "rectangular")
        drv = pkg.md_driver(U, action, steps=1, smearing=net, precision="mixed")
        filler = None
        if fill:
            filler = torch.empty(free_bytes(torch) - int(blocks * link64), dtype=torch.uint8, device="cuda")
        try:
            return pkg.md_hamiltonian(U, P, drv)
        finally:
            del filler
            torch.cuda.empty_cache()

    want = energy(False)
    assert energy(True) == pytest.approx(want, rel=1e-13)
