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
