"""GPU parity of the fixed-point kernels (gf_fixed.cu) at the sizes and on the
links where they can go wrong: fewer links than a block, a last block and a
last tile that are nearly empty, links whose exponents differ (not unitary,
over many orders of magnitude), and a NaN.

Tolerances: 1e-13 of the largest entry, two orders above fp64 rounding of the
sums involved (the oracle's own).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2, 2), (2, 4, 2, 6), (6, 2, 10, 2), (4, 6, 10, 14), (34, 2, 2, 6)]
TOL = 1e-13


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
