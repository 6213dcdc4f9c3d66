"""Performance cases: what programs built on this package spend their time on.

Each case is one pass through the public entry points on device-resident
fields: a measurement, a force, a link update, a gradient-flow stretch, a
stout smearing with its adjoint, or a whole molecular-dynamics call, in the
precision forms that md_driver and gradient_flow offer. Lattices are the ones
the tests, the benchmark and its scale mode use (8^4 to 48^4) and ragged ones
whose volume is no multiple of a thread block.

Fields are compared in the device layout of gf_field_device_ptr: even/odd
sites, links [4][9][V] complex128 and momenta [4][8][V] float64.
"""
import importlib.util
import math
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package, imported from its directory (its name is no identifier)."""
    name = "gaugefields_gb300"
    if name not in sys.modules:
        folder = os.path.join(ROOT, "gaugefields.jl_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
MAX_EXACT_SMEARED_LINKS = 3_000_000  # links x levels whose autograd reference runs in a few seconds
MAX_EXACT_LINKS = 12_000_000         # links x force evaluations of the reference without smearing


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(op, lattice, precision="fp64", levels=0, steps=0, name=None):
    nx, ny, nz, nt = lattice
    c = {"op": op, "nx": nx, "ny": ny, "nz": nz, "nt": nt, "precision": precision, "levels": levels, "steps": steps}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small lattice's plaquette: the call's latency, as in a thermalisation log
        _case("plaquette", (8, 8, 8, 8), name="plaquette_8"),
        # the same measurement on a production-size lattice
        _case("plaquette", (32, 32, 32, 64), name="plaquette_32x64"),
        # the Wilson force of the plain form (md_force!), the kernel of quenched HMC
        _case("wilson_force", (24, 24, 24, 24), name="wilson_force_24"),
        # scale setting: the RK3 Wilson flow in the reference's arithmetic
        _case("flow", (32, 32, 32, 32), steps=2, name="flow_32"),
        # the flow's double-float form on a lattice whose extents are no powers of two
        _case("flow", (22, 14, 18, 30), "dfloat", steps=5, name="flow_dfloat_ragged"),
        # differentiating through two smearing levels: forward with history, then back_prop
        _case("smear_grad", (16, 16, 16, 16), levels=2, name="smear_grad_16"),
        # one momentum update of the benchmark's stout HMC, its default form
        _case("stout_force", (32, 32, 32, 32), "dfloat", levels=2, name="stout_force_dfloat_32"),
        # the fp32-force form on a large lattice with three levels, as in the scale mode
        _case("stout_force", (48, 48, 48, 48), "mixed", levels=3, name="stout_force_mixed_48"),
        # an improved (plaquette + rectangle) action's momentum update, ragged lattice
        _case("rect_force", (10, 14, 18, 26), name="rect_force_ragged"),
        # the link update of the mixed and double-float forms at the precision study's size
        _case("link_update", (48, 48, 48, 48), "dfloat", name="link_update_dfloat_48"),
        # a whole plain-form Wilson trajectory of a small lattice
        _case("trajectory", (8, 8, 8, 8), steps=20, name="trajectory_8"),
        # a whole stout HMC update: momentum refresh, trajectory, accept or reject
        _case("hmc", (16, 16, 16, 16), "dfloat", levels=2, steps=10, name="hmc_stout_dfloat_16"),
    ]


# op: (precisions, levels, steps, smallest and largest volume). The largest
# volumes keep every drawn pass below the cost of the listed ones.
RANGES = {
    "plaquette": (("fp64",), (0,), (0,), 4 ** 4, 40 ** 4),
    "wilson_force": (("fp64",), (0,), (0,), 4 ** 4, 36 ** 4),
    "flow": (("fp64", "dfloat"), (0,), (1, 2, 3), 6 ** 4, 28 ** 4),
    "smear_grad": (("fp64",), (1, 2, 3), (0,), 4 ** 4, 24 ** 4),
    "stout_force": (("fp64", "mixed", "dfloat"), (1, 2, 3), (0,), 4 ** 4, 28 ** 4),
    "rect_force": (("fp64", "dfloat"), (0,), (0,), 6 ** 4, 24 ** 4),
    "link_update": (("fp64", "dfloat"), (0,), (0,), 4 ** 4, 40 ** 4),
    "trajectory": (("fp64", "dfloat"), (0, 1, 2), (2, 4, 8), 4 ** 4, 14 ** 4),
    "hmc": (("fp64", "dfloat"), (0, 1, 2), (2, 4, 8), 4 ** 4, 16 ** 4),
}


def draw(rng):
    op = rng.choice(sorted(RANGES))
    precisions, levels, steps, low, high = RANGES[op]
    volume = math.exp(rng.uniform(math.log(low), math.log(high)))
    # four even extents around volume^(1/4), the last one taking up what remains
    side = volume ** 0.25
    ext = [max(2, 2 * round(side * math.exp(rng.uniform(-0.35, 0.35)) / 2)) for _ in range(3)]
    last = max(2, 2 * int(volume / (ext[0] * ext[1] * ext[2]) / 2))
    lattice = ext + [last]
    while math.prod(lattice) > high:
        lattice[lattice.index(max(lattice))] -= 2
    return _case(op, lattice, rng.choice(precisions), rng.choice(levels), rng.choice(steps))


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
BETA, RHO, C_PLAQ, C_RECT = 6.0, 0.1, 3.648, -0.331 * 0.5  # Wilson; stout; Iwasaki-like loop coefficients
TAU = 0.5
ORDER = 3.1  # weight of the identity in a link: plaquettes of about 0.58, as at beta = 6


def _lattice(case):
    return [case["nx"], case["ny"], case["nz"], case["nt"]]


def _volume(case):
    return math.prod(_lattice(case))


def _dag(a):
    return a.mH


def _mm(a, b):
    """Product of arrays of 3x3 matrices, entry by entry."""
    out = a[..., :, 0:1] * b[..., 0:1, :]
    out = out + a[..., :, 1:2] * b[..., 1:2, :]
    return out + a[..., :, 2:3] * b[..., 2:3, :]


def _su3(gen, shape, weight):
    """SU(3) matrices: Gram-Schmidt of weight * 1 + complex Gaussian, phase divided out (Haar for weight 0)."""
    z = torch.randn(*shape, 3, 3, 2, dtype=torch.float64, device=DEVICE, generator=gen) * math.sqrt(0.5)
    m = torch.view_as_complex(z)
    m = m + weight * torch.eye(3, dtype=m.dtype, device=m.device)
    r1 = m[..., 0, :]
    r1 = r1 / r1.abs().square().sum(-1, keepdim=True).sqrt()
    r2 = m[..., 1, :]
    r2 = r2 - (r1.conj() * r2).sum(-1, keepdim=True) * r1
    r2 = r2 / r2.abs().square().sum(-1, keepdim=True).sqrt()
    r3 = torch.linalg.cross(r1, r2).conj()
    return torch.stack([r1, r2, r3], dim=-2)


def _shift(a, mu, d):
    """a(x + d e_mu) of an array over [NT, NZ, NY, NX, ...]."""
    return torch.roll(a, -d, 3 - mu)


def _links(case, seed):
    """Links like a thermalised configuration's: locally ordered, in a random gauge. [4, NT, NZ, NY, NX, 3, 3]."""
    gen = torch.Generator(device=DEVICE).manual_seed(7919 * seed + 1)
    shape = _lattice(case)[::-1]
    g = _su3(gen, shape, 0.0)
    out = torch.empty(4, *shape, 3, 3, dtype=torch.complex128, device=DEVICE)
    for mu in range(4):
        out[mu] = _mm(_mm(g, _su3(gen, shape, ORDER)), _dag(_shift(g, mu, 1)))
    return out


def _momenta(case, seed):
    """Unit Gaussian su(3) coefficients, [4, 8, NT, NZ, NY, NX]."""
    gen = torch.Generator(device=DEVICE).manual_seed(7919 * seed + 2)
    return torch.randn(4, 8, *_lattice(case)[::-1], dtype=torch.float64, device=DEVICE, generator=gen)


def _derivative(case, seed):
    """A general dS/dUbar: complex Gaussian matrices, [4, NT, NZ, NY, NX, 3, 3]."""
    gen = torch.Generator(device=DEVICE).manual_seed(7919 * seed + 3)
    z = torch.randn(4, *_lattice(case)[::-1], 3, 3, 2, dtype=torch.float64, device=DEVICE, generator=gen)
    return torch.view_as_complex(z)


# ---------------------------------------------------------------------------
# the device layout
# ---------------------------------------------------------------------------
def _device_sites(case):
    """Lexicographic index of each even/odd-ordered site."""
    nx, ny, nz, nt = _lattice(case)
    lex = torch.arange(nx * ny * nz * nt, device=DEVICE)
    parity = (lex % nx + lex // nx % ny + lex // (nx * ny) % nz + lex // (nx * ny * nz)) % 2
    return torch.cat([lex[parity == 0], lex[parity == 1]])


def _to_device_links(case, u):
    """[4, NT, NZ, NY, NX, 3, 3] -> [4, 9, V]."""
    return u.reshape(4, -1, 9).index_select(1, _device_sites(case)).transpose(1, 2)


def _to_device_momenta(case, p):
    return p.reshape(4, 8, -1).index_select(2, _device_sites(case))


class _DeviceArray:
    """A field's device buffer for torch, through the address that the library gives out."""

    def __init__(self, field, components, typestr):
        self.field = field
        self.__cuda_array_interface__ = {"shape": (4, components, field.ctx.V), "typestr": typestr,
                                         "data": (field.device_ptr(), False), "version": 3, "strides": None}


def _links_of(u):
    return torch.as_tensor(_DeviceArray(u.field, 9, "<c16"), device=DEVICE)


def _momenta_of(p):
    return torch.as_tensor(_DeviceArray(p.field, 8, "<f8"), device=DEVICE)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    gf = _package()
    op, s = case["op"], {"op": case["op"], "gf": gf}
    u = s["U"] = gf.gauge_configuration(_lattice(case), start="cold")
    u.ctx.sync()
    s["links"] = _links_of(u)
    s["links"].copy_(_to_device_links(case, _links(case, seed)))
    net = None
    if case["levels"]:
        net = s["net"] = gf.CovNeuralnet(u)
        for _ in range(case["levels"]):
            gf.push_(net, gf.STOUT_Layer("plaquette", RHO))
    if op in ("wilson_force", "rect_force", "stout_force", "link_update", "trajectory", "hmc"):
        p = s["P"] = gf.gauge_momenta(u)
        u.ctx.sync()
        s["momenta"] = _momenta_of(p)
        s["momenta"].copy_(_to_device_momenta(case, _momenta(case, seed)))
        action = s["action"] = gf.GaugeAction(u)
        if op == "rect_force":
            gf.push_(action, C_PLAQ, "plaquette")
            gf.push_(action, C_RECT, "rectangular")
        else:
            gf.push_(action, BETA / 2, "plaquette")
        s["driver"] = gf.md_driver(u, action, steps=max(1, case["steps"]), trajectory_length=TAU, smearing=net,
                                   precision=case["precision"])
    if op == "flow":
        s["flow"] = gf.gradient_flow(u, steps=case["steps"], step_size=0.01, precision=case["precision"])
    if op == "smear_grad":
        d = s["D"] = gf.Gaugefields4D(u.ctx, gf._lib.GF_MAT64)
        _links_of(d).copy_(_to_device_links(case, _derivative(case, seed)))
    if op == "hmc":
        s["seed"], s["sweep"] = seed, 0
    if torch.cuda.is_available():
        torch.cuda.synchronize()
    return s


STEP = 0.05  # momentum and link step size of the single updates


def run(s):
    gf, op, u = s["gf"], s["op"], s["U"]
    if op == "plaquette":
        return gf.measure_plaquette(u)
    if op == "wilson_force":
        gf.md_force_(s["P"], s["action"], u)
        return s["momenta"]
    if op in ("rect_force", "stout_force"):
        gf.update_momenta_(s["P"], u, STEP, s["driver"])
        return s["momenta"]
    if op == "link_update":
        gf.update_gaugefields_(u, s["P"], STEP, s["driver"])
        return s["links"]
    if op == "flow":
        gf.flow_(u, s["flow"])
        return s["links"]
    if op == "smear_grad":
        smeared, history, _ = gf.calc_smearedU(u, s["net"])
        grad = gf.back_prop(s["D"], s["net"], history, u)
        return {"smeared": _links_of(smeared), "gradient": _links_of(grad)}
    if op == "trajectory":
        r = gf.md_trajectory_(u, s["P"], s["driver"])
    else:
        s["sweep"] += 1
        r = gf.hmc_update_(u, s["P"], s["driver"], seed=s["seed"], sweep=s["sweep"], unif=0.5)
    return {"links": s["links"], "momenta": s["momenta"], "initial": r.initial_hamiltonian,
            "final": r.final_hamiltonian}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: every input read once, every output written once (links 144 B,
    momenta 64 B per link, fp64 in memory in every form). Flops per link: a
    complex 3x3 product is 198, an accumulated one 216."""
    n = 4 * _volume(case)
    mul, mac = 198, 216
    staples = 6 * (mul + mac)
    force = staples + mul
    update = 2 * mul + 400                      # exp(i eps P) and its product with the link
    forward = staples + 2 * mul + 600           # staples, U S, exponential and its product
    adjoint = 8 * mul + 900 + 3 * (4 * mul + 6 * mac)  # local part, then the factored pull-back
    rect = 3 * (18 * mul + 6 * mac)
    op, levels, steps = case["op"], case["levels"], case["steps"]
    kick = force + levels * (forward + adjoint)
    plaquette = 6 * (2 * mul + 36) / 4
    if op == "plaquette":
        b, f = 144, plaquette
    elif op == "wilson_force":
        b, f = 144 + 64, force
    elif op == "rect_force":
        b, f = 144 + 128, force + rect
    elif op == "stout_force":
        b, f = 144 + 128, kick
    elif op == "link_update":
        b, f = 64 + 288, update
    elif op == "flow":
        b, f = 288, 3 * steps * (force + update)
    elif op == "smear_grad":
        b, f = 144 * 4, levels * (forward + adjoint)
    else:
        b, f = 288 + 128, steps * (kick + update) + update + 2 * (plaquette + levels * forward)
    return {"bytes": b * n, "flops": f * n}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------
def _up_down(u, mu, nu):
    """The two staples of U_mu in the mu-nu plane, as the rest of each plaquette after U_mu(x)."""
    a = _mm(_mm(_shift(u[nu], mu, 1), _dag(_shift(u[mu], nu, 1))), _dag(u[nu]))
    w = _mm(_mm(_dag(_shift(u[nu], mu, 1)), _dag(u[mu])), u[nu])
    return a + _shift(w, nu, -1)


def _staples(u, mu):
    return sum(_up_down(u, mu, nu) for nu in range(4) if nu != mu)


def _rectangle_staples(u, mu):
    """The eighteen rectangle staples of U_mu(x), in the same sense."""
    total = 0
    for nu in range(4):
        if nu == mu:
            continue
        n1, m1 = _shift(u[nu], mu, 1), _shift(u[mu], mu, 1)
        two_n = _mm(u[nu], _shift(u[nu], nu, 1))
        # 1x2, above and below
        total = total + _mm(_mm(_shift(two_n, mu, 1), _dag(_shift(u[mu], nu, 2))), _dag(two_n))
        w = _mm(_mm(_dag(_shift(two_n, mu, 1)), _dag(u[mu])), two_n)
        total = total + _shift(w, nu, -2)
        # 2x1 with U_mu(x) first
        two_m = _mm(u[mu], m1)
        n2 = _shift(u[nu], mu, 2)
        total = total + _mm(_mm(_mm(m1, n2), _dag(_shift(two_m, nu, 1))), _dag(u[nu]))
        w = _mm(_mm(_dag(n2), _dag(two_m)), u[nu])
        total = total + _mm(m1, _shift(w, nu, -1))
        # 2x1 with U_mu(x) second: the staple of U_mu(x + mu), one site back
        w = _mm(_mm(n1, _dag(_shift(u[mu], nu, 1))), _mm(_dag(_shift(_shift(u[mu], nu, 1), mu, -1)),
                                                         _dag(_shift(u[nu], mu, -1))))
        total = total + _mm(w, _shift(u[mu], mu, -1))
        low = _shift(_mm(_mm(_dag(n1), _dag(u[mu])), _mm(_dag(_shift(u[mu], mu, -1)), _shift(u[nu], mu, -1))), nu, -1)
        total = total + _mm(low, _shift(u[mu], mu, -1))
    return total


def _traceless_antihermitian(m):
    a = (m - _dag(m)) / 2
    trace = a.diagonal(dim1=-2, dim2=-1).sum(-1)
    return a - trace[..., None, None] / 3 * torch.eye(3, dtype=m.dtype, device=m.device)


def _coefficients(m):
    """su(3) coefficients c_a of TA(m) = i sum_a c_a lambda_a / 2, stacked first."""
    x12, x13, x23 = (m[..., i, j] - m[..., j, i].conj() for i, j in ((0, 1), (0, 2), (1, 2)))
    d1, d2, d3 = (m[..., i, i].imag for i in range(3))
    return torch.stack([x12.imag, x12.real, d1 - d2, x13.imag, x13.real, x23.imag, x23.real,
                        (d1 + d2 - 2 * d3) / math.sqrt(3.0)])


def _algebra(p):
    """i sum_a p_a lambda_a / 2 of coefficients [8, ...]."""
    r = 1 / math.sqrt(3.0)
    rows = [[torch.complex(p[2] + r * p[7], 0 * p[0]), torch.complex(p[0], -p[1]), torch.complex(p[3], -p[4])],
            [torch.complex(p[0], p[1]), torch.complex(r * p[7] - p[2], 0 * p[0]), torch.complex(p[5], -p[6])],
            [torch.complex(p[3], p[4]), torch.complex(p[5], p[6]), torch.complex(-2 * r * p[7], 0 * p[0])]]
    return 0.5j * torch.stack([torch.stack(row, dim=-1) for row in rows], dim=-2)


def _exp(q):
    """Matrix exponential: Horner form of the power series, 22 terms of q / 4, squared twice."""
    eye = torch.eye(3, dtype=q.dtype, device=q.device).expand_as(q)
    q, e = q / 4, eye
    for n in range(22, 0, -1):
        e = eye + _mm(q, e) / n
    return _mm(*(2 * [_mm(e, e)]))


def _smear(u):
    out = []
    for mu in range(4):
        q = -RHO * _traceless_antihermitian(_mm(u[mu], _staples(u, mu)))
        out.append(_mm(_exp(q), u[mu]))
    return torch.stack(out)


def _plaquette_sum(u):
    total = 0.0
    for mu in range(4):
        for nu in range(mu + 1, 4):
            a = _mm(u[mu], _shift(u[nu], mu, 1))
            b = _mm(u[nu], _shift(u[mu], nu, 1))
            total = total + (a * b.conj()).real.sum()
    return total


def _pull_back(u, levels, d_top):
    """dS/dU (dS = 2 Re tr(dU dS/dU)) of the thin links from a given one of the smeared links, by autograd;
    d_top None: that of BETA times the plaquette sum. Returns the smeared links too."""
    thin = u.clone().requires_grad_(True)
    top = thin
    for _ in range(levels):
        top = _smear(top)
    if d_top is None:
        d_top = torch.stack([BETA / 2 * _staples(top.detach(), mu) for mu in range(4)])
    value = 2 * (top * d_top.mT).real.sum()
    (g,) = torch.autograd.grad(value, thin)
    return _dag(g) / 2, top.detach()


def _force(case, u):
    """F_mu = -(1/3) TA(U dS/dU) in su(3) coefficients, [4, 8, ...]."""
    if case["levels"]:
        d, _ = _pull_back(u, case["levels"], None)
    elif case["op"] == "rect_force":
        d = [C_PLAQ * _staples(u, mu) + C_RECT * _rectangle_staples(u, mu) for mu in range(4)]
    else:
        d = [BETA / 2 * _staples(u, mu) for mu in range(4)]
    return torch.stack([_coefficients(_mm(u[mu], d[mu])) for mu in range(4)]) / -3


def _unitarise(u):
    r1, r2 = u[..., 0, :], u[..., 1, :]
    r2 = r2 - (r1.conj() * r2).sum(-1, keepdim=True) / r1.abs().square().sum(-1, keepdim=True) * r1
    r1 = r1 / r1.abs().square().sum(-1, keepdim=True).sqrt()
    r2 = r2 / r2.abs().square().sum(-1, keepdim=True).sqrt()
    return torch.stack([r1, r2, torch.linalg.cross(r1, r2).conj()], dim=-2)


def _update_links(u, p, step, unitarise=True):
    for mu in range(4):
        w = _mm(_exp(step * _algebra(p[mu])), u[mu])
        u[mu] = _unitarise(w) if unitarise else w
    return u


def _hamiltonian(case, u, p):
    top = u
    for _ in range(case["levels"]):
        top = _smear(top)
    return float(-BETA / 3 * _plaquette_sum(top) + 0.5 * p.square().sum())


def exact(case, seed):
    op, links = case["op"], 4 * _volume(case)
    if op == "hmc":
        return None  # the momenta are the library's own draws
    evaluations = max(1, case["steps"]) * (3 if op == "flow" else 1)
    if case["levels"]:
        if links * case["levels"] > MAX_EXACT_SMEARED_LINKS or links * evaluations > MAX_EXACT_SMEARED_LINKS:
            return None  # the autograd graph of the smearing would take too long
    elif links * evaluations > MAX_EXACT_LINKS * 4:
        return None
    u = _links(case, seed)
    if op == "plaquette":
        return float(_plaquette_sum(u)) / (18 * _volume(case))
    if op == "wilson_force":
        return _to_device_momenta(case, _force(case, u))
    if op in ("rect_force", "stout_force"):
        return _to_device_momenta(case, _momenta(case, seed) + STEP * _force(case, u))
    if op == "link_update":
        return _to_device_links(case, _update_links(u, _momenta(case, seed), STEP))
    if op == "smear_grad":
        d, top = _pull_back(u, case["levels"], _derivative(case, seed))
        return {"smeared": _to_device_links(case, top), "gradient": _to_device_links(case, d)}
    if op == "flow":
        eps = 0.01
        for _ in range(case["steps"]):
            g = 0
            for keep, weight, scale in ((0.0, 17 / 36, -9 / 17), (1.0, -8 / 9, 1.0), (-1.0, -3 / 4, 1.0)):
                f = torch.stack([_coefficients(_mm(u[mu], _staples(u, mu))) for mu in range(4)])
                g = keep * g + weight * eps * f
                u = _update_links(u, g, scale, unitarise=False)
        return _to_device_links(case, u)
    p = _momenta(case, seed)
    first = _hamiltonian(case, u, p)
    eps = TAU / case["steps"]
    for n in range(case["steps"]):
        u = _update_links(u, p, eps / 2 if n == 0 else eps)
        p = p + eps * _force(case, u)
    u = _update_links(u, p, eps / 2)
    return {"links": _to_device_links(case, u), "momenta": _to_device_momenta(case, p), "initial": first,
            "final": _hamiltonian(case, u, p)}
