"""The framework's performance cases: the work that its users have it do.

A case names a path through the public entry points and its sizes:

* ``coulomb``: ``B200DensityFittedCoulombExchange.coulomb(D)``, once per SCF iteration;
* ``exchange``: ``exchange(D)`` in FP64, what an SCF driver that holds only densities calls;
* ``factored``: ``exchange_factored(C)`` from the occupied orbitals, in FP64 or split BF16,
  what ``hafnium_b200.scf`` calls;
* ``setup``: a new geometry, ``DeviceHamiltonian.build`` and the first J and K on it;
* ``gradient``: ``hafnium_b200.gradient.gradient_from_state`` on a closed-shell state;
* ``batch``: ``hafnium_b200.batch.solve_batch`` on clusters of several sizes, to convergence.

Molecules are seeded water clusters, the auxiliary basis is def2-universal-jkfit.
Densities and orbitals are those of the core Hamiltonian, the start of an SCF without a
guess. ``host`` cases pass and return NumPy arrays, as the reference's driver does.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from hafnium_b200 import _lib
from hafnium_b200.basis import ShellTable
from hafnium_b200.batch import solve_batch
from hafnium_b200.gradient import gradient_from_state
from hafnium_b200.molecule import water_cluster
from hafnium_b200.scf import DeviceHamiltonian

AUXILIARY = "def2-universal-jkfit"
FP64 = torch.float64


def _case(path, waters, *, basis="cc-pvdz", host=False, precision="fp64", signed=False, clusters=1, largest=0, name=None):
    case = {"path": path, "waters": waters, "basis": basis, "host": host, "precision": precision, "signed": signed,
            "clusters": clusters, "largest": largest}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one water: every iteration of a small molecule's SCF, where latency counts
        _case("coulomb", 1, name="coulomb_1"),
        # an ordinary cluster whose 288 orbitals fill neither 64-wide nor 128-wide tiles
        _case("coulomb", 12, name="coulomb_12"),
        # the size of the split-precision workload (768 orbitals, an 8.9 GB fitted tensor)
        _case("coulomb", 32, name="coulomb_32"),
        # the exchange of a small molecule's SCF from its density alone
        _case("exchange", 2, name="exchange_2"),
        # the unchanged reference driver on an ordinary cluster: NumPy density in, NumPy K out
        _case("exchange", 12, host=True, name="exchange_12_host"),
        # the plain FP64 path and the anchor builds of the mixed schedule
        _case("factored", 32, name="factored_32"),
        # early iterations of the mixed schedule: a ragged size and the large one
        _case("factored", 14, precision="bf16", name="factored_bf16_14"),
        _case("factored", 32, precision="bf16", name="factored_bf16_32"),
        # a geometry scan: integrals, fit, first J and K at a new geometry
        _case("setup", 2, name="setup_2"),
        _case("setup", 16, name="setup_16"),
        # one step of a geometry optimisation or of molecular dynamics
        _case("gradient", 8, name="gradient_8"),
        # screening and training data: many small clusters converged together
        _case("batch", 2, clusters=12, largest=4, name="batch_12"),
    ]


def draw(rng):
    """Another case of the listed ranges: sizes log-uniform, every shipped orbital basis,
    host and device arrays, unsigned and signed factors."""
    path = rng.choice(["coulomb", "exchange", "factored", "factored", "setup", "gradient", "batch"])
    top = {"coulomb": 32, "exchange": 28, "factored": 32, "setup": 16, "gradient": 10, "batch": 3}[path]
    low = {"batch": 2}.get(path, 1)
    waters = min(top, max(low, int(math.exp(rng.uniform(math.log(low), math.log(top + 0.99))))))
    basis = rng.choice(["cc-pvdz", "cc-pvdz", "def2-svp", "sto-3g"])
    host = path in ("coulomb", "exchange", "factored") and rng.random() < 0.35
    precision = "bf16" if path == "factored" and rng.random() < 0.5 else "fp64"
    signed = path == "factored" and rng.random() < 0.25
    if path == "batch":
        return _case(path, waters, basis=basis, clusters=rng.randint(3, 10), largest=waters + rng.randint(0, 1))
    return _case(path, waters, basis=basis, host=host, precision=precision, signed=signed)


def _core_orbitals(ham):
    """Occupied orbitals of the core Hamiltonian, [n_ao, n_occ]."""
    w, v = torch.linalg.eigh(ham.s)
    x = v / torch.sqrt(w)[None, :]
    _, c = torch.linalg.eigh(x.T @ ham.h @ x)
    return (x @ c[:, : int(ham.n_alpha)]).contiguous()


def prepare(case, seed):
    if case["path"] == "batch":
        sizes = [case["waters"] + i % (case["largest"] - case["waters"] + 1) for i in range(case["clusters"])]
        return {"case": case, "molecules": [water_cluster(w, seed + 7919 * i) for i, w in enumerate(sizes)]}
    molecule = water_cluster(case["waters"], seed)
    ham = DeviceHamiltonian.build(molecule, case["basis"], AUXILIARY)
    occupied = _core_orbitals(ham)
    state = {"case": case, "molecule": molecule, "two_body": ham.two_body, "occupied": occupied,
             "density": (occupied @ occupied.T).contiguous(), "weights": None}
    if case["path"] == "coulomb":
        state["density"] = 2.0 * state["density"]
    elif case["path"] == "setup":
        del state["two_body"]  # the new geometry has its own
    elif case["path"] == "gradient":
        j, k = ham.two_body.coulomb(2.0 * state["density"]), ham.two_body.exchange(state["density"])
        state["fock"] = ham.h + j - k
    if case["signed"]:  # a difference density: its factor has columns of either sign
        gen = torch.Generator().manual_seed(seed)
        sign = torch.where(torch.rand(occupied.shape[1], generator=gen, dtype=FP64) < 0.5, -1.0, 1.0)
        state["weights"] = (sign * torch.rand(occupied.shape[1], generator=gen, dtype=FP64)).to(occupied.device)
    if case["host"]:
        for key in ("occupied", "density", "weights"):
            state[key] = None if state[key] is None else state[key].cpu().numpy()
    return state


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "coulomb":
        return state["two_body"].coulomb(state["density"])
    if path == "exchange":
        return state["two_body"].exchange(state["density"])
    if path == "factored":
        precision = _lib.PREC_BF16X3 if case["precision"] == "bf16" else _lib.PREC_FP64
        return state["two_body"].exchange_factored(state["occupied"], state["weights"], precision)
    if path == "setup":
        ham = DeviceHamiltonian.build(state["molecule"], case["basis"], AUXILIARY)
        return {"s": ham.s, "h": ham.h, "j": ham.two_body.coulomb(2.0 * state["density"]),
                "k": ham.two_body.exchange(state["density"])}
    if path == "gradient":
        g = gradient_from_state(state["two_body"], state["occupied"], state["fock"], state["molecule"])
        return [g.one_electron, g.overlap, g.coulomb, g.exchange, g.total]
    result = solve_batch(state["molecules"], case["basis"], AUXILIARY, keep_densities=True)
    return [result.energies, *result.densities]


@functools.lru_cache(maxsize=None)
def _sizes(waters, basis):
    """(n_ao, n_aux, n_occ) of a water cluster."""
    molecule = water_cluster(1, 0)
    n, naux = (ShellTable.build(b, molecule.symbols, molecule.positions).n_functions for b in (basis, AUXILIARY))
    return waters * n, waters * naux, 5 * waters


def work(case):
    """Each input once, each output once, B as packed upper triangles; K as the half-transform
    and one triangle of X X^T; a fit as the metric's factor, its inverse and their product with
    (P|uv). The integrals' own arithmetic depends on screening and is not counted."""
    n, naux, o = _sizes(case["waters"], case["basis"])
    tri = n * (n + 1) / 2
    packed = 8.0 * naux * tri
    fit = naux**2 * tri + naux**3 * (2.0 / 3.0)
    coulomb, exchange = 4.0 * naux * tri, 3.0 * naux * n * n * o
    path = case["path"]
    if path == "coulomb":
        return {"bytes": packed + 16.0 * n * n, "flops": coulomb}
    if path == "exchange":
        return {"bytes": packed + 16.0 * n * n, "flops": exchange}
    if path == "factored":
        return {"bytes": packed + 8.0 * n * (n + o), "flops": exchange}
    if path == "setup":
        return {"bytes": packed + 48.0 * n * n, "flops": fit + coulomb + exchange}
    if path == "gradient":
        # C^T B_Q C, its product with L^-1, Gamma Gamma^T, and the exchange weights C Gamma_P C^T
        flops = 2.0 * naux * n * o * (n + o) + 2.0 * naux**2 * o * o + 2.0 * naux * n * o * (o + n)
        return {"bytes": packed + 8.0 * n * (n + o), "flops": flops + naux**3 * (2.0 / 3.0)}
    total = {"bytes": 0.0, "flops": 0.0}
    for i in range(case["clusters"]):
        n, naux, o = _sizes(case["waters"] + i % (case["largest"] - case["waters"] + 1), case["basis"])
        tri = n * (n + 1) / 2
        # about twelve iterations, each a J, a K and the density of a Fock matrix
        total["bytes"] += 8.0 * (naux * tri + n * n)
        total["flops"] += naux**2 * tri + 12.0 * (4.0 * naux * tri + 3.0 * naux * n * n * o + 10.0 * n**3)
    return total


def tolerance(case):
    path = case["path"]
    if path == "factored" and case["precision"] == "bf16":
        # 16-bit significands and 32-bit sums: about 3e-5 from the 64-bit value
        return {"rel": 1e-4, "max": 4e-3}
    # the fit's error is the metric's condition (below 1e6) times rounding; an SCF stops at a
    # gradient of 1e-6, where its density is good to about 1e-8
    return {"setup": {"rel": 1e-10, "max": 1e-8}, "gradient": {"rel": 1e-8, "max": 1e-6},
            "batch": {"rel": 1e-7, "max": 1e-5}}.get(path, {"rel": 2e-13, "max": 1e-11})


# ------------------------------------------------------------------ 64-bit values


def exact(case, seed):
    """J and K in plain torch from the fitted tensor that the caller's handle holds (read out
    once); a setup's S, h, J and K from integrals in plain torch (up to three waters: the dense
    primitive tensors of larger clusters take too long). A gradient and a converged SCF have no
    plain form that ends in seconds."""
    path = case["path"]
    if path == "setup":
        return _exact_setup(case, seed) if case["waters"] <= 3 else None
    if path in ("gradient", "batch"):
        return None
    state = prepare(case, seed)
    two_body = state["two_body"]
    dev = torch.device("cuda", two_body.context.device)
    eye = torch.eye(two_body.n_ao, dtype=FP64, device=dev)
    b = two_body.orbital_tensor(eye, eye)
    if path == "coulomb":
        d = torch.as_tensor(state["density"], device=dev)
        out = torch.einsum("quv,q->uv", b, torch.einsum("quv,uv->q", b, d))
    elif path == "exchange":
        out = _plain_exchange(b, torch.as_tensor(state["density"], device=dev))
    else:
        c = torch.as_tensor(state["occupied"], device=dev)
        w = state["weights"]
        out = _plain_exchange(b, c @ c.T if w is None else (c * torch.as_tensor(w, device=dev)[None, :]) @ c.T)
    return out.cpu().numpy() if case["host"] else out


def _plain_exchange(b, d):
    out = torch.zeros_like(d)
    for q in range(0, b.shape[0], 128):
        part = b[q:q + 128]
        out += torch.einsum("quw,qwv->uv", part @ d, part)
    return out


def _boys(order, t):
    """F_0 .. F_order from the regularised incomplete gamma function and downward recursion."""
    a = torch.full_like(t, order + 0.5)
    safe = t.clamp(min=1e-6)
    top = 0.5 * math.gamma(order + 0.5) * torch.special.gammainc(a, safe) * safe ** -(order + 0.5)
    series = 1.0 / (2 * order + 1) - t / (2 * order + 3) + t * t / (2 * (2 * order + 5))
    f = [torch.where(t < 1e-6, series, top)]
    for m in range(order, 0, -1):
        f.append((2.0 * t * f[-1] + torch.exp(-t)) / (2 * m - 1))
    return f[::-1]


def _hermite_coulomb(order, alpha, r):
    """{(t, u, v): R_tuv} of the Hermite Coulomb recursion (Helgaker 9.9.18-20)."""
    f = _boys(order, alpha * (r * r).sum(-1))
    level = {}
    for n in range(order, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** n * f[n]}
        for s in range(1, order - n + 1):
            for t in range(s + 1):
                for u in range(s - t + 1):
                    key = [t, u, s - t - u]
                    axis = next(x for x in range(3) if key[x])
                    key[axis] -= 1
                    low = tuple(key)
                    value = r[..., axis] * level[low]
                    if key[axis]:
                        lower = list(low)
                        lower[axis] -= 1
                        value = value + key[axis] * level[tuple(lower)]
                    key[axis] += 1
                    new[tuple(key)] = value
        level = new
    return level


def _hermite_e(la, lb, p, pa, pb, e00):
    """e[i][j][t], one axis of the Hermite expansion of a pair (Helgaker 9.5.6-7)."""
    e = {(0, 0, 0): e00}

    def get(i, j, t):
        return e.get((i, j, t), 0.0) if 0 <= t <= i + j else 0.0

    for i in range(la + 1):
        for j in range(lb + 1):
            if i or j:
                a, b, x = (i - 1, j, pa) if i else (i, j - 1, pb)
                for t in range(i + j + 1):
                    e[i, j, t] = 0.5 / p * get(a, b, t - 1) + x * get(a, b, t) + (t + 1) * get(a, b, t + 1)
    return e


@functools.lru_cache(maxsize=None)
def _harmonics(l):
    """[(m row)][((i, j, k), coefficient)]: sphere-normalised real solid harmonics (Helgaker
    6.4.47), p ordered x, y, z."""
    rows = []
    for m in ([1, -1, 0] if l == 1 else range(-l, l + 1)):
        am, terms = abs(m), {}
        norm = math.sqrt(2.0 * math.factorial(l + am) * math.factorial(l - am) / (2.0 if m == 0 else 1.0))
        norm *= math.sqrt((2 * l + 1) / (4.0 * math.pi)) / (2.0**am * math.factorial(l))
        for t in range((l - am) // 2 + 1):
            for u in range(t + 1):
                for v2 in range(1 if m < 0 else 0, am + 1, 2):
                    c = (-1.0) ** (t + v2 // 2) * 0.25**t * math.comb(l, t) * math.comb(l - t, am + t)
                    key = (2 * t + am - 2 * u - v2, 2 * u + v2, l - 2 * t - am)
                    terms[key] = terms.get(key, 0.0) + norm * c * math.comb(t, u) * math.comb(am, v2)
        rows.append(tuple((k, c) for k, c in terms.items() if c))
    return tuple(rows)


def _primitives(table, dev):
    """Per l: exponents, centres and the contraction matrix [functions, primitive, m]."""
    offsets, fn = table.primitive_offsets, table.function_offsets()
    out, coef = {}, 0
    total = table.n_functions
    for s in range(table.n_shells):
        l, p0, p1, k = int(table.angular_momenta[s]), int(offsets[s]), int(offsets[s + 1]), int(table.n_contractions[s])
        rows = np.asarray(table.coefficients[coef:coef + k * (p1 - p0)]).reshape(k, p1 - p0)
        coef += k * (p1 - p0)
        group = out.setdefault(l, ([], [], []))
        for i in range(p1 - p0):
            group[0].append(float(table.exponents[p0 + i]))
            group[1].append(table.centers[s])
            matrix = np.zeros((total, 2 * l + 1))
            for c in range(k):
                for m in range(2 * l + 1):
                    matrix[int(fn[s]) + c * (2 * l + 1) + m, m] = rows[c, i]
            group[2].append(matrix)
    return {l: (torch.tensor(e, dtype=FP64, device=dev), torch.tensor(np.array(x), dtype=FP64, device=dev),
                torch.tensor(np.stack(c, axis=1), dtype=FP64, device=dev)) for l, (e, x, c) in out.items()}


def _pairs(la, lb, ga, gb, kinetic=0):
    """All primitive pairs of two groups: exponent p, centre, and the one-axis tables."""
    a, b = ga[0][:, None], gb[0][None, :]
    p = (a + b).reshape(-1)
    ra, rb = ga[1][:, None, :], gb[1][None, :, :]
    centre = (a[..., None] * ra + b[..., None] * rb).reshape(-1, 3) / p[:, None]
    full = (len(ga[0]), len(gb[0]), 3)
    ra, rb = ra.expand(full).reshape(-1, 3), rb.expand(full).reshape(-1, 3)
    mu = (a * b).reshape(-1) / p
    e = [_hermite_e(la, lb + kinetic, p, centre[:, x] - ra[:, x], centre[:, x] - rb[:, x],
                    torch.exp(-mu * (ra[:, x] - rb[:, x]) ** 2)) for x in range(3)]
    return p, centre, e, b.expand(full[:2]).reshape(-1)


def _spherical_hermite(la, lb, e):
    """{(t, u, v): [pair, m_a, m_b]}: a pair's Hermite coefficients of spherical functions."""
    out = {}
    like = e[0][0, 0, 0]
    for ma, row_a in enumerate(_harmonics(la)):
        for mb, row_b in enumerate(_harmonics(lb)):
            for (i, ca) in row_a:
                for (j, cb) in row_b:
                    for t in range(i[0] + j[0] + 1):
                        for u in range(i[1] + j[1] + 1):
                            for v in range(i[2] + j[2] + 1):
                                block = out.setdefault((t, u, v), like.new_zeros(len(like), 2 * la + 1, 2 * lb + 1))
                                block[:, ma, mb] += ca * cb * (e[0][i[0], j[0], t] * e[1][i[1], j[1], u] * e[2][i[2], j[2], v])
    return out


def _contract(values, ga, gb):
    """[pair, m_a, m_b, ...] of primitives -> [function, function, ...]."""
    values = values.reshape(len(ga[0]), len(gb[0]), *values.shape[1:])
    return torch.einsum("xam,abmn...,ybn->xy...", ga[2], values, gb[2])


def _one_electron(table, molecule, dev):
    groups = _primitives(table, dev)
    s = torch.zeros(table.n_functions, table.n_functions, dtype=FP64, device=dev)
    h = torch.zeros_like(s)
    for la, ga in groups.items():
        for lb, gb in groups.items():
            p, centre, e, b = _pairs(la, lb, ga, gb, kinetic=2)
            hermite = _spherical_hermite(la, lb, e)
            s += _contract((math.pi / p)[:, None, None] ** 1.5 * hermite[0, 0, 0], ga, gb)
            attraction = 0.0
            for z, r in zip(molecule.nuclear_charges, torch.tensor(molecule.positions, dtype=FP64, device=dev)):
                table_r = _hermite_coulomb(la + lb, p, centre - r)
                attraction = attraction - float(z) * sum(c * table_r[k][:, None, None] for k, c in hermite.items())
            kinetic = torch.zeros_like(attraction)
            for ma, row_a in enumerate(_harmonics(la)):
                for mb, row_b in enumerate(_harmonics(lb)):
                    for (i, ca) in row_a:
                        for (j, cb) in row_b:
                            plain = [e[x][i[x], j[x], 0] for x in range(3)]
                            for x in range(3):
                                second = 4.0 * b * b * e[x][i[x], j[x] + 2, 0] - 2.0 * b * (2 * j[x] + 1) * plain[x]
                                if j[x] > 1:
                                    second = second + j[x] * (j[x] - 1) * e[x][i[x], j[x] - 2, 0]
                                rest = plain[(x + 1) % 3] * plain[(x + 2) % 3]
                                kinetic[:, ma, mb] += -0.5 * ca * cb * second * rest * (math.pi / p) ** 1.5
            h += _contract(kinetic + (2.0 * math.pi / p)[:, None, None] * attraction, ga, gb)
    return s, h


def _coulomb_integrals(bra, ket, dev):
    """(ab|P) or, with an empty second bra, (Q|P): [function a, function b, function P]."""
    groups, others = _primitives(bra[0], dev), _primitives(bra[1], dev) if bra[1] is not None else None
    # the constant function one, as an s primitive of exponent zero
    root = math.sqrt(4.0 * math.pi)
    one = (torch.zeros(1, dtype=FP64, device=dev), torch.zeros(1, 3, dtype=FP64, device=dev),
           torch.full((1, 1, 1), root, dtype=FP64, device=dev))
    others = others or {0: one}
    aux = _primitives(ket, dev)
    nb = bra[1].n_functions if bra[1] is not None else 1
    out = torch.zeros(bra[0].n_functions, nb, ket.n_functions, dtype=FP64, device=dev)
    for la, ga in groups.items():
        for lb, gb in others.items():
            p, centre, e, _ = _pairs(la, lb, ga, gb)
            left = _spherical_hermite(la, lb, e)
            for lp, gp in aux.items():
                q, origin, eq, _ = _pairs(lp, 0, gp, one)
                right = {k: c[:, :, 0] * (-1.0) ** sum(k) for k, c in _spherical_hermite(lp, 0, eq).items()}
                for k0 in range(0, len(q), 8):
                    qs = q[None, k0:k0 + 8]
                    alpha = p[:, None] * qs / (p[:, None] + qs)
                    r = _hermite_coulomb(la + lb + lp, alpha, centre[:, None, :] - origin[None, k0:k0 + 8, :])
                    scale = 2.0 * math.pi**2.5 / (p[:, None] * qs * torch.sqrt(p[:, None] + qs))
                    block = 0.0
                    for h, c in left.items():
                        inner = sum(r[h[0] + g[0], h[1] + g[1], h[2] + g[2]][..., None] * w[None, k0:k0 + 8]
                                    for g, w in right.items())
                        block = block + c[:, :, :, None, None] * (scale[..., None] * inner)[:, None, None]
                    pairs = _contract(block, ga, gb)
                    out += torch.einsum("xyqm,zqm->xyz", pairs, root * gp[2][:, k0:k0 + 8])
    return out


def _exact_setup(case, seed):
    state = prepare(case, seed)
    molecule, d = state["molecule"], state["density"]
    dev = d.device
    orbital, auxiliary = (ShellTable.build(b, molecule.symbols, molecule.positions) for b in (case["basis"], AUXILIARY))
    s, h = _one_electron(orbital, molecule, dev)
    metric = _coulomb_integrals((auxiliary, None), auxiliary, dev)[:, 0, :]
    three = _coulomb_integrals((orbital, orbital), auxiliary, dev)
    low = torch.linalg.cholesky(metric)
    n, naux = orbital.n_functions, auxiliary.n_functions
    b = torch.linalg.solve_triangular(low, three.reshape(n * n, naux).T, upper=False).reshape(naux, n, n)
    return {"s": s, "h": h, "j": torch.einsum("quv,q->uv", b, torch.einsum("quv,uv->q", b, 2.0 * d)),
            "k": _plain_exchange(b, d)}
