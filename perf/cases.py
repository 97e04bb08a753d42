"""Measured workloads: operator products, multi-source Helmholtz solves and the
coarse-correction network, each through the package's public entry points.

A case is a dict of plain values; ``kind`` says which entry point it calls:

* ``apply``: ``H @ X`` and its shifted and adjoint forms for a block of device columns;
* ``solve``: ``solveLinearSystem`` for a block of sources on the device, with the
  solver (its hierarchy, workspace and factors) kept between calls as a program
  keeps it over its shot batches;
* ``net``: ``CoarseNet.forward`` / ``gradient`` for a batch of device fields.

The medium and the network's weights belong to the case (a program keeps them);
the right-hand sides and fields come from the seed.
"""
from __future__ import annotations

import json
import math

import numpy as np
import torch
import torch.nn.functional as F

from __graft_entry__ import load_package

hz = load_package()

DEV = "cuda"


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _apply(cells, columns, op="H", adjoint=False):
    return dict(kind="apply", cells="x".join(map(str, cells)), columns=columns, op=op, adjoint=adjoint)


def _solve(cells, sources, levels, cycle, precision="fp64", outer="fp64", krylov="GMRES", tol=1e-6, shift=0.5,
           gmres_smoothing=False, adjoint=False):
    return dict(kind="solve", cells="x".join(map(str, cells)), sources=sources, levels=levels, cycle=cycle,
                precision=precision, outer=outer, krylov=krylov, tol=tol, shift=shift,
                gmres_smoothing=gmres_smoothing, adjoint=adjoint)


def _net(grid, batch, what):
    return dict(kind="net", grid="x".join(map(str, grid)), batch=batch, what=what)


def listed():
    return [
        # one product on a small 2D grid, as a residual check or a user's own
        # Krylov loop takes it: launch latency
        dict(_apply((128, 128), 1), name="apply_2d_one_column"),
        # the adjoint shifted operator on a block of 3D wavefields, ragged node
        # counts and an odd number of columns
        dict(_apply((156, 130, 100), 13, op="SH", adjoint=True), name="apply_3d_block"),
        # one 2D source to a tight tolerance in the default precision
        dict(_solve((128, 128), 1, 4, "V", tol=1e-8), name="solve_2d_one_source"),
        # the default Krylov method (BiCGSTAB) with a W-cycle, a few sources
        dict(_solve((256, 128), 4, 4, "W", krylov="BiCGSTAB", tol=1e-8), name="solve_2d_bicgstab"),
        # a 2D shot gather, mixed precision, K-cycle over five levels
        dict(_solve((1024, 512), 16, 5, "K", precision="mixed"), name="solve_2d_mixed"),
        # a larger gather on a smaller odd-shaped section, emulated outer arithmetic
        dict(_solve((640, 320), 33, 5, "K", precision="mixed", outer="emulated"), name="solve_2d_emulated"),
        # the adjoint sweep of an inversion in the default precision, 3D
        dict(_solve((64, 64, 32), 8, 3, "V", tol=1e-8, adjoint=True), name="solve_3d_adjoint"),
        # 3D sources on 129^3 nodes, mixed precision, K-cycle with GMRES smoothing
        dict(_solve((128, 128, 128), 8, 4, "K", precision="mixed", shift=0.3, gmres_smoothing=True),
             name="solve_3d_mixed"),
        # the largest solve: a wide 3D section over five levels, emulated outer arithmetic
        dict(_solve((192, 160, 96), 16, 5, "K", precision="mixed", outer="emulated", shift=0.3,
                    gmres_smoothing=True), name="solve_3d_emulated"),
        # the 2D coarse-correction network applied to a block of 32 columns
        dict(_net((129, 129), 32, "forward"), name="net_2d_forward"),
        # one training step's loss and weight gradient, 2D and 3D
        dict(_net((129, 129), 32, "gradient"), name="net_2d_gradient"),
        dict(_net((33, 33, 33), 8, "gradient"), name="net_3d_gradient"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, lo, hi, multiple):
    return max(1, round(_logint(rng, lo, hi) / multiple)) * multiple


def draw(rng):
    kind = rng.choice(["apply", "apply", "solve", "solve", "solve", "solve", "net", "net"])
    if kind == "apply":
        op, adj = rng.choice(["H", "SH"]), rng.random() < 0.5
        if rng.random() < 0.5:
            return _apply((_logint(rng, 64, 1024), _logint(rng, 64, 512)), _logint(rng, 1, 64), op, adj)
        return _apply(tuple(_logint(rng, 24, 160) for _ in range(3)), _logint(rng, 1, 16), op, adj)
    if kind == "solve":
        form = rng.choice(["2d", "2d-bicgstab", "2d-block", "3d", "3d-block"])
        precision, outer = rng.choice([("mixed", "fp64"), ("mixed", "emulated")])
        if form == "2d":
            return _solve((_cells(rng, 64, 256, 8), _cells(rng, 64, 256, 8)), _logint(rng, 1, 8), 4, "V", tol=1e-8)
        if form == "2d-bicgstab":
            return _solve((_cells(rng, 64, 256, 8), _cells(rng, 64, 128, 8)), _logint(rng, 1, 8), 4, "W",
                          krylov="BiCGSTAB", tol=1e-8)
        if form == "2d-block":
            return _solve((_cells(rng, 256, 768, 16), _cells(rng, 256, 512, 16)), _logint(rng, 4, 16), 5, "K",
                          precision=precision, outer=outer)
        if form == "3d":
            return _solve((_cells(rng, 24, 64, 4), _cells(rng, 24, 64, 4), _cells(rng, 24, 32, 4)),
                          _logint(rng, 1, 8), 3, "V", tol=1e-8, adjoint=rng.random() < 0.5)
        return _solve((_cells(rng, 64, 128, 16), _cells(rng, 64, 128, 16), _cells(rng, 64, 96, 16)),
                      _logint(rng, 1, 8), 4, "K", precision=precision, outer=outer, shift=0.3, gmres_smoothing=True)
    what = rng.choice(["forward", "gradient"])
    if rng.random() < 0.5:
        return _net((8 * _logint(rng, 4, 20) + 1, 8 * _logint(rng, 4, 16) + 1), _logint(rng, 1, 32), what)
    return _net(tuple(4 * _logint(rng, 4, 8) + 1 for _ in range(3)), _logint(rng, 1, 8), what)


# ---------------------------------------------------------------------------
# Media and inputs
# ---------------------------------------------------------------------------
def _ints(text):
    return tuple(int(v) for v in text.split("x"))


def _medium(cells):
    """Layered velocity 1.5 to 4.5 km/s with an ellipsoidal inclusion, 10 points
    per wavelength, attenuation 0.01 w and a quadratic absorbing layer on every
    side but the surface (the last axis' first plane)."""
    rng = np.random.default_rng(20)
    nodes = [c + 1 for c in cells]
    dim = len(nodes)
    grids = np.ogrid[tuple(slice(0, n) for n in nodes)]
    edges = np.cumsum(rng.uniform(0.5, 1.5, size=9))
    layer = np.searchsorted(edges / edges[-1], np.arange(nodes[-1]) / nodes[-1])
    v = np.broadcast_to(np.sort(rng.uniform(1.5, 4.5, size=10))[layer], nodes).copy()
    centre, axes = rng.uniform(0.3, 0.7, size=dim), rng.uniform(0.08, 0.2, size=dim)
    v[sum(((g / c - o) / a) ** 2 for g, c, o, a in zip(grids, cells, centre, axes)) <= 1.0] = 4.5
    m = (1.0 / v**2).ravel(order="F")
    h = 0.01
    w = 0.2 * math.pi / (h * math.sqrt(m.max()))
    gamma = np.full(nodes, 0.01 * w)
    pad = max(4, min(32, min(cells) // 8))
    for d, (g, c) in enumerate(zip(grids, cells)):
        t = np.maximum(0.0, (pad - g) / pad) if d < dim - 1 else 0.0
        gamma = np.maximum(gamma, 0.95 * w * np.maximum(t, np.maximum(0.0, (g - (c - pad)) / pad)) ** 2)
    return dict(mesh=hz.getRegularMesh([v for c in cells for v in (0.0, h * c)], list(cells)), nodes=nodes, h=h, m=m,
                w=w, gamma=gamma.ravel(order="F"))


_kept = {}  # what the program of one case keeps: its operator, solver or network


def _keep(case, make):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _kept:
        _kept.clear()
        _kept[key] = make()
    return _kept[key]


def _param(med):
    return hz.HelmholtzParam(med["mesh"], med["gamma"], med["m"], med["w"], True, True)


def _make_operator(case):
    med = _medium(_ints(case["cells"]))
    H = hz.GetHelmholtzOperator(_param(med))
    A = H + hz.GetHelmholtzShiftOP(med["m"], med["w"], 0.5) if case["op"] == "SH" else H
    return A.adjoint() if case["adjoint"] else A


def _make_solver(case):
    med = _medium(_ints(case["cells"]))
    MG = hz.getMGparam(complex, int, case["levels"], 1, 200 if case["krylov"] == "GMRES" else 1000, case["tol"],
                       "Jac-GMRES" if case["gmres_smoothing"] else "Jac", 0.8, 1, 1, case["cycle"], "Julia", 0.5, 0.0,
                       precision=case["precision"], outerArithmetic=case["outer"],
                       relaxFrom=1 if case["gmres_smoothing"] else 0)
    return hz.getShiftedLaplacianMultigridSolver(_param(med), MG, case["shift"], case["krylov"], 10)


# (input, output) channels of the networks' layers, forward order
_LAYERS = {2: [(4, 16), (16, 32), (32, 64), (64, 64), (128, 64), (96, 32), (48, 16), (16, 2)],
           3: [(4, 8), (8, 16), (16, 32), (48, 16), (24, 8), (8, 2)]}


def _weights(dim):
    """He-normal weights, layer after layer [cout][taps][cin]."""
    rng = np.random.default_rng(30 + dim)
    return np.concatenate([rng.standard_normal(b * 3**dim * a) * math.sqrt(2.0 / (3**dim * a))
                           for a, b in _LAYERS[dim]]).astype(np.float32)


def _make_net(case):
    dim = len(_ints(case["grid"]))
    net = hz.learned.CoarseNet3D(seed=1) if dim == 3 else hz.learned.CoarseNet(seed=1)
    net.set_weights(_weights(dim))
    return net


def _wavefields(nodes, columns, gen, dtype):
    """Columns of wave-like complex fields, (columns, prod(nodes)) with the first
    axis fastest: a few plane waves at about 10 points per wavelength, and noise."""
    out = 0.1 * torch.randn((columns, *nodes[::-1]), dtype=dtype, generator=gen, device=DEV)
    for _ in range(3):
        phase = torch.rand((columns,) + (1,) * len(nodes), generator=gen, device=DEV, dtype=torch.float64) * 6.28
        for d, n in enumerate(nodes):
            k = (torch.rand((columns,) + (1,) * len(nodes), generator=gen, device=DEV, dtype=torch.float64) - 0.5) * 1.2
            shape = [1] * (len(nodes) + 1)
            shape[-1 - d] = n
            phase = phase + k * torch.arange(n, device=DEV, dtype=torch.float64).reshape(shape)
        out += torch.polar(torch.ones_like(phase), phase).to(dtype)
    return out.reshape(columns, -1)


def _sources(case, seed):
    """Sources of random strength at random surface positions (one node deep);
    adjoint: data residuals along lines of receivers on the surface."""
    nodes = [c + 1 for c in _ints(case["cells"])]
    rng = np.random.default_rng(1000 + seed)
    R, N, nx = case["sources"], math.prod(nodes), nodes[0]
    B = torch.zeros((R, N), dtype=torch.complex128, device=DEV)
    depth = nx if len(nodes) == 2 else nx * nodes[1]
    for c in range(R):
        row = depth + (0 if len(nodes) == 2 else nx * int(rng.integers(nodes[1] // 5, nodes[1] * 4 // 5)))
        if case["adjoint"]:
            i0, i1 = nx // 10, nx - nx // 10
            vals = rng.standard_normal(i1 - i0) + 1j * rng.standard_normal(i1 - i0)
            B[c, row + i0:row + i1] = torch.from_numpy(vals).to(DEV)
        else:
            B[c, row + int(rng.integers(nx // 10, nx - nx // 10))] = 5e3 * complex(*rng.standard_normal(2))
    return B.t()


def _net_inputs(case, seed):
    """(fields and medium, targets) as the solver hands them to the network."""
    nodes = _ints(case["grid"])
    gen = torch.Generator(device=DEV).manual_seed(7000 + seed)
    B = case["batch"]
    r, e = (_wavefields(nodes, B, gen, torch.complex64) for _ in range(2))
    r, e = (v / torch.linalg.vector_norm(v, dim=1, keepdim=True) * math.sqrt(v.shape[1]) for v in (r, e))
    mass = 0.7 + 5.6 * torch.rand(r.shape, generator=gen, device=DEV)
    att = 0.01 + 0.5 * torch.rand(r.shape, generator=gen, device=DEV) ** 4
    x = torch.stack([r.real, r.imag, mass, att], dim=-1).reshape(B, *nodes[::-1], 4).float().contiguous()
    t = (0.2 * torch.stack([e.real, e.imag], dim=-1)).reshape(B, *nodes[::-1], 2).float().contiguous()
    return x, t


def prepare(case, seed):
    if case["kind"] == "apply":
        gen = torch.Generator(device=DEV).manual_seed(5000 + seed)
        X = _wavefields([c + 1 for c in _ints(case["cells"])], case["columns"], gen, torch.complex128)
        return dict(case=case, A=_keep(case, lambda: _make_operator(case)), X=X.t())
    if case["kind"] == "solve":
        return dict(case=case, solver=_keep(case, lambda: _make_solver(case)), B=_sources(case, seed))
    x, t = _net_inputs(case, seed)
    return dict(case=case, net=_keep(case, lambda: _make_net(case)), x=x, t=t)


def run(state):
    case = state["case"]
    if case["kind"] == "apply":
        return state["A"] @ state["X"]
    if case["kind"] == "solve":
        X, _ = hz.solveLinearSystem(None, state["B"], state["solver"], int(case["adjoint"]))
        # wavefields of a 1e-6 solve are kept in single precision, as programs store them
        return X.to(torch.complex64) if case["precision"] == "mixed" else X
    if case["what"] == "forward":
        return state["net"].forward(state["x"])
    loss, grad = state["net"].gradient(state["x"], state["t"])
    return dict(loss=loss, grad=grad)


def work(case):
    if case["kind"] == "apply":
        nodes = [c + 1 for c in _ints(case["cells"])]
        N, R = math.prod(nodes), case["columns"]
        return dict(bytes=N * (32 * R + 16), flops=N * R * (8 * len(nodes) + 8))
    if case["kind"] == "solve":
        N, R = math.prod(c + 1 for c in _ints(case["cells"])), case["sources"]
        return dict(bytes=N * (16 * R + (8 if case["precision"] == "mixed" else 16) * R + 16), flops=0)
    nodes = _ints(case["grid"])
    dim, N = len(nodes), math.prod(nodes)
    levels = [0, 1, 2, 3, 2, 1, 0, 0] if dim == 2 else [0, 1, 2, 1, 0, 0]
    flops = case["batch"] * sum(2 * 3**dim * a * b * math.prod((n - 1) // 2**g + 1 for n in nodes)
                                for (a, b), g in zip(_LAYERS[dim], levels))
    w = 4 * sum(3**dim * a * b for a, b in _LAYERS[dim])
    if case["what"] == "forward":
        return dict(bytes=case["batch"] * N * 24 + w, flops=flops)
    return dict(bytes=case["batch"] * N * 24 + 2 * w, flops=3 * flops)


# ---------------------------------------------------------------------------
# The same results in 64 bits, from the definitions
# ---------------------------------------------------------------------------
def _axis_matrix(n, h):
    """(-d2/dx2) on n nodes: second-order reflecting boundary rows."""
    L = torch.zeros((n, n), dtype=torch.complex128, device=DEV)
    i = torch.arange(n, device=DEV)
    L[i, i] = 2.0 / h**2
    L[i[1:], i[:-1]] = -1.0 / h**2
    L[i[:-1], i[1:]] = -1.0 / h**2
    L[0, 1] = L[n - 1, n - 2] = -2.0 / h**2
    return L


def _mass(med, nodes):
    """The diagonal -w^2 m (1 - i gamma / w) minus the radiation term of the
    outer faces (all but the surface), shaped like the reversed node counts."""
    w, h, dim = med["w"], med["h"], len(nodes)
    m, g = (torch.from_numpy(med[k]).to(DEV).reshape(nodes[::-1]) for k in ("m", "gamma"))
    mass = -(w**2) * m * (1.0 - 1j * g / w)
    for d in range(dim):
        for end in ((0, nodes[d] - 1) if d < dim - 1 else (nodes[d] - 1,)):
            at = [slice(None)] * dim
            at[dim - 1 - d] = end
            mass[tuple(at)] += 1j * w * (2.0 / h) * torch.sqrt(m[tuple(at)])
    return mass


def _exact_apply(case, seed):
    med = _medium(_ints(case["cells"]))
    nodes, R = med["nodes"], case["columns"]
    gen = torch.Generator(device=DEV).manual_seed(5000 + seed)
    X = _wavefields(nodes, R, gen, torch.complex128).reshape(R, *nodes[::-1])
    diag = _mass(med, nodes)
    if case["op"] == "SH":
        diag = diag + 0.5j * med["w"] ** 2 * torch.from_numpy(med["m"]).to(DEV).reshape(nodes[::-1])
    Y = (diag.conj() if case["adjoint"] else diag) * X
    for d, n in enumerate(nodes):
        L = _axis_matrix(n, med["h"])
        L = L.mH if case["adjoint"] else L
        Y += torch.movedim(torch.tensordot(X, L, dims=([len(nodes) - d], [1])), -1, len(nodes) - d)
    return Y.reshape(R, -1).t()


def _exact_solve(case, seed):
    """Block elimination along the longest axis, plane by plane."""
    med = _medium(_ints(case["cells"]))
    nodes, R = med["nodes"], case["sources"]
    dim = len(nodes)
    s = max(range(dim), key=lambda d: nodes[d])
    rest = [d for d in range(dim) if d != s]
    M = math.prod(nodes[d] for d in rest)
    if M > 2200 or nodes[s] * M**3 > 7e11 or nodes[s] * M**2 > 5e9:
        return None
    adj = case["adjoint"]
    mats = [(L.mH.contiguous() if adj else L) for L in (_axis_matrix(n, med["h"]) for n in nodes)]
    mass = torch.movedim(_mass(med, nodes), dim - 1 - s, 0).reshape(nodes[s], M)
    mass = mass.conj() if adj else mass
    plane = torch.zeros((M, M), dtype=torch.complex128, device=DEV)
    for d in rest:
        part = torch.ones((1, 1), dtype=torch.complex128, device=DEV)
        for q in rest:  # the first axis is the fastest index of a plane
            part = torch.kron(mats[q] if q == d else torch.eye(nodes[q], dtype=part.dtype, device=DEV), part)
        plane += part
    B = torch.movedim(_sources(case, seed).t().reshape(R, *nodes[::-1]), dim - s, 0).reshape(nodes[s], R, M)
    Ls, inv, y = mats[s], [], []
    for k in range(nodes[s]):
        S = plane + torch.diag(mass[k] + Ls[k, k])
        b = B[k].t()
        if k:
            S -= (Ls[k, k - 1] * Ls[k - 1, k]) * inv[-1]
            b = b - Ls[k, k - 1] * (inv[-1] @ y[-1])
        inv.append(torch.linalg.inv(S))
        y.append(b)
    X = torch.empty((nodes[s], R, M), dtype=torch.complex128, device=DEV)
    u = None
    for k in reversed(range(nodes[s])):
        u = inv[k] @ (y[k] if u is None else y[k] - Ls[k, k + 1] * u)
        X[k] = u.t()
    shape = [nodes[d] for d in reversed(rest)]
    return torch.movedim(X.reshape(nodes[s], R, *shape), 0, dim - s).reshape(R, -1).t()


def _transfer(n):
    """1D restriction (full weighting, rows summing to one) and prolongation."""
    nc = (n - 1) // 2 + 1
    P = torch.zeros((n, nc), dtype=torch.float64, device=DEV)
    i = torch.arange(n, device=DEV)
    P[i, i // 2] += 0.5
    P[i, (i + 1) // 2] += 0.5
    return P.t() / P.sum(0)[:, None], P


def _resample(x, restrict):
    for ax in range(2, x.dim()):
        n = x.shape[ax]
        T = _transfer(n)[0] if restrict else _transfer(2 * n - 1)[1]
        x = torch.movedim(torch.tensordot(x, T, dims=([ax], [1])), -1, ax)
    return x


def _exact_net(case, seed):
    nodes = _ints(case["grid"])
    dim = len(nodes)
    x, t = _net_inputs(case, seed)
    w = torch.from_numpy(_weights(dim)).to(DEV).double().requires_grad_(True)
    convs, k = [], 0
    for a, b in _LAYERS[dim]:
        n = b * 3**dim * a
        convs.append(torch.movedim(w[k:k + n].reshape(b, *([3] * dim), a), -1, 1))
        k += n
    conv = F.conv3d if dim == 3 else F.conv2d
    v = torch.movedim(x.double(), -1, 1)
    depth, skips = 2 if dim == 3 else 3, []
    for q in range(depth + 1):
        v = torch.relu(conv(_resample(v, True) if q else v, convs[q], padding=1))
        skips.append(v)
    for q in range(depth):
        v = torch.cat([_resample(v, False), skips[depth - 1 - q]], dim=1)
        v = torch.relu(conv(v, convs[depth + 1 + q], padding=1))
    y = torch.movedim(conv(v, convs[-1], padding=1), 1, -1)
    if case["what"] == "forward":
        return y.detach()
    e, td = (y - t.double()).flatten(1), t.double().flatten(1)
    loss = (e.square().sum(1) / td.square().sum(1)).mean()
    loss.backward()
    return dict(loss=float(loss.detach()), grad=w.grad.cpu().numpy())


def exact(case, seed):
    return dict(apply=_exact_apply, solve=_exact_solve, net=_exact_net)[case["kind"]](case, seed)
