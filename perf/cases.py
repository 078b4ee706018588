"""Performance cases: the evaluations that a user of the matchgate library runs, through its
public entry points, from one small gradient call to a share of an L=16 trace.

A case is a dict of plain values.  Its "kind" names the entry point:

  gradient   matchgate_brickwall_unitary_target_and_projected_gradient (host buffers)
  plan       a kept gradient plan: new gates, one evaluation, results read back
  columns    mg_brickwall_target_and_gradient_columns over [b0, b1)
  hessian    matchgate_brickwall_unitary_target_gradient_vector_hessian_matrix
  ti         matchgate_ti_brickwall_unitary_target_gradient_hessian
  circuit_value, circuit_hessian   the same for general circuits (any qubit count)
  batch      a kept batch of fits of different sizes: new gates, one run, results read back
  fit        mg_optimize_brickwall (trust-region iterations)

"target" is "random" (Haar matchgate brickwall or circuit, depth layers or gates), "hubbard"
(spinful Fermi-Hubbard second-order Trotter circuit of `depth` steps) or "spinless" (spinless
Hubbard brickwall, `depth` steps of the 6th-order Suzuki rule).  "prec" is fp64, mixed or fp32.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rqcopt_hpc-matchgate_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mgcu  # noqa: E402
import targets as T  # noqa: E402

PREC = {"fp64": mgcu.PREC_FP64, "mixed": mgcu.PREC_MIXED, "fp32": mgcu.PREC_FP32}


def listed():
    return [
        # the smallest evaluation, called thousands of times by a host optimiser: latency
        {"name": "gradient_L4_fp64", "kind": "gradient", "target": "random", "L": 4, "layers": 3, "depth": 6, "prec": "fp64"},
        # the reference's plain test configuration: L=8, 4 layers, depth-8 random target, f + gradient + Hessian
        {"name": "hessian_L8_fp64", "kind": "hessian", "target": "random", "L": 8, "layers": 4, "depth": 8, "prec": "fp64"},
        # an odd number of qubits and a ragged gate list: f alone of a general circuit, as a line search asks for it
        {"name": "circuit_value_L13_fp32", "kind": "circuit_value", "target": "random", "L": 13, "gates": 47, "depth": 131, "prec": "fp32"},
        # one parameter block per gate on an odd chain: the per-gate Newton step
        {"name": "circuit_hessian_L9_mixed", "kind": "circuit_hessian", "target": "random", "L": 9, "gates": 19, "depth": 37, "prec": "mixed"},
        # a random target of twice the fitted depth (the batch and serving workload), one fit at a time
        {"name": "plan_random_L12_mixed", "kind": "plan", "target": "random", "L": 12, "layers": 7, "depth": 14, "prec": "mixed"},
        # the spinful Hubbard target in the library's default precision
        {"name": "gradient_hubbard_L12_fp64", "kind": "gradient", "target": "hubbard", "L": 12, "layers": 5, "depth": 64, "prec": "fp64"},
        # the larger fit of the Hubbard configurations: L=14, 9 layers, the optimiser's kept plan
        {"name": "plan_hubbard_L14_mixed", "kind": "plan", "target": "hubbard", "L": 14, "layers": 9, "depth": 64, "prec": "mixed"},
        # one rank's share of the headline trace (L=16, 5 layers, 64 Trotter steps), ragged range
        {"name": "columns_hubbard_L16_mixed", "kind": "columns", "target": "hubbard", "L": 16, "layers": 5, "depth": 64,
         "b0": 20011, "b1": 26012, "prec": "mixed"},
        # the published benchmark's model: spinless target, 5 layers, f + gradient + per-layer Hessian
        {"name": "hessian_spinless_L12_fp64", "kind": "hessian", "target": "spinless", "L": 12, "layers": 5, "depth": 12, "prec": "fp64"},
        # its translation-invariant Hessian, deeper fit
        {"name": "ti_spinless_L12_mixed", "kind": "ti", "target": "spinless", "L": 12, "layers": 9, "depth": 4, "prec": "mixed"},
        # many fits of uneven size and depth at once
        {"name": "batch_L8_12_fp32", "kind": "batch", "target": "random", "L": 8, "L2": 12, "count": 12, "prec": "fp32"},
        # two trust-region iterations of the native optimiser
        {"name": "fit_spinless_L10_mixed", "kind": "fit", "target": "spinless", "L": 10, "layers": 5, "depth": 3, "iters": 2, "prec": "mixed"},
    ]


def draw(rng):
    limit = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["gradient", "plan", "columns", "hessian", "ti", "circuit_value", "circuit_hessian", "batch", "fit"])
        c = {"kind": kind, "prec": rng.choice(["fp64", "mixed", "fp32"] if kind != "fit" else ["fp64", "mixed"])}
        c["target"] = rng.choice(["random", "hubbard", "spinless"])
        if kind in ("circuit_value", "circuit_hessian"):
            c["target"] = "random"
            c["L"] = rng.randint(4, 14 if kind == "circuit_value" else 10)
            c["gates"] = rng.randint(2 * c["L"], 6 * c["L"]) if kind == "circuit_value" else rng.randint(c["L"], 3 * c["L"])
            c["depth"] = rng.randint(2 * c["L"], 16 * c["L"])
        elif kind == "batch":
            c.update(target="random", L=2 * rng.randint(3, 5), L2=2 * rng.randint(5, 6), count=rng.randint(2, 24))
        else:
            if kind == "columns":
                c["L"] = 2 * rng.randint(6, 8)
            elif kind in ("gradient", "plan"):
                c["L"] = 2 * rng.randint(2, 7)
            else:
                c["L"] = 2 * rng.randint(2, 6) if kind != "fit" else 2 * rng.randint(2, 5)
            c["layers"] = rng.randint(2, 9)
            if c["target"] == "random":
                c["depth"] = rng.randint(2, 18)
            elif c["target"] == "hubbard":
                c["depth"] = int(round(2 ** rng.uniform(2, 6)))
            else:
                c["depth"] = int(round(2 ** rng.uniform(0, 3.6)))
            if kind == "columns":
                n = 1 << c["L"]
                w = int(round(math.exp(rng.uniform(math.log(200), math.log(min(n, 8000))))))
                c["b0"] = rng.randint(0, n - w)
                c["b1"] = c["b0"] + w
            if kind == "fit":
                c["iters"] = rng.randint(1, 2)
        if _cost(c) <= limit:
            return c


# ----------------------------------------------------------------------------- inputs
def _target(case, rng):
    """(gates, wires) of the target circuit"""
    L, d = case["L"], case["depth"]
    if case["target"] == "random":
        if "layers" not in case:
            return T.haar_matchgates(d, rng), _chain_wires(L, d, rng)
        u, p = T.haar_matchgates(d, rng), T.brickwall_perms(L, d)
        return _expand(u, p, L)
    if case["target"] == "hubbard":
        J, U = 1.0 + 0.1 * rng.uniform(-1, 1), 4.0 + rng.uniform(-1, 1)
        return T.hubbard_trotter_circuit(L // 2, J, U, 0.25, d)[:2]
    g = 1.5 + 0.5 * rng.uniform(-1, 1)
    u, p = T.spinless_hubbard_brickwall(L, 1.0, g, d / 12.0, d, 6)
    return _expand(u, p, L)


def _expand(layers, perms, L):
    """brickwall layers as a gate list"""
    g = np.repeat(np.asarray(layers), L // 2, axis=0)
    return g, np.asarray(perms, np.int32).reshape(-1, 2)


def _chain_wires(L, n, rng):
    """n nearest-neighbour pairs in random places and orders"""
    a = rng.integers(0, L - 1, size=n)
    w = np.stack([a, a + 1], axis=1)
    flip = rng.integers(0, 2, size=n).astype(bool)
    w[flip] = w[flip][:, ::-1]
    return w.astype(np.int32)


def _fit_gates(case, rng):
    """initial fitted layers: a spinless fit starts from the model's own second-order splitting,
    perturbed inside the particle-conserving gates; the others from the identity plus noise or
    random layers, as their configurations do"""
    L, nl = case["L"], case["layers"]
    if case["target"] == "random":
        return T.haar_matchgates(nl, rng), T.brickwall_perms(L, nl)
    if case["target"] == "hubbard":
        return T.near_identity_brickwall(nl, rng), T.brickwall_perms(L, nl)
    t = case["depth"] / 12.0
    v = np.array([T.spinless_hubbard_gate(1.0, 1.5 + 0.1 * rng.uniform(-1, 1), t / nl * (1 + 0.1 * rng.uniform(-1, 1)))
                  for _ in range(nl)])
    return v, T.brickwall_perms(L, nl)


class _State:
    """what a user's program keeps: the library, the GPU target, gates and any kept plan"""

    def __init__(self, case):
        self.case, self.lib = case, mgcu.default_lib()
        self.targets, self.plan, self.batch = [], None, None

    def circuit(self, gates, wires, L):
        self.targets.append(self.lib.target_circuit(gates, wires, L))
        return self.targets[-1]

    def __del__(self):
        if self.plan:
            self.lib.lib.mg_plan_free(mgcu.P(self.plan))
        if self.batch:
            self.lib.batch_free(self.batch)
        for t in self.targets:
            self.lib.target_free(t)


def _batch_instances(case, seed):
    shape = np.random.default_rng(1000 * case["L"] + 10 * case["L2"] + case["count"])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        L = 2 * int(shape.integers(case["L"] // 2, case["L2"] // 2 + 1))
        nl = int(shape.integers(3, 10))
        ug, uw = _expand(T.haar_matchgates(2 * nl, rng), T.brickwall_perms(L, 2 * nl), L)
        out.append({"L": L, "ug": ug, "uw": uw, "v": T.haar_matchgates(nl, rng), "perms": T.brickwall_perms(L, nl)})
    return out


def _inputs(case, seed):
    """(target gates, target wires, fitted gates, perms or wires)"""
    rng = np.random.default_rng(seed)
    ug, uw = _target(case, rng)
    if case["kind"].startswith("circuit"):
        return ug, uw, T.haar_matchgates(case["gates"], rng), _chain_wires(case["L"], case["gates"], rng)
    return (ug, uw) + _fit_gates(case, rng)


def prepare(case, seed):
    s = _State(case)
    lib = s.lib
    lib.set_precision(PREC[case["prec"]])
    if case["kind"] == "batch":
        inst = _batch_instances(case, seed)
        ts = [s.circuit(x["ug"], x["uw"], x["L"]) for x in inst]
        s.v = [x["v"] for x in inst]
        s.batch = lib.batch_create(ts, s.v, [x["perms"] for x in inst], [x["L"] for x in inst])
        return s
    ug, uw, s.v, s.perms = _inputs(case, seed)
    s.t = s.circuit(ug, uw, case["L"])
    if case["kind"] == "plan":
        s.plan = lib.plan_brickwall(lib.mg_target_apply, s.t, s.v, s.perms, case["L"], mgcu.EVAL_GRADIENT)
    return s


def _ok(rc, s):
    if rc != 0:
        raise RuntimeError(s.lib.last_error())


def run(s):
    lib, case = s.lib, s.case
    kind, L, fn = case["kind"], case["L"], lib.mg_target_apply
    lib.set_precision(PREC[case["prec"]])
    if kind == "gradient":
        rc, f, g = lib.brickwall_projected_gradient(fn, s.t, s.v, s.perms, L)
        _ok(rc, s)
        return [f, g]
    if kind == "plan":
        _ok(lib.lib.mg_plan_set_gates(mgcu.P(s.plan), mgcu.gates_arr(s.v).ctypes.data_as(mgcu.P)), s)
        _ok(lib.lib.mg_plan_run(mgcu.P(s.plan)), s)
        f, dv, _, g, _ = lib.plan_results(s.plan, case["layers"], grad=True, proj=True)
        return [f, dv, g]
    if kind == "columns":
        rc, f, dv = lib.brickwall_columns(fn, s.t, s.v, s.perms, L, case["b0"], case["b1"])
        _ok(rc, s)
        return [f, dv]
    if kind == "hessian":
        rc, f, g, H = lib.brickwall_gradvec_hessmat(fn, s.t, s.v, s.perms, L)
        _ok(rc, s)
        return [f, g, H]
    if kind == "ti":
        rc, f, dv, h = lib.brickwall_target_gradient_hessian(fn, s.t, s.v, s.perms, L, ti=True)
        _ok(rc, s)
        return [f, dv, h]
    if kind == "circuit_value":
        rc, f = lib.circuit_target(fn, s.t, s.v, s.perms, L)
        _ok(rc, s)
        return [f]
    if kind == "circuit_hessian":
        rc, f, dg, h = lib.circuit_target_gradient_hessian(fn, s.t, s.v, s.perms, L)
        _ok(rc, s)
        return [f, dg, h]
    if kind == "batch":
        for i, v in enumerate(s.v):
            _ok(lib.batch_set_gates(s.batch, i, v), s)
        _ok(lib.batch_run(s.batch), s)
        return [x for i in range(len(s.v)) for x in lib.batch_results(s.batch, i)]
    f_iter, _, v = lib.optimize_native(s.t, s.v, s.perms, L, case["iters"],
                                       refine_gnorm=1e-300 if case["prec"] == "mixed" else 0.0)
    return [f_iter, v]


# ----------------------------------------------------------------------------- work
def _amplitudes(target, L):
    """nonzero amplitudes of all columns U e_b: the parity sector, or the particle number
    (per spin for the spinful model) that the target conserves"""
    if target == "hubbard":
        return math.comb(L, L // 2) ** 2
    return math.comb(2 * L, L) if target == "spinless" else 1 << (2 * L - 1)


def _counts(case):
    """(target gates, fitted gates, fraction of the columns, Hessian gate steps)"""
    L, d = case["L"], case["depth"]
    if "layers" in case:
        gw = case["layers"] * (L // 2)
        if case["target"] == "hubbard":
            n = L // 2
            hops = 2 * (n // 2), 2 * ((n - 1) // 2)
            gu = n + d * (2 * hops[0] + hops[1] + n)
        elif case["target"] == "spinless":
            gu = (d * 50 + 1) * (L // 2)
        else:
            gu = d * (L // 2)
    else:
        gu, gw = d, case["gates"]
    frac = (case["b1"] - case["b0"]) / float(1 << L) if "b0" in case else 1.0
    steps = 0
    if case["kind"] in ("hessian", "ti", "fit"):
        steps = 8 * sum(gw - i * (L // 2) for i in range(case["layers"]))
    elif case["kind"] == "circuit_hessian":
        steps = 8 * (gw * (gw - 1) // 2)
    return gu, gw, frac, steps


def _flops(case):
    if case["kind"] == "batch":
        return sum(_flops({"kind": "plan", "target": "random", "L": x["L"], "layers": len(x["v"]), "depth": 2 * len(x["v"])})
                   for x in _batch_instances(case, 0))
    gu, gw, frac, steps = _counts(case)
    amps, sector = _amplitudes(case["target"], case["L"]), 1 << (2 * case["L"] - 1)
    per = (14 if case["kind"] == "circuit_value" else 44) * gw + 8
    one = frac * (14.0 * gu * amps + (per + 30.0 * steps) * sector)
    if case["kind"] == "fit":
        one = case["iters"] * (one + (14.0 * gw + 8) * sector)
    return one


def _cost(case):
    return _flops(case) * {"fp64": 4.0, "mixed": 1.5, "fp32": 1.0}[case["prec"]]


def work(case):
    if case["kind"] == "batch":
        inst = _batch_instances(case, 0)
        nbytes = sum(128 * len(x["ug"]) + 128 * len(x["v"]) * 2 + 16 + 64 * len(x["v"]) for x in inst)
    else:
        gu, gw, _, steps = _counts(case)
        nb = case.get("layers", gw)
        nbytes = 128 * (gu + 2 * nb) + 16 + 64 * nb + (8 * 64 * nb * nb * (1 if case["kind"] == "hessian" else 2) if steps else 0)
    return {"bytes": nbytes, "flops": _flops(case)}


# ----------------------------------------------------------------------------- 64-bit values
# the trace restated with dense tensors: a state matrix holds one full 2^L vector per basis column
def _quarters(M, i, j, L):
    """views of the amplitudes |00>, |01>, |10>, |11> of wires (i, j)"""
    a, b = min(i, j), max(i, j)
    V = M.view(1 << a, 2, 1 << (b - a - 1), 2, -1)
    q = [[V[:, p, :, r] for r in (0, 1)] for p in (0, 1)]
    if i < j:
        return q[0][0], q[0][1], q[1][0], q[1][1]
    return q[0][0], q[1][0], q[0][1], q[1][1]


def _mix(p, q, m):
    """(p, q) <- m (p, q) in place"""
    if m[1] == 0 and m[2] == 0:
        if m[0] != 1:
            p.mul_(m[0])
        if m[3] != 1:
            q.mul_(m[3])
        return
    t = p * m[0]
    t.add_(q, alpha=m[1])
    q.mul_(m[3]).add_(p, alpha=m[2])
    p.copy_(t)


def _gate(M, g, w, L, how="n"):
    """one gate on the state matrix; how: n itself, t its transpose, h its adjoint"""
    g = [complex(x) for x in g]
    if how != "n":
        g = [g[0], g[2], g[1], g[3], g[4], g[6], g[5], g[7]]
    if how == "h":
        g = [x.conjugate() for x in g]
    x, y, z, ww = _quarters(M, int(w[0]), int(w[1]), L)
    _mix(y, z, g[:4])
    _mix(x, ww, g[4:])


def _contract(D, S, w, L):
    """sum_columns d_r s_c for the 8 block entries of a gate"""
    dx, dy, dz, dw = _quarters(D, int(w[0]), int(w[1]), L)
    x, y, z, ww = _quarters(S, int(w[0]), int(w[1]), L)
    return torch.stack([(p * q).sum() for p, q in ((dy, y), (dy, z), (dz, y), (dz, z), (dx, x), (dx, ww), (dw, x), (dw, ww))]).cpu().numpy()


def _basis(L, b0, b1):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    M = torch.zeros((1 << L, b1 - b0), dtype=torch.complex128, device=dev)
    r = torch.arange(b1 - b0, device=dev)
    M[r + b0, r] = 1
    return M


def _target_matrix(ug, uw, L, b0, b1):
    M = _basis(L, b0, b1)
    for g, w in zip(ug, uw):
        _gate(M, g, w, L)
    return torch.conj_physical(M).neg_()


def _evaluate(D, g, w, L, b0, b1, grad=True, items=None):
    """f, per-gate gradients and, for items = [(gates that add entry x, {later gate: weight})], the
    sums A[item][x][gate][y] of placeholder states contracted with the derivative entering each gate"""
    S = _basis(L, b0, b1)
    inputs = []
    for gg, ww in zip(g, w):
        if items is not None:
            inputs.append(S.clone())
        _gate(S, gg, ww, L)
    f = np.complex128((D * S).sum().item())
    if not grad:
        return f, None, None
    dg = np.zeros((len(g), 8), complex)
    D = D.clone()
    ders = [None] * len(g)
    for k in range(len(g) - 1, -1, -1):
        _gate(S, g[k], w[k], L, "h")
        dg[k] = _contract(D, S, w[k], L)
        if items is not None:
            ders[k] = D.clone()
        _gate(D, g[k], w[k], L, "t")
    if items is None:
        return f, dg, None
    del S, D
    A = np.zeros((len(items), 8, len(g), 8), complex)
    for n, (adds, weight) in enumerate(items):
        for x in range(8):
            B = None
            for k in range(min(adds), len(g)):
                if B is not None:
                    if k in weight:
                        A[n, x, k] = weight[k] * _contract(ders[k], B, w[k], L)
                    _gate(B, g[k], w[k], L)
                if k in adds:
                    if B is None:
                        B = torch.zeros_like(inputs[k])
                    out, src = _quarters(B, int(w[k][0]), int(w[k][1]), L), _quarters(inputs[k], int(w[k][0]), int(w[k][1]), L)
                    rows = (1, 2) if x < 4 else (0, 3)
                    out[rows[(x >> 1) & 1]].add_(src[rows[x & 1]])
    return f, dg, A


def _brickwall_hessian(D, v, perms, L, ti):
    """f, layer gradients and the complex Hessian of the layers"""
    g, w = _expand(v, perms, L)
    nl, half = len(v), L // 2
    items = []
    for l in range(nl):
        k = l * half
        if ti:   # the layer's first pair, weighted by its translated copies
            items.append(({k}, {s: half - ((s - k) if s // half == l else 0) for s in range(k + 1, nl * half)}))
        else:
            items.append((set(range(k, k + half)), {s: 1 for s in range(k + 1, nl * half)}))
    f, dg, A = _evaluate(D, g, w, L, 0, 1 << L, True, items)
    A = A.reshape(nl, 8, nl, half, 8).sum(3).reshape(8 * nl, 8 * nl)
    return f, dg.reshape(nl, half, 8).sum(1), A + A.T


def _blocks(z):
    return [np.asarray(z[:4]).reshape(2, 2), np.asarray(z[4:]).reshape(2, 2)]


def _to_real(v, z):
    """coordinates of z in the tangent space at v: entries of the anti-Hermitian part of v^H z"""
    out = []
    for a, b in zip(_blocks(v), _blocks(z)):
        m = a.conj().T @ b
        m = (m - m.conj().T) / 2
        out.append((m.real + m.imag).reshape(4))
    return np.concatenate(out)


def _antisymm(r):
    out = []
    for q in (r[:4], r[4:]):
        c = 0.5 * (q[1] - q[2]) + 0.5j * (q[1] + q[2])
        out.append(np.array([[1j * q[0], c], [-np.conj(c), 1j * q[3]]]))
    return out


def _project(v, dv, h=None):
    """Riemannian gradient and Hessian in real coordinates"""
    nb = len(v)
    grad = np.concatenate([_to_real(v[i], dv[i].conj()) for i in range(nb)])
    if h is None:
        return grad, None
    H = np.zeros((8 * nb, 8 * nb))
    for j in range(nb):
        for k in range(8):
            r = np.zeros(8)
            r[k] = 1
            Z = [a @ b for a, b in zip(_blocks(v[j]), _antisymm(r))]
            z = np.concatenate([b.reshape(4) for b in Z])
            for i in range(j + 1):
                G = _blocks((h[8 * i:8 * i + 8, 8 * j:8 * j + 8] @ z).conj())
                if i == j:
                    new = []
                    for u, p, zz, d in zip(_blocks(v[i]), G, Z, _blocks(dv[i].conj())):
                        m = u.conj().T @ p
                        p = p - u @ ((m + m.conj().T) / 2)
                        dh = d.conj().T
                        new.append(p - 0.5 * (zz @ dh @ u + u @ dh @ zz))
                    G = new
                H[8 * i:8 * i + 8, 8 * j + k] = _to_real(v[i], np.concatenate([b.reshape(4) for b in G]))
    return grad, np.triu(H) + np.triu(H, 1).T


def _tcg(g, H, radius, maxiter, abstol=1e-8, reltol=1e-6):
    """Steihaug's truncated conjugate gradients; (step, ended on the boundary)"""
    z, r, d = np.zeros_like(g), g.copy(), -g
    tol = max(abstol, reltol * np.sqrt(r @ r))
    for _ in range(maxiter):
        hd = H @ d
        dd, zd, zz = d @ d, z @ d, z @ z - radius * radius
        tb = (-zd + np.sqrt(zd * zd - dd * zz)) / dd
        a = (r @ r) / (d @ hd)
        if d @ hd <= 0 or a > tb:
            return z + tb * d, True
        rr = r @ r
        r, z = r + a * hd, z + a * d
        if np.sqrt(r @ r) <= tol:
            return z, False
        d = (r @ r) / rr * d - r
    return z, False


def _retract(v, eta):
    out = []
    for a, b in zip(_blocks(v), _antisymm(eta)):
        u, _, vh = np.linalg.svd(a @ (np.eye(2) + b))
        out.append((u @ vh).reshape(4))
    return np.concatenate(out)


def _exact_fit(D, v, perms, L, iters):
    nl, radius, fs = len(v), 0.01, []
    fx = None
    for _ in range(iters):
        f, dv, h = _brickwall_hessian(D, v, perms, L, False)
        grad, H = _project(v, dv, h)
        fs.append(f.real)
        eta, edge = _tcg(grad, H, radius, 2 * 16 * nl)
        vn = np.array([_retract(v[i], eta[8 * i:8 * i + 8]) for i in range(nl)])
        fn = _evaluate(D, *_expand(vn, perms, L), L, 0, 1 << L, False)[0].real
        rho = (fn - f.real) / (grad @ eta + 0.5 * eta @ H @ eta)
        if rho < 0.25:
            radius *= 0.25
        elif rho > 0.75 and edge:
            radius = min(2 * radius, 0.1)
        if rho > 0.125:
            v, fx = vn, fn
        elif fx is None:
            fx = f.real
    return [np.array(fs + [fx]), v]


def exact(case, seed):
    kind, L = case["kind"], case["L"]
    if not torch.cuda.is_available() and _flops(case) > 1e10:
        return None
    if kind == "batch":
        out = []
        for x in _batch_instances(case, seed):
            D = _target_matrix(x["ug"], x["uw"], x["L"], 0, 1 << x["L"])
            f, dg, _ = _evaluate(D, *_expand(x["v"], x["perms"], x["L"]), x["L"], 0, 1 << x["L"])
            dv = dg.reshape(len(x["v"]), -1, 8).sum(1)
            out += [f, dv, _project(x["v"], dv)[0]]
        return out
    ug, uw, v, perms = _inputs(case, seed)
    b0, b1 = case.get("b0", 0), case.get("b1", 1 << L)
    if float(b1 - b0) * (1 << L) * (len(ug) + 10 * len(perms)) > 2e12:
        return None   # over about 20 seconds
    D = _target_matrix(ug, uw, L, b0, b1)
    if kind == "fit":
        return _exact_fit(D, v, perms, L, case["iters"])
    if kind in ("hessian", "ti"):
        f, dv, h = _brickwall_hessian(D, v, perms, L, kind == "ti")
        return [f, dv, h] if kind == "ti" else [f, *_project(v, dv, h)]
    if kind == "circuit_value":
        return [_evaluate(D, v, perms, L, b0, b1, False)[0]]
    if kind == "circuit_hessian":
        n = len(v)
        f, dg, A = _evaluate(D, v, perms, L, b0, b1, True, [({k}, {s: 1 for s in range(k + 1, n)}) for k in range(n)])
        A = A.reshape(8 * n, 8 * n)
        return [f, dg, A + A.T]
    f, dg, _ = _evaluate(D, *_expand(v, perms, L), L, b0, b1)
    dv = dg.reshape(case["layers"], -1, 8).sum(1)
    if kind == "columns":
        return [f, dv]
    g = _project(v, dv)[0]
    return [f, dv, g] if kind == "plan" else [f, g]
