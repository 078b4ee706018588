"""The sector sweep of targets that conserve particle numbers against the full sweep
(MG_OPT_TARGET_DENSE), which applies the same operations to each amplitude in the same order:
f and gradients must be equal bit for bit, for every block kind, for one, two and many
components, with and without Jordan-Wigner strings, for whole traces and ragged column ranges,
and for sectors that take one, two and four blocks per SM.  Where a sector does not fit in
shared memory (the last case) the tiled sweep runs."""
import numpy as np
import pytest

import mgcu
import targets as T

pytestmark = pytest.mark.gpu


def _center(kind, rng):
    a, s = rng.uniform(0.1, 1.4), np.exp(1j * rng.uniform(0, 6, size=4))
    return {"id": [1, 0, 0, 1], "swap": [0, 1, 1, 0], "neg": [1, 0, 0, -1], "d1": [1, 0, 0, s[0]], "diag": [s[0], 0, 0, s[1]],
            "anti": [0, s[0], s[1], 0], "hop": [np.cos(a), 1j * np.sin(a), 1j * np.sin(a), np.cos(a)],
            "ri": [np.cos(a), np.sin(a), -np.sin(a), np.cos(a)],
            "gen": T.haar_matchgates(1, rng)[0][:4]}[kind]


def _corner(kind, rng):
    s = np.exp(1j * rng.uniform(0, 6, size=2))
    return {"id": [1, 0, 0, 1], "neg": [1, 0, 0, -1], "d1": [1, 0, 0, s[0]], "diag": [s[0], 0, 0, s[1]]}[kind]


def _circuit(L, n, rng, groups, diagonal_only=False):
    """n gates; amplitudes move only within each group of wires"""
    g, w = [], []
    moving, still = ["swap", "anti", "hop", "hop", "ri", "gen", "fswap"], ["id", "neg", "d1", "diag"]
    for _ in range(n):
        grp = groups[int(rng.integers(len(groups)))]
        if len(grp) > 1 and not diagonal_only and rng.random() < 0.7:
            i, j = rng.choice(grp, 2, replace=False)
            kind = moving[int(rng.integers(len(moving)))]
        else:
            i, j = rng.choice(L, 2, replace=False)
            kind = still[int(rng.integers(len(still)))]
        if kind == "fswap":
            # a pair of fermionic swaps around a hop leaves a string (and the order) behind
            k = [q for q in grp if q not in (i, j)]
            if not k:
                continue
            for gg, ww in ((T.FSWAP, (j, k[0])), (T.hop_gate(1.0, 0.3), (i, j)), (T.FSWAP, (j, k[0]))):
                g.append(gg)
                w.append(ww)
            continue
        corner = ["id", "neg", "d1", "diag"][int(rng.integers(4))]
        g.append(np.concatenate([_center(kind, rng), _corner(corner, rng)]).astype(complex))
        w.append((i, j))
    return np.array(g), np.array(w, np.int32)


CASES = [  # L, components, columns (None: all)
    (4, [[0, 1, 2, 3]], None),
    (6, [[0, 2, 4], [1, 3, 5]], None),
    (6, [[0], [1], [2], [3], [4], [5]], None),
    (8, [[0, 1, 2, 3, 4], [5, 6], [7]], (3, 250)),
    (12, [list(range(12))], None),
    (12, [[0, 2, 4, 6, 8, 10], [1, 3, 5, 7, 9, 11]], (1017, 3010)),
    (14, [list(range(14))], (5000, 5300)),
    (16, [list(range(0, 16, 2)), list(range(1, 16, 2))], (21800, 21861)),
    (16, [list(range(16))], (21800, 21861)),
    (18, [list(range(18))], (87000, 87013)),
]


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"L{c[0]}x{len(c[1])}")
def test_sector_sweep_equals_full_sweep(mglib, case, prec):
    lib = mglib
    L, groups, cols = case
    rng = np.random.default_rng(L + 10 * len(groups))
    g, w = _circuit(L, 40, rng, groups)
    v, perms = T.haar_matchgates(2, rng), T.brickwall_perms(L, 2)
    t = lib.target_circuit(g, w, L)
    assert lib.lib.mg_target_conserves_weight(mgcu.P(t)) == 1
    lib.set_precision(prec)
    out = []
    try:
        for dense in (0, 1):
            lib.set_option(mgcu.OPT_TARGET_DENSE, dense)
            out.append(lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, *(cols or (0, 1 << L))))
    finally:
        lib.set_option(mgcu.OPT_TARGET_DENSE, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    (rc0, f0, dv0), (rc1, f1, dv1) = out
    assert rc0 == 0 and rc1 == 0, lib.last_error()
    assert f0 == f1 and np.array_equal(dv0, dv1)


@pytest.mark.parametrize("parts,prec", [(3, mgcu.PREC_FP64), (3, mgcu.PREC_MIXED), (3, mgcu.PREC_FP32), (2, mgcu.PREC_FP32)])
def test_sector_sweep_at_18_qubits(mglib, parts, prec):
    """the largest size of the sector sweep, with conserved numbers enough for its sectors to fit (8000
    rows with three, 15 876 with two): the sector kernel runs and has the full sweep's bits"""
    lib, rng = mglib, np.random.default_rng(parts)
    L = 18
    g, w = _circuit(L, 14, rng, [list(range(i, L, parts)) for i in range(parts)])
    v, perms = T.haar_matchgates(2, rng), T.brickwall_perms(L, 2)
    t = lib.target_circuit(g, w, L)
    lib.set_precision(prec)
    out = []
    try:
        plan = lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_TARGET)
        assert lib.plan_target_kernel(plan) == "k_sector"
        lib.lib.mg_plan_free(mgcu.P(plan))
        for dense in (0, 1):
            lib.set_option(mgcu.OPT_TARGET_DENSE, dense)
            out.append(lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, 87000, 87013))
    finally:
        lib.set_option(mgcu.OPT_TARGET_DENSE, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    (rc0, f0, dv0), (rc1, f1, dv1) = out
    assert rc0 == 0 and rc1 == 0, lib.last_error()
    assert f0 == f1 and np.array_equal(dv0, dv1)
