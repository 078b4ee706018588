"""The factored fitted circuit (the default for gradients from 10 qubits, for f alone from 12)
against the general kernels (kept by an explicit MG_OPT_THREADS), which apply the unfactored
blocks: single tiles, several tiles per pass, odd qubit counts with an idle wire, gates whose
off-diagonal entries dominate, gates on the dropped last qubit in both orders, diagonal and
antidiagonal blocks, blocks of gates with equal matrices and one block per gate, non-unitary
gates, ragged column ranges, and gates that do not factor (the general kernels run).

Tolerances: both sides round each amplitude independently, so they agree within the precision of
the sweep: 1e-12 in complex128, 1e-9 in float-float, 1e-4 in FP32, relative to the largest
gradient entry, as elsewhere in these tests."""
import numpy as np
import pytest

import mgcu
import targets as T

pytestmark = pytest.mark.gpu

TOL = {mgcu.PREC_FP64: 1e-12, mgcu.PREC_MIXED: 1e-9, mgcu.PREC_FP32: 1e-4}


def _both(lib, call, tile_bits):
    """the factored result and the general kernels'"""
    out = []
    for threads in (0, 256):
        lib.set_option(mgcu.OPT_THREADS, threads)
        lib.set_option(mgcu.OPT_TILE_BITS, tile_bits)
        try:
            out.append(call())
        finally:
            lib.set_option(mgcu.OPT_THREADS, 0)
            lib.set_option(mgcu.OPT_TILE_BITS, 0)
    return out


def _check(out, tol):
    (rc0, f0, dv0), (rc1, f1, dv1) = out
    assert rc0 == 0 and rc1 == 0
    assert abs(f0 - f1) <= tol * max(abs(f1), np.max(np.abs(dv1)))
    assert np.max(np.abs(dv0 - dv1)) <= tol * np.max(np.abs(dv1))


def _layers(kind, n, rng):
    if kind == "haar":
        return T.haar_matchgates(n, rng)
    if kind == "near":
        return T.near_identity_brickwall(n, rng)
    v = T.haar_matchgates(n, rng)
    if kind == "special":   # diagonal, antidiagonal, identity and swapped blocks
        for i in range(n):
            c, k = [([1, 0, 0, 1j], [0, 1, 1j, 0]), ([0, 1, 1, 0], [1, 0, 0, 1]), ([1, 0, 0, 1], v[i, 4:]),
                    (v[i, :4], [1, 0, 0, -1])][i % 4]
            v[i] = np.concatenate([c, k])
    if kind == "scaled":    # not unitary, well conditioned
        v = v * (1 + 0.3 * rng.uniform(-1, 1, size=v.shape))
    if kind == "singular":  # does not factor
        v[n // 2, :4] = [1, 1, 1, 1]
    return v


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
@pytest.mark.parametrize("L,nl,kind,tile_bits,cols", [
    (10, 1, "haar", 0, None), (10, 5, "near", 0, None), (10, 4, "special", 0, (3, 1001)), (10, 3, "scaled", 6, None),
    (10, 3, "singular", 0, None), (10, 4, "haar", 5, None), (12, 3, "special", 7, (100, 1900)), (12, 6, "haar", 0, (5, 6)),
    (14, 2, "haar", 0, (4000, 4500)), (16, 2, "haar", 0, (30000, 30100))])
def test_brickwall_gradient(mglib, L, nl, kind, tile_bits, cols, prec):
    lib, rng = mglib, np.random.default_rng(L + nl)
    v, perms = _layers(kind, nl, rng), T.brickwall_perms(L, nl)
    t = lib.target_brickwall(T.haar_matchgates(4, rng), T.brickwall_perms(L, 4), L)
    lib.set_precision(prec)
    try:
        _check(_both(lib, lambda: lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, *(cols or (0, 1 << L))), tile_bits), TOL[prec])
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
@pytest.mark.parametrize("L,ng,tile_bits,grad", [(11, 1, 0, True), (11, 23, 0, True), (12, 17, 6, True), (13, 31, 0, True),
                                                 (12, 40, 0, False), (13, 29, 8, False)])
def test_circuit(mglib, L, ng, tile_bits, grad, prec):
    lib, rng = mglib, np.random.default_rng(L + ng)
    w = np.array([rng.choice(L, 2, replace=False) for _ in range(ng)], np.int32)   # any pairs, both orders, some on wire L - 1
    w[: ng // 3, 1] = L - 1
    w[: ng // 3, 0] = rng.integers(0, L - 1, size=ng // 3)
    w[::2] = w[::2, ::-1]
    g = T.haar_matchgates(ng, rng)
    u = T.haar_matchgates(20, rng)
    uw = np.array([rng.choice(L, 2, replace=False) for _ in range(20)], np.int32)
    t = lib.target_circuit(u, uw, L)
    lib.set_precision(prec)
    try:
        if grad:
            out = _both(lib, lambda: lib.circuit_target_and_gradient(lib.mg_target_apply, t, g, w, L), tile_bits)
        else:
            out = [(rc, f, np.ones(1) * np.sqrt(2.0 ** L)) for rc, f in _both(lib, lambda: lib.circuit_target(lib.mg_target_apply, t, g, w, L), tile_bits)]
        _check(out, TOL[prec])
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
@pytest.mark.parametrize("L,nl,kind,ti", [(8, 1, "haar", False), (8, 4, "special", False), (8, 4, "scaled", True), (10, 3, "haar", True),
                                          (10, 5, "near", False), (8, 3, "singular", False), (12, 2, "haar", False)])
def test_layer_hessian(mglib, L, nl, kind, ti, prec):
    """factored Hessian items against k_hessian's; the same tolerances, relative to the largest entry"""
    lib, rng = mglib, np.random.default_rng(L + nl)
    v, perms = _layers(kind, nl, rng), T.brickwall_perms(L, nl)
    t = lib.target_brickwall(T.haar_matchgates(4, rng), T.brickwall_perms(L, 4), L)
    lib.set_precision(prec)
    try:
        out = _both(lib, lambda: lib.brickwall_target_gradient_hessian(lib.mg_target_apply, t, v, perms, L, ti=ti), 0)
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    _check([o[:3] for o in out], TOL[prec])
    assert np.max(np.abs(out[0][3] - out[1][3])) <= TOL[prec] * np.max(np.abs(out[1][3]))


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
@pytest.mark.parametrize("L,ng", [(7, 1), (7, 20), (9, 17), (11, 9)])
def test_gate_hessian(mglib, L, ng, prec):
    lib, rng = mglib, np.random.default_rng(L + ng)
    w = np.array([rng.choice(L, 2, replace=False) for _ in range(ng)], np.int32)
    w[: ng // 3, 1], w[: ng // 3, 0] = L - 1, rng.integers(0, L - 1, size=ng // 3)
    w[::2] = w[::2, ::-1]
    g, u = T.haar_matchgates(ng, rng), T.haar_matchgates(20, rng)
    t = lib.target_circuit(u, np.array([rng.choice(L, 2, replace=False) for _ in range(20)], np.int32), L)
    lib.set_precision(prec)
    try:
        out = _both(lib, lambda: lib.circuit_target_gradient_hessian(lib.mg_target_apply, t, g, w, L), 0)
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    _check([o[:3] for o in out], TOL[prec])
    assert np.max(np.abs(out[0][3] - out[1][3])) <= TOL[prec] * max(np.max(np.abs(out[1][3])), np.max(np.abs(out[1][2])))


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
@pytest.mark.parametrize("L,nu,cols", [(10, 1, None), (10, 33, (5, 1020)), (11, 40, None), (13, 25, (300, 420)), (14, 30, (9000, 9040)),
                                       (15, 30, (9000, 9040)), (16, 40, (65000, 65020))])
def test_target_columns(mglib, L, nu, cols, prec):
    """columns of a target without conserved numbers by k_fit (the default from 10 qubits) against
    the full sweep (MG_OPT_TARGET_DENSE): whole blocks in the same order in FP32, so the same
    bits; factored otherwise"""
    lib, rng = mglib, np.random.default_rng(L + nu)
    u = T.haar_matchgates(nu, rng)
    uw = np.array([rng.choice(L, 2, replace=False) for _ in range(nu)], np.int32)
    uw[:: 5, 0], uw[:: 5, 1] = L - 1, rng.integers(0, L - 1, size=len(uw[:: 5]))
    t = lib.target_circuit(u, uw, L)
    lib.set_precision(prec)
    out = []
    try:
        for dense in (0, 1):
            lib.set_option(mgcu.OPT_TARGET_DENSE, dense)
            if L % 2 == 0:
                v, perms = T.haar_matchgates(2, np.random.default_rng(1)), T.brickwall_perms(L, 2)
                out.append(lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, *(cols or (0, 1 << L))))
            else:
                rc, f, dg = lib.circuit_target_and_gradient(lib.mg_target_apply, t, T.haar_matchgates(3, np.random.default_rng(1)),
                                                            [[0, 1], [L - 1, 2], [3, L - 1]], L)
                out.append((rc, f, dg))
    finally:
        lib.set_option(mgcu.OPT_TARGET_DENSE, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    if prec == mgcu.PREC_FP32:
        assert out[0][1] == out[1][1] and np.array_equal(out[0][2], out[1][2])
    _check(out, TOL[prec])


def _conserving(n, rng):
    """random gates with diagonal corner blocks"""
    v = T.haar_matchgates(n, rng)
    v[:, 4:] = 0
    v[:, 4], v[:, 7] = np.exp(1j * rng.uniform(0, 6, n)), np.exp(1j * rng.uniform(0, 6, n))
    v[::3, :4] = np.array([T.hop_gate(1.0, x)[:4] for x in rng.uniform(0, 1.5, len(v[::3]))])
    return v


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
@pytest.mark.parametrize("L,n,kind", [(8, 1, "layer"), (8, 4, "layer"), (10, 3, "ti"), (10, 4, "layer"), (12, 2, "ti"), (14, 1, "layer"),
                                      (7, 1, "gate"), (7, 18, "gate"), (9, 14, "gate"), (11, 7, "gate")])
def test_conserving_hessian(mglib, L, n, kind, prec):
    """fits and targets that conserve the particle number: number sectors against k_hessian's items,
    with and without the conservation broken in one gate (then the parity sectors run)"""
    lib, rng = mglib, np.random.default_rng(L + n)
    u = _conserving(24, rng)
    t = lib.target_circuit(u, np.array([rng.choice(L, 2, replace=False) for _ in range(24)], np.int32), L)
    w = np.array([rng.choice(L, 2, replace=False) for _ in range(n)], np.int32)
    lib.set_precision(prec)
    try:
        for broken in (False, True):
            v = _conserving(n, rng)
            if broken:
                v[n // 2] = T.haar_matchgates(1, rng)[0]
            if kind == "gate":
                out = _both(lib, lambda: lib.circuit_target_gradient_hessian(lib.mg_target_apply, t, v, w, L), 0)
            else:
                out = _both(lib, lambda: lib.brickwall_target_gradient_hessian(lib.mg_target_apply, t, v, T.brickwall_perms(L, n), L, ti=kind == "ti"), 0)
            _check([o[:3] for o in out], TOL[prec])
            assert np.max(np.abs(out[0][3] - out[1][3])) <= TOL[prec] * max(np.max(np.abs(out[1][3])), np.max(np.abs(out[1][2])))
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
def test_batch_gates_change_kernels(mglib, prec):
    """a captured batch whose gates stop factoring and factor again: each run equals the same fits
    run as plans"""
    lib, rng = mglib, np.random.default_rng(5)
    Ls, nls = [10, 12, 12], [3, 2, 4]
    ts = [lib.target_brickwall(T.haar_matchgates(4, rng), T.brickwall_perms(L, 4), L) for L in Ls]
    perms = [T.brickwall_perms(L, nl) for L, nl in zip(Ls, nls)]
    good = [T.haar_matchgates(nl, rng) for nl in nls]
    bad = [_layers("singular", nl, rng) for nl in nls]
    lib.set_precision(prec)
    try:
        b = lib.batch_create(ts, good, perms, Ls)
        for vs in (good, bad, good):
            for i, v in enumerate(vs):
                assert lib.batch_set_gates(b, i, v) == 0
            assert lib.batch_run(b) == 0
            for i, (t, v, L) in enumerate(zip(ts, vs, Ls)):
                f, dv, _ = lib.batch_results(b, i)
                _check([(0, f, dv), lib.brickwall_target_and_gradient(lib.mg_target_apply, t, v, perms[i], L)], TOL[prec])
        lib.batch_free(b)
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        for t in ts:
            lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
def test_batch_gates_change_factors(mglib, prec):
    """a captured batch whose gates go from unitary to scaled (complex q) and back: each run equals
    the same fits run as plans"""
    lib, rng = mglib, np.random.default_rng(6)
    Ls, nls = [12, 12], [3, 2]
    ts = [lib.target_brickwall(T.haar_matchgates(4, rng), T.brickwall_perms(L, 4), L) for L in Ls]
    perms = [T.brickwall_perms(L, nl) for L, nl in zip(Ls, nls)]
    unitary, scaled = [[_layers(kind, nl, rng) for nl in nls] for kind in ("haar", "scaled")]
    lib.set_precision(prec)
    try:
        b = lib.batch_create(ts, unitary, perms, Ls)
        for vs in (unitary, scaled, [unitary[0], scaled[1]], unitary):
            for i, v in enumerate(vs):
                assert lib.batch_set_gates(b, i, v) == 0
            assert lib.batch_run(b) == 0
            for i, (t, v, L) in enumerate(zip(ts, vs, Ls)):
                f, dv, _ = lib.batch_results(b, i)
                _check([(0, f, dv), lib.brickwall_target_and_gradient(lib.mg_target_apply, t, v, perms[i], L)], TOL[prec])
        lib.batch_free(b)
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        for t in ts:
            lib.target_free(t)


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e-160, 1e5])
def test_extreme_gate_entries(mglib, bad):
    """an entry that is not finite, denormal-like or huge gives what the general kernels give"""
    lib, rng = mglib, np.random.default_rng(3)
    L = 10
    v, perms = T.haar_matchgates(3, rng), T.brickwall_perms(L, 3)
    v[1, 1] = bad
    t = lib.target_brickwall(T.haar_matchgates(2, rng), T.brickwall_perms(L, 2), L)
    try:
        (rc0, f0, dv0), (rc1, f1, dv1) = _both(lib, lambda: lib.brickwall_target_and_gradient(lib.mg_target_apply, t, v, perms, L), 0)
    finally:
        lib.target_free(t)
    assert rc0 == 0 and rc1 == 0
    np.testing.assert_allclose([f0, *dv0.reshape(-1)], [f1, *dv1.reshape(-1)], rtol=1e-12, atol=1e-12 * np.nanmax(np.abs(dv1)) if np.isfinite(bad) else 0)


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
def test_resident_columns_follow_the_sweep(mglib, prec, first):
    """a resident target evaluated with the factored sweep and with the full one
    (MG_OPT_TARGET_DENSE), in both orders: each result has the bits of the same sweep on a target
    that is not resident, whatever filled the columns before"""
    lib, rng = mglib, np.random.default_rng(11)
    L = 10
    ul, up = T.haar_matchgates(8, rng), T.brickwall_perms(L, 8)
    v, perms = T.haar_matchgates(3, rng), T.brickwall_perms(L, 3)

    def run(t, dense):
        lib.set_option(mgcu.OPT_TARGET_DENSE, dense)
        rc, f, dv = lib.brickwall_target_and_gradient(lib.mg_target_apply, t, v, perms, L)
        assert rc == 0, lib.last_error()
        return f, dv
    lib.set_precision(prec)
    ts = [lib.target_brickwall(ul, up, L) for _ in range(2)]
    try:
        want = [run(ts[0], dense) for dense in (0, 1)]
        assert not np.array_equal(want[0][1], want[1][1])   # the two sweeps round differently
        assert lib.target_set_resident(ts[1], True) == 0
        for dense in (first, 1 - first, first):
            f, dv = run(ts[1], dense)
            assert f == want[dense][0] and np.array_equal(dv, want[dense][1])
    finally:
        lib.set_option(mgcu.OPT_TARGET_DENSE, 0)
        lib.set_precision(mgcu.PREC_FP64)
        for t in ts:
            lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
def test_batch_created_with_gates_that_do_not_factor(mglib, prec):
    """the reduction's flags from creation on: gates that do not factor, then some that do, then
    none again, without a run between two changes of the same instance"""
    lib, rng = mglib, np.random.default_rng(8)
    Ls, nls = [12, 12, 10], [2, 3, 2]
    ts = [lib.target_brickwall(T.haar_matchgates(4, rng), T.brickwall_perms(L, 4), L) for L in Ls]
    perms = [T.brickwall_perms(L, nl) for L, nl in zip(Ls, nls)]
    good, bad = [[_layers(kind, nl, rng) for nl in nls] for kind in ("haar", "singular")]
    lib.set_precision(prec)
    try:
        b = lib.batch_create(ts, bad, perms, Ls)
        for steps in ((bad,), (good, [bad[0], good[1], good[2]]), (bad, good, bad)):
            for vs in steps:
                for i, v in enumerate(vs):
                    assert lib.batch_set_gates(b, i, v) == 0
            assert lib.batch_run(b) == 0
            for i, (t, v, L) in enumerate(zip(ts, vs, Ls)):
                f, dv, _ = lib.batch_results(b, i)
                _check([(0, f, dv), lib.brickwall_target_and_gradient(lib.mg_target_apply, t, v, perms[i], L)], TOL[prec])
        lib.batch_free(b)
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        for t in ts:
            lib.target_free(t)


def _free_bytes(lib):
    import ctypes
    lib.lib.mgcu_device_free_bytes.restype = ctypes.c_double
    return lib.lib.mgcu_device_free_bytes()


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
def test_deep_target_keeps_no_tables(mglib, prec):
    """a target whose factored tables would pass their limit (70 layers of 4 MB): the tiled sweep
    runs, and what the target keeps once the plan is gone is its gate program, not the tables"""
    lib, rng = mglib, np.random.default_rng(3)
    L, ul = 18, 70
    v, perms = T.haar_matchgates(1, rng), T.brickwall_perms(L, 1)
    t = lib.target_brickwall(T.haar_matchgates(ul, rng), T.brickwall_perms(L, ul), L)
    lib.set_precision(prec)
    out = []
    try:
        before = _free_bytes(lib)
        plan = lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_TARGET)
        lib.lib.mg_plan_free(mgcu.P(plan))
        assert before - _free_bytes(lib) < 64 << 20
        for dense in (0, 1):
            lib.set_option(mgcu.OPT_TARGET_DENSE, dense)
            out.append(lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, 1000, 1003))
        assert out[0][0] == 0 and out[1][0] == 0
        assert out[0][1] == out[1][1] and np.array_equal(out[0][2], out[1][2])
    finally:
        lib.set_option(mgcu.OPT_TARGET_DENSE, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
def test_deep_fit_plans_stay_small(mglib, prec):
    """a fitted circuit whose factored tables would pass a plan's limit (600 layers of 4 MB): the
    general kernels run, in about the memory that they take by themselves (MG_OPT_THREADS)"""
    lib, rng = mglib, np.random.default_rng(4)
    L, nl = 18, 600
    v, perms = T.haar_matchgates(nl, rng), T.brickwall_perms(L, nl)
    t = lib.target_brickwall(T.haar_matchgates(2, rng), T.brickwall_perms(L, 2), L)
    lib.set_precision(prec)
    used = []
    try:
        for threads in (256, 0, 256):   # (the first also makes what the target keeps)
            lib.set_option(mgcu.OPT_THREADS, threads)
            before = _free_bytes(lib)
            plan = lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_TARGET)
            used.append(before - _free_bytes(lib))
            lib.lib.mg_plan_free(mgcu.P(plan))
        assert abs(used[1] - used[2]) < 512 << 20
        lib.set_option(mgcu.OPT_THREADS, 0)
        _check([(rc, f, np.ones(1)) for rc, f, _ in _both(lib, lambda: lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, 7, 9, gradient=False), 0)],
               TOL[prec])
    finally:
        lib.set_option(mgcu.OPT_THREADS, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
@pytest.mark.parametrize("nl,updates", [(3, 400), (140, 12)])
def test_updates_queued_without_waiting(mglib, prec, nl, updates):
    """gates set and runs queued one after the other, with no result read in between (many small
    uploads, and uploads of 700 gates, past 64 KB): the results are the last gates', bit for bit
    those of a plan that had them from the start"""
    lib, rng = mglib, np.random.default_rng(6)
    L = 10
    perms = T.brickwall_perms(L, nl)
    t = lib.target_brickwall(T.haar_matchgates(4, rng), T.brickwall_perms(L, 4), L)
    vs = [np.ascontiguousarray(T.haar_matchgates(nl, rng)) for _ in range(updates)]
    lib.set_precision(prec)
    out = []
    try:
        for first, rest in ((vs[-1], []), (vs[0], vs[1:])):
            plan = lib.plan_brickwall(lib.mg_target_apply, t, first, perms, L, mgcu.EVAL_GRADIENT)
            assert lib.lib.mg_plan_run(mgcu.P(plan)) == 0
            for v in rest:
                assert lib.lib.mg_plan_set_gates(mgcu.P(plan), v.ctypes.data_as(mgcu.P)) == 0
                assert lib.lib.mg_plan_run(mgcu.P(plan)) == 0
            out.append(lib.plan_results(plan, nl, grad=True))
            lib.lib.mg_plan_free(mgcu.P(plan))
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])


def _on_own_stream(lib, work):
    """work() on a host thread with a stream of its own, as the request server's plan lane has"""
    import ctypes
    import threading
    L = lib.lib
    L.mgcu_stream_create.restype = ctypes.c_void_p
    err = []

    def body():
        s = L.mgcu_stream_create()
        L.mgcu_stream_set(ctypes.c_void_p(s))
        try:
            work()
            assert L.mgcu_stream_sync() == 0
        except BaseException as x:   # handed to the caller's thread
            err.append(x)
        finally:
            L.mgcu_stream_set(None)
            L.mgcu_stream_destroy(ctypes.c_void_p(s))
    th = threading.Thread(target=body)
    th.start()
    return th, err


def _two_streams(lib, prec, L, conserving, resident, rounds=12):
    """two plans of one target whose sweeps differ in tile size, so that each replaces the other's
    gate program, run by two threads on two streams without waiting for results in between"""
    rng = np.random.default_rng(L)
    ul = T.brickwall_perms(L, 6)
    u = T.haar_matchgates(6, rng)
    if conserving:
        u[:, 4:] = [1, 0, 0, np.exp(0.3j)]
    v, perms = T.haar_matchgates(3, rng), T.brickwall_perms(L, 3)
    t = lib.target_brickwall(u, ul, L)
    lib.set_precision(prec)
    plans, want, got = [], [], [[], []]
    try:
        assert lib.target_set_resident(t, resident) == 0
        for bits in (0, 7):
            lib.set_option(mgcu.OPT_TARGET_TILE_BITS, bits)
            plans.append(lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_GRADIENT))
            assert lib.lib.mg_plan_run(mgcu.P(plans[-1])) == 0
            want.append(lib.plan_results(plans[-1], 3, grad=True))

        def runs(i):
            for _ in range(rounds):
                for _ in range(3):
                    assert lib.lib.mg_plan_run(mgcu.P(plans[i])) == 0
                got[i].append(lib.plan_results(plans[i], 3, grad=True))
        th, err = _on_own_stream(lib, lambda: runs(1))
        runs(0)
        th.join()
        assert not err, err
    finally:
        lib.set_option(mgcu.OPT_TARGET_TILE_BITS, 0)
        lib.set_precision(mgcu.PREC_FP64)
        for plan in plans:
            lib.lib.mg_plan_free(mgcu.P(plan))
        lib.target_free(t)
    for i in range(2):
        for f, dv, *_ in got[i]:
            assert f == want[i][0] and np.array_equal(dv, want[i][1])


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
@pytest.mark.parametrize("conserving", [False, True])
def test_two_streams_share_a_target(mglib, prec, conserving):
    _two_streams(mglib, prec, 12, conserving, False)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED])
def test_two_streams_share_resident_columns(mglib, prec):
    """the same with the target's columns resident: each plan's sweep replaces the other's columns"""
    _two_streams(mglib, prec, 12, False, True)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
def test_largest_brickwall(mglib, oracle, prec):
    """18 qubits, the largest size of the factored kernels: columns of the target and gradient of the
    fit by k_fit in several passes, against the oracle and the general kernels on a few columns"""
    lib, rng = mglib, np.random.default_rng(18)
    L, nl, ul = 18, 3, 4
    u, up = T.haar_matchgates(ul, rng), T.brickwall_perms(L, ul)
    v, perms = _layers("scaled", nl, rng), T.brickwall_perms(L, nl)
    t = lib.target_brickwall(u, up, L)
    lib.set_precision(prec)
    try:
        plan = lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_TARGET)
        assert lib.plan_target_kernel(plan) == "k_fit"
        lib.lib.mg_plan_free(mgcu.P(plan))
        for cols in ((0, 3), (200001, 200004)):
            out = _both(lib, lambda: lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, *cols), 0)
            _check(out, TOL[prec])
            f_o, dv_o = oracle.brickwall_target_and_gradient(oracle.Target("brickwall", L, ulist=u, uperms=up), v, perms, L, col_range=cols)
            _check([out[0], (0, f_o, dv_o)], TOL[prec])
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)


@pytest.mark.parametrize("prec", [mgcu.PREC_FP64, mgcu.PREC_MIXED, mgcu.PREC_FP32])
def test_largest_odd_circuit(mglib, prec):
    """17 qubits, whole trace: k_fit's columns and gradient against the full sweep and the general kernels"""
    lib, rng = mglib, np.random.default_rng(17)
    L, ng = 17, 5
    pairs = lambda n: np.array([rng.choice(L, 2, replace=False) for _ in range(n)], np.int32)   # noqa: E731
    w = pairs(ng)
    w[0] = (L - 1, 3)
    g, t = T.haar_matchgates(ng, rng), lib.target_circuit(T.haar_matchgates(4, rng), pairs(4), L)
    lib.set_precision(prec)
    out = []
    try:
        for dense, threads in ((0, 0), (1, 256)):
            lib.set_option(mgcu.OPT_TARGET_DENSE, dense)
            lib.set_option(mgcu.OPT_THREADS, threads)
            out.append(lib.circuit_target_and_gradient(lib.mg_target_apply, t, g, w, L))
        _check(out, TOL[prec])
    finally:
        lib.set_option(mgcu.OPT_TARGET_DENSE, 0)
        lib.set_option(mgcu.OPT_THREADS, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
