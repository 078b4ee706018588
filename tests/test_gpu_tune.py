"""The target sweep's block size chosen by timing (MG_OPT_TARGET_TUNE): every candidate
applies the same operations to each amplitude in the same order, so plans that tuned and
plans that did not must give bit-identical f and gradients, for the weight-restricted sweep
(a Hubbard Trotter target) and the full sweep (Haar matchgate brickwall target), and the
chosen configuration must be one of the candidates."""
import os
import sys

import numpy as np
import pytest

import mgcu
import targets as T

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

pytestmark = pytest.mark.gpu


def _run(lib, t, v, perms, L, tune):
    lib.set_option(mgcu.OPT_TARGET_TUNE, tune)
    try:
        plan = lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_GRADIENT)
    finally:
        lib.set_option(mgcu.OPT_TARGET_TUNE, 0)
    try:
        cfg = lib.plan_target_config(plan)
        assert lib.lib.mg_plan_run(mgcu.P(plan)) == 0, lib.last_error()
        f, dv, _, _, _ = lib.plan_results(plan, len(v), grad=True)
    finally:
        lib.lib.mg_plan_free(mgcu.P(plan))
    return cfg, f, dv


@pytest.mark.parametrize("kind,L,prec", [("hubbard", 12, mgcu.PREC_MIXED), ("hubbard", 14, mgcu.PREC_FP64),
                                         ("haar", 12, mgcu.PREC_MIXED), ("haar", 14, mgcu.PREC_FP32)])
def test_tuned_sweep_is_bit_identical(mglib, kind, L, prec):
    lib = mglib
    rng = np.random.default_rng(L + prec)
    if kind == "hubbard":
        g, w, v, perms = bench.workload(L, 3, 4, seed=L)
        t = lib.target_circuit(g, w, L)
    else:
        ul, up = T.haar_matchgates(6, rng), T.brickwall_perms(L, 6)
        v, perms = T.haar_matchgates(3, rng), T.brickwall_perms(L, 3)
        t = lib.target_brickwall(ul, up, L)
    lib.set_precision(prec)
    try:
        c1, f1, dv1 = _run(lib, t, v, perms, L, 1)   # the static choice
        c2, f2, dv2 = _run(lib, t, v, perms, L, 2)   # timed
        c3, f3, dv3 = _run(lib, t, v, perms, L, 2)   # the cached choice
    finally:
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    assert c1["kind"] == (2 if kind == "hubbard" else 1)
    assert c2 == c3 and c2["kind"] == c1["kind"] and c2["tile_bits"] == c1["tile_bits"]
    if c2["kind"] == 2:
        assert (c2["threads"], c2["per_thread"]) in [(128, 2), (256, 1)]
    else:
        assert c2["threads"] in (128, 256, 512)
    assert f1 == f2 == f3
    assert np.array_equal(dv1, dv2) and np.array_equal(dv1, dv3)


# The tiled sweeps by themselves: by default a target whose sectors fit in shared memory is swept by
# k_sector and others from L = 10 by k_fit, which have no block size to choose.  CTAS_PER_SM (32: no
# limit in effect) keeps k_target_w, TARGET_DENSE keeps k_target.
TILED = {"hubbard": ("k_target_w", mgcu.OPT_CTAS_PER_SM, 32), "haar": ("k_target", mgcu.OPT_TARGET_DENSE, 1)}


def _target(lib, kind, L, rng):
    if kind == "hubbard":
        g, w, v, perms = bench.workload(L, 3, 4, seed=L)
        return lib.target_circuit(g, w, L), v, perms
    ul, up = T.haar_matchgates(6, rng), T.brickwall_perms(L, 6)
    return lib.target_brickwall(ul, up, L), T.haar_matchgates(3, rng), T.brickwall_perms(L, 3)


@pytest.mark.parametrize("kind,L,prec", [("hubbard", 12, mgcu.PREC_MIXED), ("hubbard", 14, mgcu.PREC_FP64), ("hubbard", 14, mgcu.PREC_FP32),
                                         ("haar", 14, mgcu.PREC_MIXED), ("haar", 14, mgcu.PREC_FP32), ("haar", 14, mgcu.PREC_FP64)])
def test_tiled_sweep_is_timed(mglib, kind, L, prec):
    """the timing runs on the tiled sweeps: plans of the static, the timed and the cached choice run
    the named kernel with the same bits, and only the timed one launches sweeps as it is made"""
    lib, rng = mglib, np.random.default_rng(L + prec)
    name, opt, value = TILED[kind]
    t, v, perms = _target(lib, kind, L, rng)
    lib.set_precision(prec)
    lib.set_option(opt, value)
    launched, res = [], []
    try:
        for tune in (1, 2, 2):   # the static choice, timed, the cached choice
            lib.set_option(mgcu.OPT_TARGET_TUNE, tune)
            n = lib.launch_count()
            plan = lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_GRADIENT)
            launched.append(lib.launch_count() - n)
            assert lib.plan_target_kernel(plan) == name
            cfg = lib.plan_target_config(plan)
            assert lib.lib.mg_plan_run(mgcu.P(plan)) == 0, lib.last_error()
            f, dv, _, _, _ = lib.plan_results(plan, len(v), grad=True)
            lib.lib.mg_plan_free(mgcu.P(plan))
            res.append((cfg, f, dv))
    finally:
        lib.set_option(mgcu.OPT_TARGET_TUNE, 0)
        lib.set_option(opt, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    assert launched[1] >= launched[0] + 4 and launched[2] == launched[0]   # two runs of two candidates or more
    assert res[1][0] == res[2][0]
    assert (res[1][0]["threads"], res[1][0]["per_thread"]) in ([(128, 2), (256, 1)] if kind == "hubbard" else [(128, 1), (256, 1), (512, 1)])
    for _, f, dv in res[1:]:
        assert f == res[0][1] and np.array_equal(dv, res[0][2])


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("L,cols,prec", [(12, (0, 4096), mgcu.PREC_MIXED), (12, (1000, 1031), mgcu.PREC_FP64), (14, (5000, 5101), mgcu.PREC_FP32),
                                         (16, (21800, 21837), mgcu.PREC_MIXED), (16, (65530, 65536), mgcu.PREC_FP64)])
def test_weight_restricted_tiled_sweep(mglib, oracle, L, cols, prec, threads):
    """k_target_w at both of its block sizes against the full sweep, bit for bit, and (a few columns)
    against the oracle at the precision's tolerance elsewhere in these tests"""
    lib = mglib
    g, w, v, perms = bench.workload(L, 3, 2, seed=L)
    t = lib.target_circuit(g, w, L)
    lib.set_precision(prec)
    out = []
    try:
        for dense in (0, 1):
            lib.set_option(mgcu.OPT_TARGET_DENSE, dense)
            lib.set_option(mgcu.OPT_TARGET_THREADS, 0 if dense else threads)
            plan = lib.plan_brickwall(lib.mg_target_apply, t, v, perms, L, mgcu.EVAL_TARGET)
            assert lib.plan_target_kernel(plan) == ("k_target" if dense else "k_target_w")
            assert dense or lib.plan_target_config(plan)["threads"] == threads
            lib.lib.mg_plan_free(mgcu.P(plan))
            out.append([lib.brickwall_columns(lib.mg_target_apply, t, v, perms, L, *r) for r in (cols, (cols[0], cols[0] + 3))])
    finally:
        lib.set_option(mgcu.OPT_TARGET_DENSE, 0)
        lib.set_option(mgcu.OPT_TARGET_THREADS, 0)
        lib.set_precision(mgcu.PREC_FP64)
        lib.target_free(t)
    for (rc0, f0, dv0), (rc1, f1, dv1) in zip(*out):
        assert rc0 == 0 and rc1 == 0
        assert f0 == f1 and np.array_equal(dv0, dv1)
    f_o, dv_o = oracle.brickwall_target_and_gradient(oracle.Target("circuit", L, gates=g, wires=w), v, perms, L, col_range=(cols[0], cols[0] + 3))
    tol = {mgcu.PREC_FP64: 1e-12, mgcu.PREC_MIXED: 1e-9, mgcu.PREC_FP32: 1e-4}[prec]
    _, f, dv = out[0][1]
    assert abs(f - f_o) <= tol * np.max(np.abs(dv_o)) and np.max(np.abs(dv - dv_o)) <= tol * np.max(np.abs(dv_o))
