"""Which tables, scratch and kernels the transforms on the tensor cores take (csrc/digit_gemm.cu), and what happens
where they are not there.

Tolerances as tests/test_gpu_digits.py: 1e-12 for FP64 transforms against the oracle's naive form or against
band-limited data, 1e-11 where the oracle's seminaive form on noise is meant, 5e-7 for FP32.
"""
import numpy as np
import pytest

from s2kit_gb300 import api
from tests._util import harmonic_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cutoff", [1, 4])
def test_low_orders_are_seminaive_below_the_cutoff_only(oracle, cutoff):
    """bw 1024, noise: odd orders 1, 3, 5 as the reference has them, by the cosine series below the cutoff (whose
    rounding shows: 4e-11 at order 1) and by the naive sum from it on."""
    import torch

    import s2kit_gb300 as s2
    bw, S = 1024, 2048
    noise = np.random.default_rng(1025).standard_normal((S, S))
    plan = api.Plan(bw, cutoff)
    rc, ic = (torch.empty(1, bw * bw, dtype=torch.float64, device="cuda") for _ in range(2))
    plan.fst(torch.from_numpy(noise).cuda(), None, rc, ic, 1, api.REAL)
    plan.sync_status()
    rc, ic = rc.cpu().numpy()[0], ic.cpu().numpy()[0]
    del plan
    s2.load().s2g_cache_clear()
    w = oracle.weights(bw)
    for m in (1, 3, 5):
        x = np.fft.rfft(noise, axis=1)[:, m] * (np.sqrt(2 * np.pi) / S)
        if m < cutoff:
            tab = oracle.cos_pml_table(bw, m)
            er, ei = (oracle.dlt_semi(p, bw, m, tab, w) for p in (x.real, x.imag))
        else:
            tab = oracle.pml_table(bw, m)
            er, ei = (oracle.dlt_naive(p, bw, m, w, tab) for p in (x.real, x.imag))
        at = harmonic_index(m, np.arange(m, bw), bw)
        e = np.hypot(rc[at] - er, ic[at] - ei).max() / np.hypot(er, ei).max()
        assert e <= (1e-11 if m < cutoff else 1e-12), (m, e)


def _cuda(*shape, dtype="float64"):
    import torch
    return torch.randn(*shape, dtype=getattr(torch, dtype), device="cuda", generator=torch.Generator("cuda").manual_seed(7))


def _expire(lib, call):
    """call() with the digit kernels' table copies left out: every wait runs out (half a second), nothing hangs."""
    import torch
    assert lib.s2g_test_stall_digits(1) == 0
    try:
        call()
        torch.cuda.synchronize()
    finally:
        lib.s2g_test_stall_digits(0)


def test_expired_wait_is_reported_to_its_own_plan():
    import s2kit_gb300 as s2
    lib, bw, nb = s2.load(), 48, 4
    grid, oc = _cuda(nb, 4 * bw * bw), [_cuda(nb, bw * bw) for _ in range(2)]
    plan, other = api.Plan(bw, bw), api.Plan(bw, bw)
    plan.fst(grid, None, oc[0], oc[1], nb, api.REAL)
    want = oc[0].clone()
    _expire(lib, lambda: plan.fst(grid, None, oc[0], oc[1], nb, api.REAL))
    assert lib.s2g_plan_sync_status(other.h) == 0
    assert lib.s2g_plan_sync_status(plan.h) == 5  # S2G_ERR_TIMEOUT, read and cleared
    assert lib.s2g_plan_sync_status(plan.h) == 0
    plan.fst(grid, None, oc[0], oc[1], nb, api.REAL)
    plan.sync_status()
    assert (oc[0] == want).all()


def test_expired_wait_is_reported_to_its_own_group():
    import s2kit_gb300 as s2
    lib, bws = s2.load(), [77, 77, 32]
    group, other = api.Group(bws), api.Group(bws)
    grid = _cuda(group.grid_total, dtype="float32")
    oc = [_cuda(group.coeff_total, dtype="float32") for _ in range(2)]
    _expire(lib, lambda: group.fst(grid, oc[0], oc[1]))
    assert lib.s2g_group_sync_status(other.h) == 0
    assert lib.s2g_group_sync_status(group.h) == 5
    assert lib.s2g_group_sync_status(group.h) == 0


def test_expired_wait_is_reported_by_the_convolution_drop_in(capfd):
    import s2kit_gb300 as s2
    lib, bw = s2.load(), 48
    a = np.random.default_rng(3).standard_normal((6, 4 * bw * bw))
    api.ConvOn2SphereSemiMemo(*a, bw)
    want = a[4].copy()
    assert capfd.readouterr().err == ""
    _expire(lib, lambda: api.ConvOn2SphereSemiMemo(*a, bw))
    assert "ConvOn2SphereSemiMemo failed (5)" in capfd.readouterr().err
    api.ConvOn2SphereSemiMemo(*a, bw)
    assert capfd.readouterr().err == "" and (a[4] == want).all()
