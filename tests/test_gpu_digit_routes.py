"""Which tables, scratch and kernels the transforms on the tensor cores take (csrc/digit_gemm.cu), and what happens
where they are not there.

Tolerances as tests/test_gpu_digits.py: 1e-12 for FP64 transforms against the oracle's naive form or against
band-limited data, 1e-11 where the oracle's seminaive form on noise is meant, 5e-7 for FP32.
"""
import ctypes
import json

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
    assert lib.s2g_test_digits(1) == 0
    try:
        call()
        torch.cuda.synchronize()
    finally:
        lib.s2g_test_digits(0)


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


# ---- the kernels that run where the digit tables, or the scratch they need, are not there --------------------------
# The tests of those kernels, with their own tolerances, which by default meet the digit products.
@pytest.fixture(params=[2, 3], ids=["no-tables", "no-scratch"])
def withheld(request):
    import s2kit_gb300 as s2
    lib = s2.load()
    assert lib.s2g_test_digits(request.param) == 0
    lib.s2g_prof_enable(1)
    try:
        yield
        buf = ctypes.create_string_buffer(1 << 16)
        assert lib.s2g_prof_report(buf, len(buf)) == 0
        kernels = json.loads(buf.value)
        assert kernels and not [k for k in kernels if k.startswith(("dg_rows", "dg_leg_"))], kernels
    finally:
        lib.s2g_prof_enable(0)
        lib.s2g_test_digits(0)


def test_without_digits_fp64_plans(withheld, oracle):
    from tests import test_gpu_fp64 as t
    for bw, cutoff in ((64, 64), (32, 10), (256, 256)):
        t.test_batched_real_fast_path(oracle, bw, cutoff)
    t.test_batched_complex_and_conv(oracle)
    t.test_single_function_bw256_fwd_inv_conv(oracle)
    for bw, fmt in ((31, api.REAL), (48, api.COMPLEX), (127, api.REAL)):
        t.test_fp64_non_power_of_two_bandwidths_vs_oracle(oracle, bw, fmt)


def test_without_digits_fly_plans(withheld, oracle):
    from tests import test_gpu_fly as t
    for bw, fmt, nb in ((100, api.COMPLEX, 2), (256, api.COMPLEX, 8), (64, api.REAL, 9)):
        t.test_fly_plan_vs_oracle(oracle, bw, fmt, nb)


@pytest.mark.parametrize("bw,nb", [(255, 8), (64, 9), (1024, 16)])
def test_without_digits_refinement(withheld, bw, nb):
    from tests import test_gpu_configs as t
    t.test_split_with_fp64_residual_refinement(bw, nb, api.PREC_BF16X3)


@pytest.mark.parametrize("prec", [api.PREC_BF16X3, api.PREC_FP16X2])
def test_without_digits_chirp_z_stages(withheld, oracle, prec):
    from tests import test_gpu_complex, test_gpu_split as t
    for bw, nb in ((65, 3), (100, 70), (127, 2), (130, 5), (255, 33)):
        t.test_split_forward_inverse_vs_fp64(bw, nb, prec)
    if prec == api.PREC_BF16X3:
        for bw in (101, 255):
            t.test_split_non_power_of_two_vs_oracle(oracle, bw)
        for bw, nb in ((101, 3), (100, 2)):
            test_gpu_complex.test_split_complex_vs_fp64_path(bw, nb)


def test_without_digits_groups(withheld):
    from tests import test_gpu_group as t
    t.test_group_equals_uniform_path_bitwise(api.PREC_FP16X2, [77, 64, 100, 16, 77, 255, 256, 17, 101, 33])


def test_without_digits_host_buffers(withheld):
    import torch
    bw, nb = 77, 150  # several chunks
    plan = api.Plan(bw, bw)
    g = _cuda(nb, 4 * bw * bw, dtype="float32")
    oc = [torch.empty(nb, bw * bw, dtype=torch.float32, device="cuda") for _ in range(2)]
    plan.fst_real_f32(g, oc[0], oc[1], nb, api.PREC_BF16X3)
    hc = [np.zeros((nb, bw * bw), np.float32) for _ in range(2)]
    plan.fst_real_f32_host(g.cpu().numpy(), hc[0], hc[1], nb, api.PREC_BF16X3)
    for a, b in zip(oc, hc):
        assert (a.cpu().numpy() == b).all()


@pytest.mark.parametrize("warm", [False, True], ids=["tables-not-there", "tables-there"])
def test_capture_before_the_first_digit_call(warm):
    """Nothing can be allocated under capture: the call takes the FP64 kernels, whose scratch a zonal transform has
    sized, whether or not another plan of the bandwidth has built the digit tables."""
    import torch
    bw, nb = 45 if warm else 46, 4
    grid, oc = _cuda(nb, 4 * bw * bw), [_cuda(nb, bw * bw) for _ in range(2)]
    if warm:
        other = api.Plan(bw, bw)
        other.fst(grid, None, oc[0], oc[1], nb, api.REAL)
    plan = api.Plan(bw, bw)
    plan.fzt(grid, None, oc[0], oc[1], nb, api.REAL)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.fst(grid, None, oc[0], oc[1], nb, api.REAL, stream=torch.cuda.current_stream())
    grid.mul_(2.0)
    graph.replay()
    torch.cuda.synchronize()
    got = [c.clone() for c in oc]
    plan.fst(grid, None, oc[0], oc[1], nb, api.REAL)
    plan.sync_status()
    scale = torch.hypot(oc[0], oc[1]).max()
    assert (torch.hypot(got[0] - oc[0], got[1] - oc[1]).max() / scale).item() <= 1e-11


@pytest.mark.parametrize("kind,bw,nb", [("fly", 256, 2), ("fly", 64, 9), ("fly", 512, 1), ("f64", 100, 5), ("f64", 16, 3),
                                        ("conv", 64, 9), ("complex32", 255, 64), ("complex32", 128, 40), ("real32", 101, 64)])
def test_workspace_size_covers_the_scratch_a_call_takes(kind, bw, nb):
    import torch
    f32 = kind.endswith("32")
    dt, prec = ("float32", api.PREC_BF16X3) if f32 else ("float64", api.PREC_FP64)
    grid, out = ([_cuda(nb, 4 * bw * bw, dtype=dt) for _ in range(2)] for _ in range(2))
    oc = [_cuda(nb, bw * bw, dtype=dt) for _ in range(2)]

    def call(plan):
        if kind == "complex32":
            plan.fst_complex_f32(*grid, *oc, nb, prec)
        elif kind == "real32":
            plan.fst_real_f32(grid[0], *oc, nb, prec)
        elif kind == "conv":
            plan.conv(*grid, *grid, *out, nb)
        else:
            plan.fst(*grid, *oc, nb, api.COMPLEX)
        plan.sync_status()

    plans = [api.Plan(bw, bw, fly=kind == "fly") for _ in range(2)]
    call(plans[0])  # builds the shared tables, loads the kernels
    free = torch.cuda.mem_get_info()[0]
    call(plans[1])
    took = free - torch.cuda.mem_get_info()[0]
    # scratch grows by an eighth more than it needs, in pages of 2 MiB
    assert took <= 1.125 * plans[1].workspace_size(nb, prec) + 3 * 2 ** 21


@pytest.mark.parametrize("first,then", [("real32", "f64"), ("real32", "complex32"), ("f64", "imag64"), ("fly", "imagfly")])
def test_captured_call_keeps_its_scratch_when_another_needs_more(first, then):
    """A captured call has the scratch's address; a larger need of another call of the same batch leaves that buffer."""
    import torch
    bw, nb = (64, 3) if then in ("f64", "imagfly") else (101, 3)
    f32 = first.endswith("32")
    grid = _cuda(nb, 4 * bw * bw, dtype="float32" if f32 else "float64")
    oc = [_cuda(nb, bw * bw, dtype="float32" if f32 else "float64") for _ in range(2)]
    g2 = _cuda(nb, 4 * bw * bw, dtype="float32" if then == "complex32" else "float64")
    o2 = [torch.empty(nb, bw * bw, dtype=g2.dtype, device="cuda") for _ in range(2)]
    plan = api.Plan(bw, bw, fly=first == "fly")

    def call(**kw):
        if f32:
            plan.fst_real_f32(grid, *oc, nb, api.PREC_BF16X3, **kw)
        elif first == "fly":
            plan.fst(grid, None, *oc, 1, api.REAL, **kw)
        else:
            plan.fst(grid, None, *oc, nb, api.REAL, **kw)

    call()
    torch.cuda.synchronize()
    want = [c.clone() for c in oc]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(stream=torch.cuda.current_stream())
    if then == "complex32":
        plan.fst_complex_f32(g2, g2, *o2, nb, api.PREC_BF16X3)
    else:
        plan.fst(g2, g2 if then.startswith("imag") else None, *o2, nb, api.REAL)
    torch.cuda.synchronize()
    junk = [torch.full((2 ** k,), float("nan"), device="cuda") for k in range(16, 25)]  # takes what was freed
    for c in oc:
        c.zero_()
    graph.replay()
    torch.cuda.synchronize()
    plan.sync_status()
    assert all(torch.isnan(j).all() for j in junk)
    n = 1 if first == "fly" else nb
    assert (oc[0][:n] == want[0][:n]).all() and (oc[1][:n] == want[1][:n]).all()


def test_plans_of_several_threads_do_not_disturb_each_other():
    """One plan and stream a thread, the same kernels at different sizes: every call is accepted, every result the one a
    thread alone gets."""
    import threading

    import torch
    errors = []

    def worker(make, stream, want):
        try:
            with torch.cuda.stream(stream):
                run, out = make(stream)
                for _ in range(300):
                    run()
                stream.synchronize()
                if want is not None:
                    assert all((a == b).all() for a, b in zip(out, want))
            return [o.clone() for o in out]
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    def f32(bw):
        g = _cuda(3, 4 * bw * bw, dtype="float32")

        def make(stream):
            plan, out = api.Plan(bw, bw), [torch.zeros(3, bw * bw, dtype=torch.float32, device="cuda") for _ in range(2)]
            back = torch.zeros_like(g)

            def run():
                plan.fst_real_f32(g, *out, 3, api.PREC_BF16X3, stream=stream)
                plan.inv_fst_real_f32(*out, back, 3, api.PREC_BF16X3, stream=stream)
            return run, [*out, back]
        return make

    def f64(bw, fly):
        g = _cuda(1, 4 * bw * bw)

        def make(stream):
            plan, out = api.Plan(bw, bw, fly=fly), [torch.zeros(1, bw * bw, dtype=torch.float64, device="cuda") for _ in range(2)]
            back = torch.zeros_like(g)

            def run():
                plan.fst(g, None, *out, 1, api.REAL, stream=stream)
                plan.inv_fst(*out, back, None, 1, api.REAL, stream=stream)
            return run, [*out, back]
        return make

    makes = [f32(17), f32(31), f32(33), f32(47), f64(16, False), f64(128, True), f64(32, True), f64(48, False)]
    streams = [torch.cuda.Stream() for _ in makes]
    torch.cuda.synchronize()
    alone = [worker(m, s, None) for m, s in zip(makes, streams)]
    threads = [threading.Thread(target=worker, args=a) for a in zip(makes, streams, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("kind,bw,nb", [("f64", 256, 70), ("real32", 20, 3000), ("real32", 16, 9), ("real32", 255, 140),
                                        ("complex32", 255, 140), ("real32", 64, 9), ("f64", 40, 9), ("f64", 16, 9)])
def test_results_may_overlap_what_they_are_made_from(kind, bw, nb):
    """The coefficients in the first half of the samples' buffer, there and back: the same bits as apart."""
    import torch
    n, c, two = 4 * bw * bw, bw * bw, kind == "complex32"
    dt = "float64" if kind == "f64" else "float32"
    plan = api.Plan(bw, bw)

    def fwd(g, h, rc, ic):
        if kind == "f64":
            plan.fst(g, None, rc, ic, nb, api.REAL)
        elif two:
            plan.fst_complex_f32(g, h, rc, ic, nb, api.PREC_BF16X3)
        else:
            plan.fst_real_f32(g, rc, ic, nb, api.PREC_BF16X3)

    def inv(rc, ic, g, h):
        if kind == "f64":
            plan.inv_fst(rc, ic, g, None, nb, api.REAL)
        elif two:
            plan.inv_fst_complex_f32(rc, ic, g, h, nb, api.PREC_BF16X3)
        else:
            plan.inv_fst_real_f32(rc, ic, g, nb, api.PREC_BF16X3)

    g, h = _cuda(nb, n, dtype=dt), _cuda(nb, n, dtype=dt)
    rc, ic = (torch.empty(nb, c, dtype=g.dtype, device="cuda") for _ in range(2))
    gi, hi = g.clone(), h.clone()
    ri, ii = (gi.view(-1)[k * nb * c:(k + 1) * nb * c] for k in range(2))
    fwd(g, h, rc, ic)
    fwd(gi, hi, ri, ii)
    torch.cuda.synchronize()
    assert (ri == rc.view(-1)).all() and (ii == ic.view(-1)).all()
    inv(rc, ic, g, h)
    inv(ri, ii, gi, hi)
    plan.sync_status()
    assert (gi == g).all() and (not two or (hi == h).all())


def test_group_results_may_overlap_what_they_are_made_from():
    import torch
    group = api.Group([16, 77, 20, 64, 16, 255, 20, 128, 17, 77, 16] * 4)
    gt, ct = group.grid_total, group.coeff_total
    g = _cuda(gt, dtype="float32")
    rc, ic, back = (torch.empty(k, dtype=torch.float32, device="cuda") for k in (ct, ct, gt))
    start = g.clone()
    group.fst_inv(g, rc, ic, back)
    buf = torch.empty(gt, dtype=torch.float32, device="cuda")
    for _ in range(2):  # at once, then as the captured graph
        buf.copy_(start)
        ri, ii = buf[:ct], buf[(ct + 3) // 4 * 4:][:ct]
        group.fst(buf, ri, ii)
        torch.cuda.synchronize()
        assert (ri == rc).all() and (ii == ic).all()
        group.inv_fst(ri, ii, buf)
        group.sync_status()
        assert (buf == back).all()


@pytest.mark.parametrize("bw,group", [(256, 4), (256, 6), (512, 2), (512, 3), (1024, 1), (1024, 2)])
def test_digits_that_agree_in_sign(bw, group):
    """The digit products' accumulators are FP32: a group of digit products is exact up to 2^24, which these groups stay
    below for any data.  Data made for one row of the forward Legendre table (l = 4, m = 0; rows of samples constant),
    the digits of the latitudes chosen so that all products of the group agree in sign.  Allowed: the table's own
    rounding, two units in the last place of each value."""
    import torch
    S, ld, l = 2 * bw, np.longdouble, 4
    w = np.zeros(4 * bw)
    api.GenerateWeightsForDLT(bw, w)
    th = (np.arange(bw).astype(ld) * 2 + 1) * np.arctan(ld(1)) * 2 / S
    x, prev, cur = np.cos(th), np.zeros(bw, ld), np.full(bw, np.sqrt(ld(0.5)))
    for k in range(l):
        d = ld(k + 1) ** 2
        nxt = np.sqrt((2 * k + 3) * ld(2 * k + 1) / d) * x * cur
        if k:
            nxt -= np.sqrt((2 * k + 3) * ld(k) ** 2 / ((2 * k - 1) * d)) * prev
        prev, cur = cur, nxt
    row = cur * w[:bw] * np.sqrt(8 * np.arctan(ld(1))) / S
    tb, vb = {256: (54, 56), 512: (55, 54), 1024: (54, 54)}[bw]  # bits of table and data values
    u = np.ldexp(row.astype(float), tb - np.frexp(float(np.abs(row).max()))[1])
    u = np.rint(u).astype(np.int64) + 0x0000808080808080
    T = [u >> 48] + [((u >> (8 * (6 - b))) & 255) - 128 for b in range(1, 7)]
    v, s = np.zeros(bw, np.int64), 0
    for b in range(group + 1):
        digit = np.where(T[group - b] >= 0, 1, -1) * (2 ** (vb - 48) - 1 if b == 0 else 127)
        v += digit << (8 * (6 - b))
        s += int((digit * T[group - b]).sum())
    assert 2 ** 22 < s < 2 ** 24  # the group's sum
    samples = np.repeat(np.concatenate([v, v[::-1]]).astype(float)[:, None], S, 1) * 2.0 ** -vb
    plan = api.Plan(bw, bw)
    rc, ic = (torch.empty(1, bw * bw, dtype=torch.float64, device="cuda") for _ in range(2))
    plan.fst(torch.from_numpy(samples).cuda(), None, rc, ic, 1, api.REAL)
    plan.sync_status()
    X = v.astype(ld) * ld(2.0) ** -vb * (2 * S)
    e = abs(ld(rc[0, int(harmonic_index(0, l, bw))].item()) - (row * X).sum())
    assert e <= 2.0 ** -51 * float((np.abs(row) * np.abs(X)).sum())


def test_groups_of_classes_transformed_whole_hold_no_intermediates():
    import torch
    api.Group([16, 20])  # tables
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    group = api.Group([16] * 8192 + [20] * 4096)  # samples: 58 MB
    assert free - torch.cuda.mem_get_info()[0] <= 4 * 2 ** 21
    del group


def test_first_digit_call_while_another_thread_captures():
    """A plan whose scratch is there allocates nothing in its FP64 calls but for the digit tables and their scratch: that
    neither fails nor ends a capture of another thread."""
    import threading

    import torch
    bw, nb = 53, 4
    grid, oc = _cuda(nb, 4 * bw * bw), [_cuda(nb, bw * bw) for _ in range(2)]
    plan = api.Plan(bw, bw)
    plan.fzt(grid, None, *oc, nb, api.REAL)
    torch.cuda.synchronize()
    x, s, errors = torch.ones(1000, device="cuda"), torch.cuda.Stream(), []

    def worker():
        try:
            plan.fst(grid, None, *oc, nb, api.REAL, stream=s)
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        x.mul_(2.0)
        t = threading.Thread(target=worker)
        t.start()
        t.join()
    assert not errors, errors
    graph.replay()
    torch.cuda.synchronize()
    plan.sync_status()
    assert (x == 2.0).all()
    first = [c.clone() for c in oc]
    plan.fst(grid, None, *oc, nb, api.REAL)
    plan.sync_status()
    assert (oc[0] == first[0]).all() and (oc[1] == first[1]).all()
