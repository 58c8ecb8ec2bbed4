"""The FP64 plan transforms on the tensor cores (exact digit products, csrc/digit_gemm.cu) against the
oracle, at the sizes where tiles, folds and column blocks have remainders.

Tolerance: the digit path rounds operands to 53 bits and more of their row's largest value, a few
1e-15 normwise; the oracle's recurrence adds up to 1e-13 at these bandwidths, so 1e-12 holds for both.
"""
import numpy as np
import pytest

from s2kit_gb300 import api
from tests._util import degree_of_index, real_field_coeffs, rel_err_norm

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _run(bw, nb, mode, cutoff, rc, ic, gr, gi, shift=0, fly=False):
    """Inverse of (rc, ic) and forward of (gr, gi); device buffers start `shift` doubles into an allocation."""
    import torch

    def dev(x):
        t = torch.full((x.size + shift,), 7.0, dtype=torch.float64, device="cuda")
        t[shift:] = torch.from_numpy(np.ascontiguousarray(x)).cuda().reshape(-1)
        return t[shift:]

    fmt = api.COMPLEX if mode == "complex" else api.REAL
    two = mode != "real"
    plan = api.Plan(bw, cutoff, fly=fly)
    n, c = 4 * bw * bw, bw * bw
    og, oc = [dev(np.full((nb, n), 7.0)) for _ in range(2)], [dev(np.full((nb, c), 7.0)) for _ in range(2)]
    plan.inv_fst(dev(rc), dev(ic), og[0], og[1] if two else None, nb, fmt)
    plan.fst(dev(gr), dev(gi) if two else None, oc[0], oc[1], nb, fmt)
    torch.cuda.synchronize()
    plan.sync_status()
    og, oc = [g.cpu().numpy().reshape(nb, n) for g in og], [x.cpu().numpy().reshape(nb, c) for x in oc]
    if not two:
        assert (og[1] == 7.0).all()
        og[1] = np.zeros_like(og[0])
    return og, oc


def _data(bw, nb, mode):
    rng = np.random.default_rng(bw * 1000 + nb)
    rc, ic = real_field_coeffs(rng, bw, 1.0, nb)
    if mode == "complex":
        rc, ic = rng.standard_normal(rc.shape), rng.standard_normal(rc.shape)
    elif mode == "imag":  # REAL with imaginary arrays: Im f(l, 0) counts
        ic += (degree_of_index(bw)[1] == 0) * rng.standard_normal(ic.shape)
    gr = rng.standard_normal((nb, 4 * bw * bw))
    gi = rng.standard_normal(gr.shape) if mode != "real" else np.zeros_like(gr)
    return rc, ic, gr, gi


@pytest.mark.parametrize("bw,nb,mode,cutoff", [
    (9, 1, "complex", 9), (12, 9, "real", 5), (15, 70, "real", 15), (31, 3, "complex", 31), (32, 8, "real", 32),
    (33, 17, "imag", 20), (34, 16, "complex", 34), (48, 9, "real", 48), (96, 2, "imag", 96), (64, 33, "real", 64), (100, 5, "imag", 100), (127, 2, "real", 64),
    (130, 9, "complex", 130), (255, 1, "real", 255), (256, 1, "imag", 256), (256, 40, "real", 256),
    (257, 2, "real", 257), (258, 1, "complex", 200), (511, 1, "real", 511), (512, 1, "real", 512)])
def test_digit_path_matches_oracle(oracle, bw, nb, mode, cutoff):
    rc, ic, gr, gi = _data(bw, nb, mode)
    og, oc = _run(bw, nb, mode, cutoff, rc, ic, gr, gi)
    fmt = api.COMPLEX if mode == "complex" else api.REAL
    for f in {0, nb // 2, nb - 1}:
        er, ei = oracle.inv_fst(rc[f], ic[f], bw, fmt, cutoff)
        assert rel_err_norm(og[0][f], og[1][f], er, ei if mode != "real" else 0.0) <= TOL
        # the samples are noise: the oracle's naive form (cutoff 1), since the seminaive form's tables are
        # themselves up to 3e-12 off at order 1 on samples that are not band-limited
        er, ei = oracle.fst(gr[f], gi[f], bw, fmt, 1)
        assert rel_err_norm(oc[0][f], oc[1][f], er, ei) <= TOL


@pytest.mark.parametrize("bw,nb,mode", [(64, 2, "real"), (65, 9, "complex"), (100, 33, "real"), (127, 1, "imag"),
                                        (255, 3, "complex"), (256, 17, "real"), (300, 2, "real"), (512, 2, "real")])
def test_digit_path_without_tables_matches_oracle(oracle, bw, nb, mode):
    """On-the-fly plans: the digit tables generated chunk by chunk in scratch (one chunk up to several)."""
    rc, ic, gr, gi = _data(bw, nb, mode)
    og, oc = _run(bw, nb, mode, bw, rc, ic, gr, gi, fly=True)
    fmt = api.COMPLEX if mode == "complex" else api.REAL
    for f in {0, nb - 1}:
        er, ei = oracle.inv_fst(rc[f], ic[f], bw, fmt, bw)
        assert rel_err_norm(og[0][f], og[1][f], er, ei if mode != "real" else 0.0) <= TOL
        assert rel_err_norm(oc[0][f], oc[1][f], *oracle.fst(gr[f], gi[f], bw, fmt, 1)) <= TOL


def test_digit_path_unaligned_buffers():
    """8-byte aligned device pointers give the same bits as 16-byte aligned ones."""
    for mode in ("real", "imag", "complex"):
        d = _data(40, 3, mode)
        a, b = _run(40, 3, mode, 40, *d), _run(40, 3, mode, 40, *d, shift=1)
        for x, y in zip(a[0] + a[1], b[0] + b[1]):
            assert (x == y).all()


@pytest.mark.parametrize("bw", [33, 64])
def test_digit_path_special_values(oracle, bw):
    """A NaN or an infinity stays within its function; zeros, tiny and huge scales keep their precision."""
    rc, ic, gr, gi = _data(bw, 5, "real")
    gr[1, 7] = np.nan
    gr[2, bw] = np.inf
    rc[1, 3], ic[2, bw + 2] = np.nan, -np.inf
    gr[3], rc[3], ic[3] = 0.0, 0.0, 0.0
    rc[4], ic[4], gr[4] = rc[4] * 1e-290, ic[4] * 1e-290, gr[4] * 1e290
    og, oc = _run(bw, 5, "real", bw, rc, ic, gr, gi)
    for f in (1, 2):
        assert np.isnan(og[0][f]).all() and np.isnan(oc[0][f]).all()
    assert (og[0][3] == 0).all() and (oc[0][3] == 0).all() and (oc[1][3] == 0).all()
    for f in (0, 4):
        er, _ = oracle.inv_fst(rc[f], ic[f], bw, api.REAL, bw)
        assert rel_err_norm(og[0][f], 0 * er, er, 0 * er) <= TOL
        s = 1e-290 if f == 4 else 1.0  # the metric squares its arguments
        er, ei = oracle.fst(gr[f], gi[f], bw, api.REAL, bw)
        assert rel_err_norm(oc[0][f] * s, oc[1][f] * s, er * s, ei * s) <= TOL


def test_digit_path_under_capture():
    """A captured call on a warm plan replays with new inputs; a capture before the first call still works."""
    import torch
    bw, nb = 48, 4
    d = _data(bw, nb, "real")
    gr = torch.from_numpy(d[2]).cuda()
    rc, ic = (torch.empty(nb, bw * bw, dtype=torch.float64, device="cuda") for _ in range(2))
    plan = api.Plan(bw, bw)
    plan.fst(gr, None, rc, ic, nb, api.REAL)
    want = [rc.clone(), ic.clone()]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        plan.fst(gr, None, rc, ic, nb, api.REAL, stream=s)
    gr.mul_(2.0)
    graph.replay()
    torch.cuda.synchronize()
    plan.sync_status()
    assert (rc == 2 * want[0]).all() and (ic == 2 * want[1]).all()


def _run32(bw, nb, rc, ic, gr, gi):
    """FP32 inverse of (rc, ic) and forward of (gr, gi) at a chirp-z bandwidth (gi None: real fields)."""
    import torch

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda().reshape(-1)

    plan = api.Plan(bw, bw)
    og = [dev(np.full((nb, 4 * bw * bw), 7.0)) for _ in range(2)]
    oc = [dev(np.full((nb, bw * bw), 7.0)) for _ in range(2)]
    if gi is None:
        plan.inv_fst_real_f32(dev(rc), dev(ic), og[0], nb)
        plan.fst_real_f32(dev(gr), oc[0], oc[1], nb)
    else:
        plan.inv_fst_complex_f32(dev(rc), dev(ic), og[0], og[1], nb)
        plan.fst_complex_f32(dev(gr), dev(gi), oc[0], oc[1], nb)
    torch.cuda.synchronize()
    plan.sync_status()
    return [x.cpu().numpy().astype(np.float64).reshape(nb, -1) for x in og + oc]


# FP32 samples and coefficients: inputs and results round at 2^-24 = 6e-8; the table's 25 and the data's 30 bits
# of a row's largest value, and one more rounding between the stages, leave a few times that: 5e-7.
@pytest.mark.parametrize("bw,nb,cplx", [(65, 9, False), (65, 2, True), (66, 33, False), (77, 1, False), (100, 17, True),
                                        (127, 3, False), (130, 70, False), (250, 2, True), (254, 5, False),
                                        (255, 1, True), (255, 33, False)])
def test_fp32_digit_path_matches_oracle(oracle, bw, nb, cplx):
    rc, ic, gr, gi = (x.astype(np.float32).astype(np.float64) for x in _data(bw, nb, "complex" if cplx else "real"))
    igr, igi, orc, oic = _run32(bw, nb, rc, ic, gr, gi if cplx else None)
    fmt = api.COMPLEX if cplx else api.REAL
    for f in {0, nb // 2, nb - 1}:
        er, ei = oracle.inv_fst(rc[f], ic[f], bw, fmt, bw)
        assert rel_err_norm(igr[f], igi[f] if cplx else 0.0, er, ei if cplx else 0.0) <= 5e-7
        er, ei = oracle.fst(gr[f], gi[f], bw, fmt, 1)
        assert rel_err_norm(orc[f], oic[f], er, ei) <= 5e-7


def test_fp32_digit_path_scales_and_nan_stay_with_their_function():
    bw, nb = 90, 9
    rc, ic, gr, gi = _data(bw, nb, "real")
    want = _run32(bw, nb, rc, ic, gr, None)
    gr[3] *= 2.0 ** 60  # exact, and so are its results
    rc[4, 7], gr[5, 11] = np.nan, np.inf
    got = _run32(bw, nb, rc, ic, gr, None)
    for w, g, bad in zip(want[:1] + want[2:], got[:1] + got[2:], (4, 5, 5)):
        assert not np.isfinite(g[bad]).any()
        for f in set(range(nb)) - {bad}:
            assert (g[f] == w[f] * (2.0 ** 60 if bad == 5 and f == 3 else 1.0)).all()


@pytest.mark.parametrize("bw,nb,prec", [(16, 3, api.PREC_BF16X3), (33, 2, api.PREC_BF16X2), (64, 9, api.PREC_FP16X2),
                                        (101, 2, api.PREC_BF16X3), (512, 1, api.PREC_BF16X3)])
def test_refined_transforms_have_fp64_precision(oracle, bw, nb, prec):
    import torch

    from s2kit_gb300 import S2GError

    rc, ic, gr, gi = _data(bw, nb, "real")
    plan = api.Plan(bw, bw)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (rc, ic, gr)]
    og = torch.full_like(d[2], 7.0)
    oc = [torch.full_like(d[0], 7.0) for _ in range(2)]
    plan.inv_fst_refined(d[0], d[1], og, nb, prec)
    plan.fst_refined(d[2], oc[0], oc[1], nb, prec)
    torch.cuda.synchronize()
    for f in {0, nb - 1}:
        er, _ = oracle.inv_fst(rc[f], ic[f], bw, api.REAL, bw)
        assert rel_err_norm(og[f].cpu().numpy().ravel(), 0.0, er, 0.0) <= TOL
        er, ei = oracle.fst(gr[f], gi[f], bw, api.REAL, 1)
        assert rel_err_norm(oc[0][f].cpu().numpy(), oc[1][f].cpu().numpy(), er, ei) <= TOL
    with pytest.raises(S2GError):
        plan.fst_refined(d[2], oc[0], oc[1], nb, api.PREC_FP64)
