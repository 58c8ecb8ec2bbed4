"""FP32 transforms of bandwidths 16 to 31 (one kernel each way, csrc/small32.cuh) and 32 against the oracle, at the sizes
where folds, 4 x 4 tiles and a block's functions have remainders.

Tolerance: tables, samples and results are rounded at 2^-24 = 6e-8, the sums are two chains of at most 16
terms; a few 1e-7 normwise.
"""
import numpy as np
import pytest

from s2kit_gb300 import api
from tests._util import real_field_coeffs, rel_err_norm

pytestmark = pytest.mark.gpu
TOL = 5e-7


def _run(bw, rc, ic, gr):
    import torch

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda().reshape(-1)

    nb = len(rc)
    plan = api.Plan(bw, bw)
    og = dev(np.full((nb, 4 * bw * bw), 7.0))
    oc = [dev(np.full((nb, bw * bw), 7.0)) for _ in range(2)]
    plan.inv_fst_real_f32(dev(rc), dev(ic), og, nb)
    plan.fst_real_f32(dev(gr), oc[0], oc[1], nb)
    torch.cuda.synchronize()
    plan.sync_status()
    return [x.cpu().numpy().reshape(nb, -1) for x in [og] + oc]


def _data(bw, nb):
    rng = np.random.default_rng(bw * 100 + nb)
    rc, ic = real_field_coeffs(rng, bw, 1.0, nb)
    gr = rng.standard_normal((nb, 4 * bw * bw))
    return [x.astype(np.float32) for x in (rc, ic, gr)]


@pytest.mark.parametrize("bw,nb", [(16, 1), (16, 6), (17, 3), (18, 1), (19, 2), (20, 5), (22, 2), (23, 1), (25, 3), (26, 4),
                                   (28, 1), (30, 3), (31, 5), (32, 1), (32, 7)])
def test_small_bandwidths_match_oracle(oracle, bw, nb):
    rc, ic, gr = _data(bw, nb)
    og, ocr, oci = _run(bw, rc, ic, gr)
    z = np.zeros(4 * bw * bw)
    for f in {0, nb // 2, nb - 1}:
        er, _ = oracle.inv_fst(rc[f].astype(float), ic[f].astype(float), bw, api.REAL, bw)
        assert rel_err_norm(og[f], 0.0, er, 0.0) <= TOL
        er, ei = oracle.fst(gr[f].astype(float), z, bw, api.REAL, 1)
        assert rel_err_norm(ocr[f], oci[f], er, ei) <= TOL


@pytest.mark.parametrize("bw", [16, 21, 32])
def test_small_results_do_not_depend_on_the_batch(bw):
    """Alone, in a batch that takes the other register split, and next to a function of NaN."""
    nb = 2500
    rc, ic, gr = _data(bw, nb)
    gr[nb - 2], rc[nb - 2] = np.nan, np.nan
    many = _run(bw, rc, ic, gr)
    for f in (0, 1, nb - 3, nb - 1):
        for a, b in zip(many, _run(bw, rc[f:f + 1], ic[f:f + 1], gr[f:f + 1])):
            assert (a[f] == b[0]).all()
    assert all(np.isnan(x[nb - 2]).any() for x in many)
