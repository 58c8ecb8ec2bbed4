"""One function at a time (the drop-ins, one-order transforms): the FP64 kernels' single-function paths and
their results in the caller's host memory, against the oracle, at remainders of the eight-lane rows, of the
shared degree ranges and of the longitude blocks.  Tolerance: the FP64 parity bar, 1e-11 normwise."""
import numpy as np
import pytest

from s2kit_gb300 import api
from tests._util import real_field_coeffs, rel_err_norm

pytestmark = pytest.mark.gpu
TOL = 1e-11


@pytest.mark.parametrize("bw,cutoff", [(2, 1), (3, 3), (5, 2), (8, 8), (24, 11), (33, 33), (64, 64), (65, 40),
                                       (127, 127), (200, 150), (256, 256)])
@pytest.mark.parametrize("fmt", [api.REAL, api.COMPLEX])
def test_drop_ins_match_oracle(oracle, bw, cutoff, fmt):
    rng = np.random.default_rng(bw + 7 * cutoff)
    n = 4 * bw * bw
    size = api.Reduced_Naive_TableSize(bw, cutoff) + api.Reduced_SpharmonicTableSize(bw, cutoff)
    fwd = api.SemiNaive_Naive_Pml_Table(bw, cutoff, np.zeros(size), None)
    inv = api.Transpose_SemiNaive_Naive_Pml_Table(fwd, bw, cutoff, np.zeros(size), None)
    w = np.zeros(4 * bw)
    api.GenerateWeightsForDLT(bw, w)
    rc, ic = real_field_coeffs(rng, bw, 1.0)
    g = np.empty((2, n))
    api.InvFSTSemiMemo(rc, ic, g[0], g[1], bw, inv, None, fmt, cutoff)
    er, ei = oracle.inv_fst(rc, ic, bw, fmt, cutoff)
    assert rel_err_norm(g[0], g[1], er, ei) <= TOL
    x = rng.standard_normal((2, n))
    c = np.empty((2, bw * bw))
    api.FSTSemiMemo(x[0], x[1], c[0], c[1], bw, fwd, None, fmt, cutoff, weights=w)
    assert rel_err_norm(c[0], c[1], *oracle.fst(x[0], x[1], bw, fmt, cutoff)) <= TOL
    # results may go where the inputs were
    y = x.copy()
    api.FSTSemiMemo(y[0], y[1], y[0][:bw * bw], y[1][:bw * bw], bw, fwd, None, fmt, cutoff, weights=w)
    assert (y[0][:bw * bw] == c[0]).all() and (y[1][:bw * bw] == c[1]).all()
    z = np.empty((2, 2 * bw))
    api.FZTSemiMemo(x[0], x[1], z[0], z[1], bw, oracle.cos_pml_table(bw, 0), None, fmt, weights=w)
    er, ei = oracle.fzt(x[0], x[1], bw, fmt)
    assert rel_err_norm(z[0][:bw], z[1][:bw], er[:bw], ei[:bw]) <= TOL
